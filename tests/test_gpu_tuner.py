"""The launch tuner times what the worker of a batch's width class can run: both forms, each at up to as many
CTAs per SM as it can have (column-resident: three of 128 threads, two of 256, one of 512)."""
import numpy as np
import pytest

from oracle import oracle as orc
from signalalign_b200 import synth
import workloads as W

pytestmark = pytest.mark.gpu

GRIDS = 4 * 3   # CTAs per region times CTAs of the emission kernel


@pytest.fixture(scope="module")
def api():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from signalalign_b200 import api as a
    return a


@pytest.mark.parametrize("expansion,width_class,column_ctas", [(50, 1, 3), (100, 2, 2), (240, 4, 1)])
def test_candidates(api, expansion, width_class, column_ctas):
    cfg = synth.config1(seed=43, n_reads=2, span=(800, 1200))
    m = W.gaussian_model(cfg)
    sm = W.gpu_model(api, m, orc.EMIT_DESCALED)
    inputs = [api.ReadInput(sm=sm, reference=rd["reference"], events=rd["events"], anchors=rd["anchors"],
                            scale=rd["scale"], shift=rd["shift"]) for rd in cfg["reads"]]
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=expansion)
    saved = api.get_launch_config(0, width_class)
    try:
        b = api.Batch(inputs, p)
        b.upload()
        best, ms, tried = api.tune_launch_config(b, None, 1)
        assert tried % GRIDS == 0 and tried >= GRIDS * (column_ctas + 1) and ms > 0
        assert api.get_launch_config(0, width_class) == best
        b.download()
        for i, rd in enumerate(cfg["reads"]):
            want = orc.aligned_pairs(W.oracle_model(m, orc.EMIT_DESCALED, rd), rd["reference"], rd["events"],
                                     rd["anchors"], orc.params(threshold=p.threshold, expansion=expansion), True, True)
            assert W.max_posterior_error(want, b.pairs(i), p.threshold) <= 1e-4
    finally:
        api.set_launch_config(0, width_class, saved)
