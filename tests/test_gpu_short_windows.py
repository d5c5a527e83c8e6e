"""Traceback windows of a few posterior anti-diagonals each, in batches that leave the GPU idle and that fill it
(the wide bands' worker is another form there): every read's pairs are those of the read alone, which are the
oracle's within the FP32 form's 1e-4."""
import numpy as np
import pytest

from oracle import oracle as orc
from signalalign_b200 import synth
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from signalalign_b200 import api as a
    return a


@pytest.mark.parametrize("expansion", [50, 200, 230])
@pytest.mark.parametrize("traceback,between", [(1, 4), (5, 12), (5, 23), (40, 50)])
def test_batches(api, expansion, traceback, between):
    cfg = synth.config1(seed=411, n_reads=2, span=(600, 700))
    m = W.gaussian_model(cfg)
    sm = W.gpu_model(api, m, orc.EMIT_DESCALED)
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=expansion, traceback_diagonals=traceback,
                                                         min_diags_between_traceback=between)
    inputs = [api.ReadInput(sm=sm, reference=rd["reference"], events=rd["events"], anchors=rd["anchors"],
                            scale=rd["scale"], shift=rd["shift"]) for rd in cfg["reads"]]
    alone = [api.align_batch([r], p) for r in inputs]
    for rd, b in zip(cfg["reads"], alone):
        want = orc.aligned_pairs(W.oracle_model(m, orc.EMIT_DESCALED, rd), rd["reference"], rd["events"], rd["anchors"],
                                 orc.params(threshold=p.threshold, expansion=expansion, min_diags=between,
                                            traceback=traceback), True, True)
        assert b.status(0) == 0 and len(want) > 100
        assert W.max_posterior_error(want, b.pairs(0), p.threshold) <= 1e-4
    many = api.align_batch(inputs * 120, p)   # 4e5 anti-diagonals
    for i in range(240):
        assert many.status(i) == 0
        assert np.array_equal(many.pairs(i), alone[i % 2].pairs(0))
        assert many.log_likelihood(i) == alone[i % 2].log_likelihood(0)
