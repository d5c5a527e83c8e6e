"""The automatic cap of forward segments (sa_setSegmentPolicy 0) where the bands are wide: their warm-up of
ten band widths leaves the cap's floor of 2,800 no room, and they are cut at 4,096.  A small batch's cap is
the floor, so the automatic cuts are those of an explicit cap of 4,096, and the results bit for bit."""
import numpy as np
import pytest

from oracle import formats
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


@pytest.fixture
def policy(api):
    saved = api.get_segment_policy()
    yield
    api.set_segment_policy(*saved)


def _run(api, inputs, p, segment_diags):
    api.set_segment_policy(segment_diags, 1024)
    return api.align_batch(inputs, p)


def _same(a, b, n):
    for i in range(n):
        assert a.status(i) == 0 and b.status(i) == 0
        assert len(a.pairs(i)) > 100 and np.array_equal(a.pairs(i), b.pairs(i))
        assert a.log_likelihood(i) == b.log_likelihood(i)


@pytest.mark.parametrize("expansion", [220, 260, 340])
def test_wide_bands_fp32(api, policy, expansion):
    cfg = synth.config1(seed=401, n_reads=2, span=(5000, 6000))
    sm = W.gpu_model(api, W.gaussian_model(cfg), orc.EMIT_DESCALED)
    inputs = [api.ReadInput(sm=sm, reference=rd["reference"], events=rd["events"], anchors=rd["anchors"],
                            scale=rd["scale"], shift=rd["shift"]) for rd in cfg["reads"]]
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=expansion)
    auto, cut = _run(api, inputs, p, 0), _run(api, inputs, p, 4096)
    info = auto.segment_info()
    assert info["stitches"] > 0 and info["stitches"] == cut.segment_info()["stitches"] and info["redone"] == 0, info
    _same(auto, cut, len(inputs))


def test_wide_bands_fp64(api, policy):
    cfg = synth.config3(seed=66, n_reads=1, span=(6000, 7000), grid_length=200, route="degenerate")
    rd = [a for a in cfg["alignments"] if a["model"] == "gauss"][0]
    m = formats.parse_model_lines(*synth.model_text("ACEGT", 6, cfg["gauss_table"]).split("\n")[:3])
    inputs = [api.ReadInput(sm=W.gpu_model(api, m, orc.EMIT_DESCALED), reference=rd["reference"], events=rd["events"],
                            anchors=rd["anchors"], scale=rd["scale"], shift=rd["shift"],
                            degenerate=api.CYTOSINE_METHYLATION2)]
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=260)
    auto, cut = _run(api, inputs, p, 0), _run(api, inputs, p, 4096)
    info = auto.segment_info()
    assert info["stitches"] > 0 and info["stitches"] == cut.segment_info()["stitches"] and info["redone"] == 0, info
    _same(auto, cut, 1)
