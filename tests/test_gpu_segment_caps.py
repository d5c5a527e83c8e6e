"""The automatic cap of forward segments (sa_setSegmentPolicy 0).

Wide bands: their warm-up of ten band widths leaves the cap's floor of 2,800 no room, and they are cut at
4,096.  A small batch's cap is the floor, so the automatic cuts are those of an explicit cap of 4,096, and
the results bit for bit.

The FP64 form sweeps regions of up to 4,096 anti-diagonals whole, so their scores are the oracle's to the
last unit."""
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


@pytest.mark.parametrize("events", [0, 3100, 3600, 4096, 4097])
def test_whole_regions_fp64(api, policy, events):
    """reads of 3,100 to 4,096 anti-diagonals (events: the anti-diagonals a read is cut to; 0: as drawn), in
    the single-read entry and with X sites in a batch"""
    cfg = synth.config1(seed=403, n_reads=1, span=(1480, 1480) if events == 0 else (1800, 1800))
    rd = cfg["reads"][0]
    lX = len(rd["reference"]) - 5
    if events:   # the reference's and the events' first parts, which end together
        cut = int(np.searchsorted(rd["true_pos"] + np.arange(len(rd["true_pos"])), events))
        lX = events - cut
        rd = dict(rd, reference=rd["reference"][:lX + 5], events=rd["events"][:cut])
        a = np.asarray(rd["anchors"]).reshape(-1, 2)
        rd["anchors"] = a[(a[:, 0] < lX - 8) & (a[:, 1] < cut - 8)]
        assert lX + cut == events
    m = W.gaussian_model(cfg)
    sm = W.gpu_model(api, m, orc.EMIT_DESCALED, rd)
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=50)
    call = lambda: api.getAlignedPairsUsingAnchors(sm, rd["reference"], rd["events"], rd["anchors"], p,
                                                   with_log_likelihood=True)
    api.set_segment_policy(0, 1024)
    got, ll = call()
    api.set_segment_policy(-1, 1024)
    whole, ll_whole = call()
    want, totals = orc.aligned_pairs(W.oracle_model(m, orc.EMIT_DESCALED, rd), rd["reference"], rd["events"],
                                     rd["anchors"], orc.params(threshold=p.threshold, expansion=50), True, True,
                                     with_total_probs=True)
    assert len(whole) == len(want) > 100
    for f in ("x", "y", "kmer"):
        assert np.array_equal(whole[f], want[f]), f
    if events != 4097:
        assert np.array_equal(got, whole) and ll == ll_whole
    else:
        assert W.max_posterior_error(whole, got, p.threshold) <= 1e-7 and abs(ll - ll_whole) <= 1e-9 * abs(ll_whole)


def test_whole_regions_fp64_in_a_batch(api, policy):
    cfg = synth.config3(seed=67, n_reads=2, span=(1250, 1450), grid_length=200, route="degenerate")
    m = formats.parse_model_lines(*synth.model_text("ACEGT", 6, cfg["gauss_table"]).split("\n")[:3])
    sm = W.gpu_model(api, m, orc.EMIT_DESCALED)
    inputs = [api.ReadInput(sm=sm, reference=rd["reference"], events=rd["events"], anchors=rd["anchors"],
                            scale=rd["scale"], shift=rd["shift"], degenerate=api.CYTOSINE_METHYLATION2)
              for rd in cfg["alignments"] if rd["model"] == "gauss"]
    assert all(3100 < len(r.reference) - 5 + len(r.events) <= 4096 for r in inputs)
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=50)
    auto, whole = _run(api, inputs, p, 0), _run(api, inputs, p, -1)
    assert auto.segment_info()["stitches"] == 0
    _same(auto, whole, len(inputs))
