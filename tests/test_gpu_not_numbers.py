"""Events and tables that are not numbers in the plain FP64 form, on both its routes: where the reference's
logAdd gives NaN, so do the kernels', whichever of its arguments it is.  An event of zero noise has no
log-probability (an infinity less an infinity), so every path through its row is NaN: the read's total is
NaN, the windows before it give their pairs and the ones it touches give none, as in the oracle."""
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


def _read(kind, bases=1500):
    cfg = synth.config1(seed=501, n_reads=1, span=(bases, bases))
    rd = dict(cfg["reads"][0])
    ev = np.array(rd["events"], dtype=np.float64)
    at = len(ev) * 2 // 3
    if kind == "zero noise":
        ev[at, 1] = 0.0
    elif kind == "zero noise, first":
        ev[0, 1] = 0.0
    elif kind == "zero noise, last":
        ev[-1, 1] = 0.0
    elif kind == "mean not a number":
        ev[at, 0] = np.nan
    elif kind == "negative noise":
        ev[at, 1] = -1.0
    elif kind == "infinite mean":      # no path: log 0, not NaN
        ev[at, 0] = np.inf
    elif kind == "infinite noise":
        ev[at, 1] = np.inf
    rd["events"] = ev
    return cfg, rd


KINDS = ["zero noise", "zero noise, first", "zero noise, last", "mean not a number", "negative noise", "infinite mean",
         "infinite noise"]


def _same_total(got, want):
    assert np.isnan(got) == np.isnan(want), (got, want)
    if np.isfinite(want):
        assert got == pytest.approx(want, rel=1e-12)
    elif not np.isnan(want):
        assert got == want


# 50 and 240: the resident route (128 and 480 threads); 500: the rings
@pytest.mark.parametrize("expansion", [50, 240, 500])
@pytest.mark.parametrize("kind", KINDS)
def test_events(api, kind, expansion):
    cfg, rd = _read(kind)
    m = W.gaussian_model(cfg)
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=expansion)
    got, ll = api.getAlignedPairsUsingAnchors(W.gpu_model(api, m, orc.EMIT_DESCALED, rd), rd["reference"], rd["events"],
                                              rd["anchors"], p, with_log_likelihood=True)
    want, totals = orc.aligned_pairs(W.oracle_model(m, orc.EMIT_DESCALED, rd), rd["reference"], rd["events"],
                                     rd["anchors"], orc.params(threshold=p.threshold, expansion=expansion), True, True,
                                     with_total_probs=True)
    _same_total(ll, dict(totals)[len(rd["reference"]) - 5 + len(rd["events"])])
    assert len(got) == len(want)
    for f in ("x", "y", "kmer"):
        assert np.array_equal(got[f], want[f]), f
    if len(want):
        assert np.abs(got["score"] - want["score"]).max() <= 1


@pytest.mark.parametrize("side", ["level mean", "skip"])
def test_tables(api, side):
    """a k-mer of the reference whose level mean or skip emission is not a number"""
    cfg, rd = _read("")
    m = dict(W.gaussian_model(cfg))
    kid = sum("ACGT".index(c) * 4 ** (5 - i) for i, c in enumerate(rd["reference"][900:906]))
    if side == "skip":
        m["gapx"] = np.array(m["gapx"], dtype=np.float64)
        m["gapx"][kid] = np.nan
    else:
        for t in ("match", "gapy"):
            m[t] = np.array(m[t], dtype=np.float64)
            m[t].reshape(-1, 5)[kid, 0] = np.nan
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=50)
    got, ll = api.getAlignedPairsUsingAnchors(W.gpu_model(api, m, orc.EMIT_DESCALED, rd), rd["reference"], rd["events"],
                                              rd["anchors"], p, with_log_likelihood=True)
    want, totals = orc.aligned_pairs(W.oracle_model(m, orc.EMIT_DESCALED, rd), rd["reference"], rd["events"],
                                     rd["anchors"], orc.params(threshold=p.threshold, expansion=50), True, True,
                                     with_total_probs=True)
    _same_total(ll, dict(totals)[len(rd["reference"]) - 5 + len(rd["events"])])
    for f in ("x", "y", "kmer"):
        assert np.array_equal(got[f], want[f]), f


@pytest.mark.parametrize("kind", ["zero noise", "infinite mean"])
def test_expectations(api, kind):
    cfg, rd = _read(kind, 900)
    m = W.gaussian_model(cfg)
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=50)
    got = api.getExpectationsUsingAnchors(W.gpu_model(api, m, orc.EMIT_DESCALED, rd), rd["reference"], rd["events"],
                                          rd["anchors"], p)
    want = orc.expectations(W.oracle_model(m, orc.EMIT_DESCALED, rd), rd["reference"], rd["events"], rd["anchors"],
                            orc.params(threshold=p.threshold, expansion=50))
    _same_total(got["likelihood"], want["likelihood"])
    for f in ("transitions", "posteriors", "event_expectations"):
        np.testing.assert_allclose(got[f], want[f], rtol=1e-9, atol=1e-9, equal_nan=True)
    assert np.array_equal(got["observed"], want["observed"])


def test_stitches(api):
    """a batch's X read with such an event in one of its forward segments, whose stitches disagree: the
    regions are run again whole"""
    from oracle import formats
    cfg = synth.config3(seed=66, n_reads=1, span=(6000, 6500), grid_length=200, route="degenerate")
    rd = dict([a for a in cfg["alignments"] if a["model"] == "gauss"][0])
    ev = np.array(rd["events"], dtype=np.float64)
    ev[len(ev) // 2, 1] = 0.0
    rd["events"] = ev
    m = formats.parse_model_lines(*synth.model_text("ACEGT", 6, cfg["gauss_table"]).split("\n")[:3])
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=50)
    b = api.align_batch([api.ReadInput(sm=W.gpu_model(api, m, orc.EMIT_DESCALED), reference=rd["reference"], events=ev,
                                       anchors=rd["anchors"], scale=rd["scale"], shift=rd["shift"],
                                       degenerate=api.CYTOSINE_METHYLATION2)], p)
    want = orc.aligned_pairs(W.oracle_model(m, orc.EMIT_DESCALED, rd), rd["reference"], ev, rd["anchors"],
                             orc.params(threshold=p.threshold, expansion=50), True, True, options="CE")
    assert b.segment_info()["stitches"] > 0
    assert b.status(0) == 0 and np.isnan(b.log_likelihood(0))
    got = b.pairs(0)
    for f in ("x", "y", "kmer"):
        assert np.array_equal(got[f], want[f]), f


@pytest.mark.parametrize("kind", KINDS)
def test_fp32_forms_agree(api, kind):
    """the batched form: the column-resident worker and the CTA form give the same, and a read beside such a
    read is untouched"""
    cfg, rd = _read(kind)
    clean = cfg["reads"][0]
    sm = W.gpu_model(api, W.gaussian_model(cfg), orc.EMIT_DESCALED)
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=50)
    one = lambda r: api.ReadInput(sm=sm, reference=r["reference"], events=r["events"], anchors=r["anchors"],
                                  scale=r["scale"], shift=r["shift"])
    saved = api.get_launch_config(0, 1)
    try:
        api.set_launch_config(0, 1, dict(saved, warp_windows=1))
        columns, alone = api.align_batch([one(rd), one(clean)], p), api.align_batch([one(clean)], p)
        api.set_launch_config(0, 1, dict(saved, warp_windows=0))
        cta = api.align_batch([one(rd), one(clean)], p)
    finally:
        api.set_launch_config(0, 1, saved)
    for i in range(2):
        assert columns.status(i) == cta.status(i)
        assert np.array_equal(columns.pairs(i), cta.pairs(i))
        assert np.array_equal(columns.log_likelihood(i), cta.log_likelihood(i), equal_nan=True)
    assert len(alone.pairs(0)) > 100 and np.array_equal(columns.pairs(1), alone.pairs(0))
