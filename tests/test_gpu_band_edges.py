"""Bands at the edges of what the kernels' threads hold.  A band's span is the number of columns from the
first to the last of any three consecutive anti-diagonals; the reads here are chosen by it (anchors
every 50 positions, one of several seeds, an expansion), and the span is checked.

FP32: 128, 256 or 512 threads hold spans of up to their number; of the last two, whose band's ends lie on
neighbouring threads, with sweeps of their own.  Every case, in a batch with a narrow read and cut
into forward segments, against the FP64 oracle (posteriors 1e-4, log-likelihood 1e-3 relative, the FP32
form's bounds) and against the CTA form, whose values the column-resident form has bit for bit."""
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


def band_span(rd, expansion, k=6):
    L, R = orc.band(rd["anchors"], len(rd["reference"]) - (k - 1), len(rd["events"]), expansion)
    d = np.arange(len(L))
    lo, hi = (d + L) // 2, (d + R) // 2
    lo3 = np.minimum(np.minimum(lo[:-2], lo[1:-1]), lo[2:])
    hi3 = np.maximum(np.maximum(hi[:-2], hi[1:-1]), hi[2:])
    return int((hi3 - lo3).max()) + 1


def read_of_span(span, bases):
    """(config, read, expansion) of a band that spans `span` columns"""
    for seed in range(70, 100):
        cfg = synth.config1(seed=seed, n_reads=1, span=(bases, bases))
        rd = cfg["reads"][0]
        first = max(2, span - 64 - span % 2)
        for expansion in range(first, first + 24, 2):
            if band_span(rd, expansion) == span:
                return cfg, rd, expansion
    raise AssertionError("no read of span %d" % span)


def _input(api, sm, rd):
    return api.ReadInput(sm=sm, reference=rd["reference"], events=rd["events"], anchors=rd["anchors"],
                         scale=rd["scale"], shift=rd["shift"])


def _width_class(rd, expansion, k=6):
    L, R = orc.band(rd["anchors"], len(rd["reference"]) - (k - 1), len(rd["events"]), expansion)
    w = int(((R - L) // 2).max()) + 1
    return 1 if w <= 128 else (2 if w <= 256 else 4)


@pytest.mark.parametrize("span", [125, 126, 127, 128, 129, 175, 176, 177, 178, 253, 254, 255, 256, 257, 300, 400,
                                  509, 510, 511, 512])
def test_fp32(api, span):
    cfg, rd, expansion = read_of_span(span, 3400 if span < 260 else 6400)
    m = W.gaussian_model(cfg)
    sm = W.gpu_model(api, m, orc.EMIT_DESCALED)
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=expansion)
    wide = _input(api, sm, rd)
    # a short narrow read beside it: one batch of both
    other = synth.config1(seed=1, n_reads=1, span=(300, 300))["reads"][0]
    inputs = [wide, _input(api, sm, other)]
    op = orc.params(threshold=p.threshold, expansion=expansion)
    wants = [orc.aligned_pairs(W.oracle_model(m, orc.EMIT_DESCALED, r), r["reference"], r["events"], r["anchors"], op,
                               True, True, with_total_probs=True) for r in (rd, other)]
    cls = _width_class(rd, expansion)
    saved, policy = api.get_launch_config(0, cls), api.get_segment_policy()
    try:
        api.set_segment_policy(0 if span < 260 else 8000, 1024)
        api.set_launch_config(0, cls, dict(saved, warp_windows=1))
        columns = api.align_batch(inputs, p)
        api.set_launch_config(0, cls, dict(saved, warp_windows=0))
        cta = api.align_batch(inputs, p)
    finally:
        api.set_launch_config(0, cls, saved)
        api.set_segment_policy(*policy)
    info = columns.segment_info()
    assert info["stitches"] > 0 and info["redone"] == 0, info
    for i, (want, totals) in enumerate(wants):
        assert columns.status(i) == 0 and len(want) > 100
        assert W.max_posterior_error(want, columns.pairs(i), p.threshold) <= 1e-4
        total = dict(totals)[len((rd, other)[i]["reference"]) - 5 + len((rd, other)[i]["events"])]
        assert abs(columns.log_likelihood(i) - total) <= 1e-3 * abs(total)
        assert np.array_equal(columns.pairs(i), cta.pairs(i))
        assert columns.log_likelihood(i) == cta.log_likelihood(i)


@pytest.mark.parametrize("span", [127, 128, 256])
@pytest.mark.parametrize("finite_sx,skips", [(True, False), (False, True), (True, True)])
def test_fp32_machines(api, span, finite_sx, skips):
    """a finite SWITCH_TO_X and skip emissions that differ between k-mers, ends not ragged"""
    cfg, rd, expansion = read_of_span(span, 1300)
    m = dict(W.gaussian_model(cfg))
    m["t"] = np.array(m["t"], dtype=np.float64)
    if finite_sx:
        m["t"][7] = m["t"][8] = -3.0
    if skips:
        m["gapx"] = np.log(np.random.Generator(np.random.PCG64(5)).uniform(0.02, 0.3, m["n_kmers"]))
    inp = _input(api, W.gpu_model(api, m, orc.EMIT_DESCALED), rd)
    inp.ragged_left = inp.ragged_right = False
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=expansion)
    want = orc.aligned_pairs(W.oracle_model(m, orc.EMIT_DESCALED, rd), rd["reference"], rd["events"], rd["anchors"],
                             orc.params(threshold=p.threshold, expansion=expansion), False, False)
    cls = _width_class(rd, expansion)
    saved = api.get_launch_config(0, cls)
    try:
        api.set_launch_config(0, cls, dict(saved, warp_windows=1))
        columns = api.align_batch([inp], p)
        api.set_launch_config(0, cls, dict(saved, warp_windows=0))
        cta = api.align_batch([inp], p)
    finally:
        api.set_launch_config(0, cls, saved)
    assert columns.status(0) == 0 and len(want) > 100
    assert W.max_posterior_error(want, columns.pairs(0), p.threshold) <= 1e-4
    assert np.array_equal(columns.pairs(0), cta.pairs(0))
    assert columns.log_likelihood(0) == cta.log_likelihood(0)
