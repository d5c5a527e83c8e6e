"""The plain FP64 form's two routes at the line between them: bands whose paths (those of any three consecutive
anti-diagonals, and a path's neighbours past them) are just what 128, 256 or 480 threads hold, and one more;
past 480 (256 where columns have several paths) the rings run.  The route is read off the launches: eight for
pairs on the resident route, one on the rings.  Against the FP64 oracle, pairs to the last unit of their
scores but for the rounding of exp() (1), expectations to 1e-9 as the form's other tests hold them."""
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


def threads_needed(rd, reference, k, expansion, n_options):
    """paths from the first to the last of any three consecutive anti-diagonals, and twice a column's"""
    lX = len(reference) - (k - 1)
    per = np.array([1] + [n_options ** reference[x:x + k].count("X") for x in range(lX)])
    first = np.concatenate([[0], np.cumsum(per)])
    L, R = orc.band(rd["anchors"], lX, len(rd["events"]), expansion)
    d = np.arange(len(L))
    lo, hi = first[(d + L) // 2], first[(d + R) // 2 + 1]
    lo3 = np.minimum(np.minimum(lo[:-2], lo[1:-1]), lo[2:])
    hi3 = np.maximum(np.maximum(hi[:-2], hi[1:-1]), hi[2:])
    return int((hi3 - lo3).max() + 2 * per.max())


def plain_read(threads, bases=1000):
    """(config, read, expansion) of a single-path band that needs that many threads"""
    for seed in range(70, 100):
        cfg = synth.config1(seed=seed, n_reads=1, span=(bases, bases))
        rd = cfg["reads"][0]
        first = max(2, threads - 64 - threads % 2)
        for expansion in range(first, first + 24, 2):
            if threads_needed(rd, rd["reference"], 6, expansion, 1) == threads:
                return cfg, rd, expansion
    raise AssertionError("no read that needs %d threads" % threads)


def path_read(threads):
    """the same with X sites, C or E: a 4-mer read whose sites are chosen for it"""
    table = synth.gaussian_table("ACEGT", 4, 77)
    for seed in range(200):
        r = np.random.Generator(np.random.PCG64(seed))
        rd = synth.make_read(synth.random_reference(420, r), "ACEGT", 4, table[:, 0], table[:, 1], table[:, 2], table[:, 3], r)
        ref = list(rd["reference"])
        for i in (0, 40, 41, 90, 92, 200 + seed % 7, 419):
            ref[i] = "X"
        ref = "".join(ref)
        for expansion in range(20, 300, 2):
            need = threads_needed(rd, ref, 4, expansion, 2)
            if need == threads:
                return dict(alphabet="ACEGT", k=4, table=table), dict(rd, reference=ref), expansion
            if need > threads + 8:
                break
    raise AssertionError("no read that needs %d threads" % threads)


def _pairs(api, cfg, rd, expansion, degenerate, options, resident):
    m = W.gaussian_model(cfg)
    sm = W.gpu_model(api, m, orc.EMIT_DESCALED, rd)
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=expansion)
    call = lambda: api.getAlignedPairsUsingAnchors(sm, rd["reference"], rd["events"], rd["anchors"], p,
                                                   degenerate=degenerate, with_log_likelihood=True)
    call()   # the machine's tables
    before = api.kernel_launch_count()
    got, ll = call()
    assert api.kernel_launch_count() - before == (8 if resident else 1)
    want, totals = orc.aligned_pairs(W.oracle_model(m, orc.EMIT_DESCALED, rd), rd["reference"], rd["events"],
                                     rd["anchors"], orc.params(threshold=p.threshold, expansion=expansion), True, True,
                                     options=options, with_total_probs=True)
    assert len(got) == len(want) > 100
    for f in ("x", "y", "kmer"):
        assert np.array_equal(got[f], want[f]), f
    assert np.abs(got["score"] - want["score"]).max() <= 1
    total = dict(totals)[len(rd["reference"]) - (cfg["k"] - 1) + len(rd["events"])]
    assert ll == pytest.approx(total, rel=1e-12)


@pytest.mark.parametrize("threads", [127, 128, 129, 255, 256, 257, 479, 480, 481, 640])
def test_pairs(api, threads):
    cfg, rd, expansion = plain_read(threads)
    _pairs(api, cfg, rd, expansion, api.CYTOSINE_METHYLATION3, "CEO", threads <= 480)


@pytest.mark.parametrize("threads", [127, 128, 129, 255, 256, 257])
def test_pairs_with_paths(api, threads):
    cfg, rd, expansion = path_read(threads)
    _pairs(api, cfg, rd, expansion, api.CYTOSINE_METHYLATION2, "CE", threads <= 256)


@pytest.mark.parametrize("expansion,resident", [(50, True), (150, True), (400, True), (500, False)])
def test_expectations(api, expansion, resident):
    """of a read in several regions, so that its accumulators go from one to the next"""
    cfg = synth.config1(seed=74, n_reads=1, span=(2200, 2200))
    rd = cfg["reads"][0]
    a = np.asarray(rd["anchors"]).reshape(-1, 2)
    rd = dict(rd, anchors=a[(a[:, 0] < 1000) | (a[:, 0] > 1200)])
    m = W.gaussian_model(cfg)
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=expansion,
                                                         split_matrix_bigger_than_this=120 * 120)
    assert len(orc.split_points(rd["anchors"], len(rd["reference"]) - 5, len(rd["events"]), 120 * 120, True, True)) > 1
    sm = W.gpu_model(api, m, orc.EMIT_DESCALED, rd)
    call = lambda: api.getExpectationsUsingAnchors(sm, rd["reference"], rd["events"], rd["anchors"], p)
    call()   # the machine's tables
    before = api.kernel_launch_count()
    got = call()
    assert api.kernel_launch_count() - before == (7 if resident else 1)
    want = orc.expectations(W.oracle_model(m, orc.EMIT_DESCALED, rd), rd["reference"], rd["events"], rd["anchors"],
                            orc.params(threshold=p.threshold, expansion=expansion, split=120 * 120))
    assert got["likelihood"] == pytest.approx(want["likelihood"], rel=1e-12)
    np.testing.assert_allclose(got["transitions"], want["transitions"], rtol=1e-9)
    np.testing.assert_allclose(got["posteriors"], want["posteriors"], rtol=1e-9)
    np.testing.assert_allclose(got["event_expectations"], want["event_expectations"], rtol=1e-9, atol=1e-9)
    assert np.array_equal(got["observed"], want["observed"])


@pytest.mark.parametrize("expansion", [20, 100, 400, 500])
def test_expectations_hdp(api, expansion):
    """20, 100 and 400: the resident route; 500: the rings"""
    hc = W.small_hdp_config(span=(600, 700), n_reads=2)
    hdp = W.hdp_dict(hc["hdp"], len(hc["alphabet"]) ** hc["k"])
    m = formats.parse_model_lines(*synth.model_text(hc["alphabet"], hc["k"], hc["table"]).split("\n")[:3])
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=expansion)
    for rd in hc["reads"]:
        need = threads_needed(rd, rd["reference"], hc["k"], expansion, 1)
        assert (need <= 480) == (expansion <= 400), need
        got = api.getExpectationsUsingAnchors(W.gpu_model(api, m, orc.EMIT_HDP, rd, hdp), rd["reference"], rd["events"],
                                              rd["anchors"], p)
        want = orc.expectations(W.oracle_model(m, orc.EMIT_HDP, rd, hdp), rd["reference"], rd["events"], rd["anchors"],
                                orc.params(threshold=p.threshold, expansion=expansion))
        assert got["likelihood"] == pytest.approx(want["likelihood"], rel=1e-9)
        np.testing.assert_allclose(got["transitions"], want["transitions"], rtol=1e-8, atol=1e-12)
        assert len(want["assignments"]) > 500 and np.array_equal(got["assignments"], want["assignments"])


def test_rerun_regions_of_several_reads(api, policy):
    """A resident set of several reads, some regions of which run again whole: reads without a stitch, reads
    of one region with stitches, and a read whose second region has some and whose first has none.  Every
    stitch disagrees (negative tolerance); the results are those of whole sweeps."""
    cfg = synth.config3(seed=69, n_reads=4, span=(6000, 6500), grid_length=50, route="degenerate")
    m = formats.parse_model_lines(*synth.model_text("ACEGT", 6, cfg["gauss_table"]).split("\n")[:3])
    sm = W.gpu_model(api, m, orc.EMIT_DESCALED)
    reads = [a for a in cfg["alignments"] if a["model"] == "gauss"][:3]
    a = np.asarray(reads[1]["anchors"]).reshape(-1, 2)
    reads[1] = dict(reads[1], anchors=a[(a[:, 0] < 900) | (a[:, 0] > 1100)])      # two regions: short and long
    L = 1200                                                                      # and a short read
    n = int(np.searchsorted(reads[2]["true_pos"], L - 5))
    b = np.asarray(reads[2]["anchors"]).reshape(-1, 2)
    short = dict(reads[2], reference=reads[2]["reference"][:L], events=reads[2]["events"][:n],
                 anchors=b[(b[:, 0] < L - 12) & (b[:, 1] < n - 8)])
    inputs = [api.ReadInput(sm=sm, reference=rd["reference"], events=rd["events"], anchors=rd["anchors"],
                            scale=rd["scale"], shift=rd["shift"], degenerate=api.CYTOSINE_METHYLATION2)
              for rd in (reads[0], short, reads[1], short, reads[2])]
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=50, split_matrix_bigger_than_this=130 * 130)

    def run(segment_diags, tolerance=None):
        api.set_segment_policy(segment_diags, 1024)
        batch = api.Batch(inputs, p)
        batch.upload()
        if tolerance is not None:
            batch.set_stitch_tolerance(tolerance)
        batch.run()
        batch.download()
        return batch

    whole, forced = run(-1), run(4096, -1.0)
    assert whole.segment_info()["segments"] == 6
    info = forced.segment_info()
    assert info["redone"] == 3 and info["stitches"] >= 6, info
    for i in range(len(inputs)):
        assert forced.status(i) == 0 and len(whole.pairs(i)) > 100
        assert np.array_equal(forced.pairs(i), whole.pairs(i))
        assert forced.log_likelihood(i) == whole.log_likelihood(i)
