"""The plain FP64 form's resident kernels at the edges of what their threads hold (128, 256, 512 and
past it, where the rings take over), with many-path columns (one and two X in a window, two to four
options), the smallest reads, several regions, and expectations; against the FP64 oracle.  Both sides
evaluate the same terms in the same order, so pairs agree to rounding of exp() (posteriors 1e-5 as
the FP64 form's other tests hold it, expectations 1e-9)."""
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


def _pairs(api, m, rd, ref, expansion, degenerate, options, split=3000 * 3000, ragged=(True, True)):
    sm = W.gpu_model(api, m, orc.EMIT_DESCALED, rd)
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=expansion,
                                                         split_matrix_bigger_than_this=split)
    got, ll = api.getAlignedPairsUsingAnchors(sm, ref, rd["events"], rd["anchors"], p, *ragged, degenerate=degenerate,
                                              with_log_likelihood=True)
    want = orc.aligned_pairs(W.oracle_model(m, orc.EMIT_DESCALED, rd), ref, rd["events"], rd["anchors"],
                             orc.params(threshold=p.threshold, expansion=expansion, split=split), *ragged,
                             options=options)
    assert len(got) == len(want) and len(want) > 0
    for f in ("x", "y", "kmer"):   # the reference's order
        assert np.array_equal(got[f], want[f]), f
    assert np.abs(got["score"] - want["score"]).max() <= 1e7 * 1e-5


@pytest.mark.parametrize("expansion", [2, 50, 60, 62, 64, 100, 124, 128, 200, 252, 256, 300])
def test_threads(api, expansion):
    cfg = synth.config1(seed=170 + expansion, n_reads=1, span=(500, 700))
    rd = cfg["reads"][0]
    _pairs(api, W.gaussian_model(cfg), rd, rd["reference"], expansion, api.CYTOSINE_METHYLATION3, "CEO")


@pytest.mark.parametrize("degenerate,options,expansion", [("CYTOSINE_METHYLATION2", "CE", 20), ("CYTOSINE_METHYLATION2", "CE", 50),
                                                          ("CYTOSINE_METHYLATION3", "CEO", 50), ("CANONICAL_VARIANTS", "ACGT", 50),
                                                          ("CYTOSINE_METHYLATION2", "CE", 120)])
def test_paths(api, degenerate, options, expansion):
    alphabet = "".join(sorted(set("ACGT" + options)))
    table = synth.gaussian_table(alphabet, 4, 77)
    r = np.random.Generator(np.random.PCG64(expansion))
    seq = synth.random_reference(420, r)
    rd = synth.make_read(seq, alphabet, 4, table[:, 0], table[:, 1], table[:, 2], table[:, 3], r)
    ref = list(seq)
    # at both ends, alone, next to one another and two columns apart
    for i in (0, 40, 41, 90, 92, 200, 419):
        ref[i] = "X"
    m = W.gaussian_model(dict(alphabet=alphabet, k=4, table=table))
    _pairs(api, m, rd, "".join(ref), expansion, getattr(api, degenerate), options)


def test_regions_and_smallest(api):
    cfg = synth.config1(seed=301, n_reads=1, span=(900, 900))
    rd, m = cfg["reads"][0], W.gaussian_model(cfg)
    gap = dict(rd, anchors=np.concatenate([rd["anchors"][:4], rd["anchors"][12:]]))
    _pairs(api, m, gap, rd["reference"], 20, api.CYTOSINE_METHYLATION3, "CEO", split=200 * 200)
    _pairs(api, m, rd, rd["reference"], 50, api.CYTOSINE_METHYLATION3, "CEO", ragged=(False, False))
    for k, e in ((6, 4), (7, 2), (9, 9), (40, 50), (130, 220)):
        small = dict(rd, events=rd["events"][:e], anchors=np.zeros((0, 2), np.int64))
        _pairs(api, m, small, rd["reference"][:k], 50, api.CYTOSINE_METHYLATION3, "CEO", ragged=(False, False))


@pytest.mark.parametrize("expansion,repeat", [(20, False), (50, True), (240, False), (300, False)])
def test_expectations(api, expansion, repeat):
    """repeat: one k-mer in long runs, so that its columns share anti-diagonals"""
    cfg = synth.config1(seed=311, n_reads=1, span=(800, 800))
    table, m = cfg["table"], W.gaussian_model(cfg)
    rd = cfg["reads"][0]
    if repeat:
        r = np.random.Generator(np.random.PCG64(3))
        seq = synth.random_reference(300, r) + "A" * 60 + synth.random_reference(200, r) + "AC" * 40
        rd = synth.make_read(seq, "ACGT", 6, table[:, 0], table[:, 1], table[:, 2], table[:, 3], r)
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=expansion)
    got = api.getExpectationsUsingAnchors(W.gpu_model(api, m, orc.EMIT_DESCALED, rd), rd["reference"], rd["events"],
                                          rd["anchors"], p)
    want = orc.expectations(W.oracle_model(m, orc.EMIT_DESCALED, rd), rd["reference"], rd["events"], rd["anchors"],
                            orc.params(threshold=p.threshold, expansion=expansion))
    assert got["likelihood"] == pytest.approx(want["likelihood"], rel=1e-12)
    np.testing.assert_allclose(got["transitions"], want["transitions"], rtol=1e-9)
    np.testing.assert_allclose(got["posteriors"], want["posteriors"], rtol=1e-9)
    np.testing.assert_allclose(got["event_expectations"], want["event_expectations"], rtol=1e-9, atol=1e-9)
    assert np.array_equal(got["observed"], want["observed"])


_NO_ROOM = """
import numpy as np, torch
from signalalign_b200 import api, synth
import workloads as W
from oracle import oracle as orc
cfg = synth.config1(seed=321, n_reads=1, span=(20000, 20000))
rd, m = cfg["reads"][0], W.gaussian_model(cfg)
sm = W.gpu_model(api, m, orc.EMIT_DESCALED, rd)
p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=50)
def call(bases, events):
    before = api.kernel_launch_count()
    anchors = rd["anchors"][(rd["anchors"][:, 0] < bases - 9) & (rd["anchors"][:, 1] < events - 3)]
    got = api.getAlignedPairsUsingAnchors(sm, rd["reference"][:bases], rd["events"][:events], anchors, p)
    return got, api.kernel_launch_count() - before
def expect():
    return api.getExpectationsUsingAnchors(sm, rd["reference"], rd["events"], rd["anchors"], p)
api.set_segment_policy(-1, 1024)           # one ring a read
call(400, 600)                             # the machine's tables
free = torch.cuda.mem_get_info()[0]
held = torch.empty(free - (100 << 20), dtype=torch.uint8, device="cuda")
(rings, few), e_rings = call(20000, len(rd["events"])), expect()
del held
torch.cuda.empty_cache()
(resident, more), e_resident = call(20000, len(rd["events"])), expect()
assert few < more, (few, more)
assert len(rings) == len(resident) > 10000
for f in ("x", "y", "kmer"):
    assert np.array_equal(rings[f], resident[f]), f
assert np.abs(rings["score"] - resident["score"]).max() <= 100     # posteriors 1e-5
np.testing.assert_allclose(e_rings["transitions"], e_resident["transitions"], rtol=1e-6)
print("ok", few, more)
"""


def test_no_room_for_the_store(api):
    """A device without room for the resident store (256 MB for this read) runs the rings, in a process
    of its own: blocks that other calls left for reuse would be room."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([root, os.path.join(root, "tests")]))
    got = subprocess.run([sys.executable, "-c", _NO_ROOM], env=env, capture_output=True, text=True, timeout=600)
    assert got.returncode == 0 and got.stdout.startswith("ok"), got.stdout + got.stderr
