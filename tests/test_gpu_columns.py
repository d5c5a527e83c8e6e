"""The column-resident FP32 kernels where they can go wrong: bands at the edge of what 128 slots hold
(and past it, where the CTA kernels take over), the smallest references and event lists, a finite
SWITCH_TO_X and skip emissions that differ between k-mers; against the FP64 oracle at the FP32 form's
tolerance (posteriors 1e-4, log-likelihood 1e-3 relative)."""
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


def _check(api, m, reads, expansion, ragged=(True, True)):
    sm = W.gpu_model(api, m, orc.EMIT_DESCALED)
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=expansion)
    b = api.align_batch([api.ReadInput(sm=sm, reference=rd["reference"], events=rd["events"], anchors=rd["anchors"],
                                       scale=rd["scale"], shift=rd["shift"], ragged_left=ragged[0],
                                       ragged_right=ragged[1]) for rd in reads], p)
    op = orc.params(threshold=p.threshold, expansion=expansion)
    for i, rd in enumerate(reads):
        want, totals = orc.aligned_pairs(W.oracle_model(m, orc.EMIT_DESCALED, rd), rd["reference"], rd["events"],
                                         rd["anchors"], op, *ragged, with_total_probs=True)
        assert b.status(i) == 0
        assert W.max_posterior_error(want, b.pairs(i), p.threshold) <= 1e-4
        # the reference's order: per window descending anti-diagonals, ascending x on each
        key = [(int(r["x"]), int(r["y"]), int(r["kmer"])) for r in b.pairs(i)]
        both = set(key) & {(int(r["x"]), int(r["y"]), int(r["kmer"])) for r in want}
        assert [k for k in key if k in both] == [k for k in ((int(r["x"]), int(r["y"]), int(r["kmer"]))
                                                             for r in want) if k in both]


@pytest.mark.parametrize("expansion", [2, 20, 50, 58, 60, 62, 64, 100, 122, 126, 200])
def test_band_widths(api, expansion):
    cfg = synth.config1(seed=70 + expansion, n_reads=2, span=(700, 1400))
    _check(api, W.gaussian_model(cfg), cfg["reads"], expansion)


@pytest.mark.parametrize("finite_sx,skips", [(True, False), (False, True), (True, True)])
def test_machines(api, finite_sx, skips):
    cfg = synth.config1(seed=91, n_reads=2, span=(900, 1300))
    m = dict(W.gaussian_model(cfg))
    m["t"] = np.array(m["t"], dtype=np.float64)
    if finite_sx:
        m["t"][7] = m["t"][8] = -3.0   # SWITCH_TO_X, SWITCH_TO_Y
    if skips:
        m["gapx"] = np.log(np.random.Generator(np.random.PCG64(5)).uniform(0.02, 0.3, m["n_kmers"]))
    _check(api, m, cfg["reads"], 50)
    _check(api, m, cfg["reads"], 20, (False, False))


def test_smallest_reads(api):
    cfg = synth.config1(seed=95, n_reads=1, span=(400, 400))
    rd = cfg["reads"][0]
    reads = []
    for k, e in ((6, 1), (6, 4), (7, 1), (9, 3), (12, 9), (40, 60), (132, 5), (7, 150), (140, 210)):
        reads.append(dict(rd, reference=rd["reference"][:k], events=rd["events"][:e], anchors=np.zeros((0, 2), np.int64)))
    _check(api, W.gaussian_model(cfg), reads, 50)
    _check(api, W.gaussian_model(cfg), reads, 2)
