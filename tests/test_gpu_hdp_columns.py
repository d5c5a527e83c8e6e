"""HDP emissions a group of 64 columns at a time: bands within a group, past it and past the staged means,
grids of an odd and an even number of knots, k-mers without a row, a machine's own scaling, and a batch
that mixes HDP and Gaussian machines; against the FP64 oracle.

Tolerance: the FP32 arithmetic's 1e-4, and one jump of the reference's logAdd.  At its cut-off its value
drops by the cubic's excess over the argument, h = 4.5e-4, and FP32 arithmetic (differences good to about
1e-5) can find itself on the other side of the cut-off than FP64 in a cell of a pair's path; that moves the
cell's logarithm by h and the posterior by at most h.  The pairs themselves (those that differ by more than
the tolerance from the threshold on either side) have to be the same.  These inputs give 1.2e-4 and less
than 1.4e-4, bit for bit the same with the emissions computed a cell at a time."""
import numpy as np
import pytest

from oracle import formats
from oracle import oracle as orc
from signalalign_b200 import synth
import workloads as W

pytestmark = pytest.mark.gpu
# the cubic's last piece at the cut-off of 7.5, less 7.5
CUTOFF_JUMP = ((-0.000458661602210 * 7.5 + 0.009695946122598) * 7.5 + 0.930734667215156) * 7.5 + 0.168037164329057 - 7.5
FP32_TOL = 1e-4 + CUTOFF_JUMP


@pytest.fixture(scope="module")
def api():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from signalalign_b200 import api as a
    return a


@pytest.mark.parametrize("expansion,grid_length", [(4, 200), (20, 201), (60, 200), (64, 333), (130, 200), (190, 151),
                                                   (240, 201)])
def test_widths(api, expansion, grid_length):
    cfg = W.small_hdp_config(seed=expansion, n_reads=3, span=(300, 700), grid_length=grid_length)
    n = len(cfg["alphabet"]) ** cfg["k"]
    hdp = W.hdp_dict(cfg["hdp"], n)
    hdp["kmer_row"][::17] = -1
    m = formats.parse_model_lines(*synth.model_text(cfg["alphabet"], cfg["k"], cfg["table"]).split("\n")[:3])
    gauss = W.gpu_model(api, m, orc.EMIT_DESCALED)
    mixed = W.gpu_model(api, m, orc.EMIT_HDP, None, hdp)
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=expansion)
    kinds = [orc.EMIT_HDP, orc.EMIT_DESCALED, orc.EMIT_HDP]
    b = api.align_batch([api.ReadInput(sm=mixed if k == orc.EMIT_HDP else gauss, reference=rd["reference"],
                                       events=rd["events"], anchors=rd["anchors"], scale=rd["scale"],
                                       shift=rd["shift"], var=v)
                         for rd, k, v in zip(cfg["reads"], kinds, (1.0, 1.0, 1.1))], p)
    for i, (rd, kind, var) in enumerate(zip(cfg["reads"], kinds, (1.0, 1.0, 1.1))):
        assert b.status(i) == 0
        om = W.oracle_model(m, kind, dict(rd, var=var), hdp if kind == orc.EMIT_HDP else None)
        want = orc.aligned_pairs(om, rd["reference"], rd["events"], rd["anchors"],
                                 orc.params(threshold=p.threshold, expansion=expansion), True, True)
        assert len(want) > 0
        assert W.max_posterior_error(want, b.pairs(i), p.threshold) <= FP32_TOL
