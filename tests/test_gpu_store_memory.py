"""Device memory of the plain FP64 form, in processes of their own (blocks that other calls left for reuse would
count): a batch uploaded again keeps the blocks it has."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_SETUP = """
import numpy as np, torch
from oracle import formats, oracle as orc
from signalalign_b200 import api, synth
import workloads as W
GB = 1 << 30
free = lambda: torch.cuda.mem_get_info()[0]
cfg = synth.config3(seed=68, n_reads=1, span=(SPAN, SPAN), grid_length=50, route="degenerate")
rd = [a for a in cfg["alignments"] if a["model"] == "gauss"][0]
m = formats.parse_model_lines(*synth.model_text("ACEGT", 6, cfg["gauss_table"]).split("\\n")[:3])
sm = W.gpu_model(api, m, orc.EMIT_DESCALED)
p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=50)
def inputs(n):
    return [api.ReadInput(sm=sm, reference=rd["reference"], events=rd["events"], anchors=rd["anchors"],
                          scale=rd["scale"], shift=rd["shift"], degenerate=api.CYTOSINE_METHYLATION2)] * n
"""

_AGAIN = _SETUP.replace("SPAN", "3000") + """
b = api.Batch(inputs(4), p)
b.upload(); b.run(); b.download()
want = b.pairs(3)
count, room = api.allocation_count(), free()
for _ in range(4):
    b.upload(); b.run(); b.download()
    assert len(want) > 1000 and np.array_equal(b.pairs(3), want)
assert api.allocation_count() == count and free() == room, (api.allocation_count(), count)
print("ok")
"""


def _run(text):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([root, os.path.join(root, "tests")]))
    got = subprocess.run([sys.executable, "-c", text], env=env, capture_output=True, text=True, timeout=600)
    assert got.returncode == 0 and got.stdout.startswith("ok"), got.stdout + got.stderr


def test_upload_again():
    _run(_AGAIN)
