"""Device memory of the plain FP64 form's resident store, in processes of their own (blocks that other calls
left for reuse would count): a store past 4 GiB takes what it needs and at most half of what is free, at most
16 GiB of stores lie idle after a call, and a batch uploaded again keeps the blocks it has."""
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

# the store of a read of 20 kb takes 0.25 GiB
_CALL = _SETUP.replace("SPAN", "20000") + """
def call(n):
    before = api.kernel_launch_count()
    b = api.align_batch(inputs(n), p)
    return b, api.kernel_launch_count() - before
api.set_segment_policy(4096, 1024)                               # every read cut alike
call(1)                                                          # the machine's tables
one, many = call(1)
want, ll = one.pairs(0), one.log_likelihood(0)
assert len(want) > 10000
del one
torch.zeros(1, device="cuda")
start = free()
"""

_KEPT = _CALL + """
b, n = call(20)
used = start - free()
assert n == many and 4.5 * GB < used < 6 * GB, (n, many, used)   # not the next power of two
assert np.array_equal(b.pairs(19), want) and b.log_likelihood(19) == ll
b, n = call(70)
assert n == many and start - free() > 17 * GB
assert np.array_equal(b.pairs(69), want)
del b
assert start - free() < 16.1 * GB, start - free()                # the larger one given back
print("ok")
"""

_HALF = _CALL + """
held = torch.empty(free() - 9 * GB, dtype=torch.uint8, device="cuda")   # it would fit, but not into half
b, n = call(20)
assert n < many, (n, many)                                       # the rings
assert free() > 4.5 * GB, free()
for i in (0, 19):
    assert b.status(i) == 0 and np.array_equal(b.pairs(i), want)
print("ok")
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


def test_idle_stores():
    _run(_KEPT)


def test_half_of_what_is_free():
    _run(_HALF)


def test_upload_again():
    _run(_AGAIN)
