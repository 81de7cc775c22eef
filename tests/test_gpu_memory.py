"""Device memory after calls that leave nothing behind, in processes that do not prove (a
proof keeps its blocks in the pool): a commit plan's is back when the plan is closed, a large
transform's when the call returns, a small one's after the next synchronization."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import sys
import numpy as np, torch
from zs_b200 import native
rng = np.random.default_rng(1)

def transform(cols, log_n):
    native.circle_fft(rng.integers(0, 2**31 - 1, (cols, 1 << log_n), dtype=np.uint32))

def plan(cols, log_rows, log_blowup, folds):
    p = native.CommitPlan(cols, log_rows, log_blowup, folds)
    p.set_challenges(rng.integers(0, 2**31 - 1, (cols, 4), dtype=np.uint32),
                     rng.integers(0, 2**31 - 1, (folds, 4), dtype=np.uint32))
    p.upload(rng.integers(0, 2**31 - 1, (cols, 1 << log_rows), dtype=np.uint32))
    p.run()
    p.results()
    p.close()

for warm in (lambda: transform(1, 10), lambda: transform(1, 14), lambda: plan(2, 8, 1, 4), lambda: plan(2, 15, 2, 4)):
    warm()  # the kernels' code comes to the device
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
{call}
if {sync}:
    torch.cuda.synchronize()
kept = (free - torch.cuda.mem_get_info()[0]) >> 20
assert kept <= 8, f"{{kept}} MB kept"
"""


@pytest.mark.parametrize("call,sync", [("transform(4, 20)", True), ("transform(1, 22)", True), ("transform(6, 20)", False),
                                       ("plan(37, 15, 3, 12)", False), ("plan(8, 18, 2, 16)", False)])
def test_memory_is_given_back(call, sync):
    env = {**os.environ, "PYTHONPATH": os.path.join(ROOT, "zig-stark_b200")}
    out = subprocess.run([sys.executable, "-c", SCRIPT.format(call=call, sync=sync)], env=env, capture_output=True,
                         text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]


PINNED = """
import numpy as np, torch
from zs_b200 import native

def pinned():  # the driver's pinned blocks are shared memory
    return next(line.split()[1] for line in open("/proc/self/status") if line.startswith("RssShmem"))

p = native.CommitPlan(8, 10, 2, 6)
p.set_challenges(np.ones((8, 4), dtype=np.uint32), np.ones((6, 4), dtype=np.uint32))
p.upload(np.ones((8, 1 << 10), dtype=np.uint32))
p.run()
torch.cuda.synchronize()
before = pinned()
{call}
assert pinned() == before, f"{{before}} -> {{pinned()}} kB"
"""


@pytest.mark.parametrize("call", ["p.results()", "native.circle_fft(np.ones((4, 1 << 18), dtype=np.uint32))",
                                  "native.binius_prove_combination(8, bytes(3 << 12), 12, 3, [([0, 1, 2], 1)])"])
def test_no_pinned_memory_stays(call):
    env = {**os.environ, "PYTHONPATH": os.path.join(ROOT, "zig-stark_b200")}
    out = subprocess.run([sys.executable, "-c", PINNED.format(call=call)], env=env, capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
