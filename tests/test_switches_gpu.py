"""Environment switches that keep a call on one of its kernels: what they name runs, also for the batches that stream
their codes otherwise."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

WORKER = r"""
import sys
import numpy as np
import torch
import __graft_entry__
qx = __graft_entry__.load_package()
m, n, k = int(sys.argv[1]), 2048, 1024
rng = np.random.Generator(np.random.Philox(key=[m, n]))
codes = rng.integers(-127, 128, (n, k), dtype=np.int8)
scales = rng.uniform(0.002, 0.03, n).astype(np.float32)
weights = qx.CanonicalWeights()
view = qx.canonical_view(qx.INT8_SYMMETRIC, qx.SCALE_CHANNEL, n, k, k, codes.view(np.uint8).reshape(-1), scales)
assert weights.prepare(view) == qx.OK, qx.last_error()
x = rng.standard_normal((m, k)).astype(np.float32)
before = qx.launch_count()
y = torch.zeros((m, n), device="cuda")
assert weights.qgemm_storage_dev(torch.from_numpy(x).cuda(), qx.F32, y, qx.F32, m) == qx.OK, qx.last_error()
launches = qx.launch_count() - before
exact = (x.astype(np.float64) @ codes.astype(np.float64).T) * scales
assert np.all(np.abs(y.cpu().numpy() - exact) <= 4e-5 * (1 + np.abs(exact)))
print("launches", launches)
"""


# two launches: streamed (or one of the digit kernels below the threshold); three: digit planes, their GEMM and the sums
@pytest.mark.parametrize("m,switch,value,launches", [
    (4, None, None, 2), (8, None, None, 2), (16, None, None, 2),
    (5, "QX_B200_CANONICAL_PREFILL_TOKENS", "5", 3),
    (16, "QX_B200_CANONICAL_PREFILL_TOKENS", "9", 3),
    (8, "QX_B200_CANONICAL_PREFILL_TOKENS", "9", 2),
    (4, "QX_B200_CANONICAL_PREFILL_TOKENS", "2", 3),
    (8, "QX_B200_INT8_GEMM_VARIANT", "dp4a", 3),
    (16, "QX_B200_INT8_GEMM_VARIANT", "dp4a", 3),
    (4, "QX_B200_INT8_GEMM_VARIANT", "dp4a", 2),
])
def test_canonical_int8(m, switch, value, launches):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = {k: v for k, v in os.environ.items() if not k.startswith("QX_B200_")}
    env["PYTHONPATH"] = root
    if switch:
        env[switch] = value
    done = subprocess.run([sys.executable, "-c", WORKER, str(m)], cwd=root, env=env, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stdout + done.stderr
    assert f"launches {launches}" in done.stdout.split("\n"), done.stdout
