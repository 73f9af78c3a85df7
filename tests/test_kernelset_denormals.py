"""Kernel sets packed on a thread that treats subnormal numbers as zero (torch.set_flush_denormal): rows whose only
nonzero weights are subnormal are rows without taps, as zeros are.  A process of its own, which a wrong scan may end."""
import subprocess
import sys

from conftest import PKG

CODE = """
import sys
sys.path.insert(0, {pkg!r})
import numpy as np, torch, lpaici
rng = np.random.default_rng(0)
w = np.zeros((4, 9, 9), np.float32)
w[:, 2:6, 3:7] = rng.uniform(0.1, 1.0, (4, 4, 4))
zero = w.copy()
w[:, 0, 4] = 1e-40
w[:, 8, :] = -1e-45
w[:, 4, 0] = 1e-41
off = np.arange(4, dtype=np.int32) * 81
n = np.full(4, 9, np.int32)
ref = lpaici.KernelSet.from_dense(zero.ravel(), off, n, n, 2, 2)
keep = lpaici.KernelSet.from_dense(w.ravel(), off, n, n, 2, 2)
if not torch.set_flush_denormal(True):
    print("same")
    sys.exit(0)
got = lpaici.KernelSet.from_dense(w.ravel(), off, n, n, 2, 2)
torch.set_flush_denormal(False)
a, b, k = ref.runs(), got.runs(), keep.runs()
assert all(np.array_equal(getattr(a, f), getattr(b, f)) for f in a.__dataclass_fields__)
assert np.array_equal(ref.nnz(), [16] * 4) and ref.radius == got.radius
assert len(k.run_len) == len(a.run_len) + 8 and keep.radius == 4
print("same")
"""


def test_subnormal_rows_taken_as_zero():
    p = subprocess.run([sys.executable, "-c", CODE.format(pkg=PKG)], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0 and p.stdout.strip() == "same", p.stderr[-2000:]
