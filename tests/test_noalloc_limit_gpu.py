"""lpaici_backward_noalloc's largest image counts the mirrored kernels as their support limit does, a run as 16 bytes and
a tap as 8, whatever layout the gather reads: kernel sets whose neighbouring rows do not overlap, or hardly do, keep the
image sizes that they always had."""
import ctypes as C

import numpy as np
import pytest

import lpaici

SIGMA, GAMMA = 0.1, 1.7
SCRATCH_BYTES = 64 << 20  # LPAICI_NOALLOC_SCRATCH_BYTES
W, D = 200, 8


def kernel_set(overlap):
    """One scale, 63 x 63: each row a run of up to eight taps, of which at most the last lies beside the row before."""
    n, rng = 63, np.random.default_rng(3)
    w = np.zeros((D, n, n), np.float32)
    for d in range(D):
        x = 0
        for y in range(n):
            m = int(rng.integers(2, 9))
            w[d, y, x:x + m] = rng.uniform(0.1, 1.0, m)
            x += m - overlap
            if x + 9 > n:
                x = 0
    w /= w.sum((1, 2), keepdims=True)
    off = np.arange(D, dtype=np.int32) * n * n
    rows = np.full(D, n, np.int32)
    return lpaici.KernelSet.from_dense(w.ravel(), off, rows, rows, D, 1)


def r256(n):
    return (n + 255) & ~255


def need(ks, H):
    """One scale: the telescoped kernels have the kernels' own runs."""
    lens = ks.runs().run_len
    words = ((D + 1 + 3) & ~3) + 4 * len(lens) + 2 * (16 + int(((lens + 1) & ~1).sum()))
    return r256(ks.info.blob_bytes) + r256(4 * ((words + 3) & ~3)) + r256(D * W * H) + 4 * W * H


def largest_rows(ks):
    H = SCRATCH_BYTES // (D + 4) // W
    while need(ks, H) > SCRATCH_BYTES:
        H -= 1
    return H


@pytest.mark.parametrize("overlap", [0, 1, 2])
def test_size_limit(overlap):
    import torch

    ks = kernel_set(overlap)
    fn, fake, H = lpaici.lib().lpaici_backward_noalloc, C.c_void_p(256), largest_rows(ks)
    assert fn(ks.handle, fake, W, fake, W, fake, W, W, H + 1, SIGMA, GAMMA, None) == lpaici.ERR_UNSUPPORTED
    assert f"needs {need(ks, H + 1)} bytes" in lpaici.lib().lpaici_last_error().decode()
    if not torch.cuda.is_available():  # accepted: stops at the first CUDA call
        assert fn(ks.handle, fake, W, fake, W, fake, W, W, H, SIGMA, GAMMA, None) not in (lpaici.OK, lpaici.ERR_UNSUPPORTED)


@pytest.mark.gpu
@pytest.mark.parametrize("overlap", [0, 1, 2])
def test_largest_image(overlap):
    import torch

    ks = kernel_set(overlap)
    H = largest_rows(ks)
    gen = torch.Generator("cuda")
    gen.manual_seed(H)
    x, g = torch.rand(H, W, device="cuda", generator=gen), torch.randn(H, W, device="cuda", generator=gen)
    out = torch.full((H, W), float("nan"), device="cuda")
    rc = lpaici.lib().lpaici_backward_noalloc(ks.handle, x.data_ptr(), W, g.data_ptr(), W, out.data_ptr(), W, W, H, SIGMA, GAMMA,
                                              C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == lpaici.OK
    assert torch.equal(out.view(torch.int32), lpaici.backward(ks, x, g, SIGMA, GAMMA).view(torch.int32))
