"""The adjoint of kernel sets near its support limit whose largest kernel does not fit shared memory twice: one or two
directions of a few thousand taps, dense and with rows that hardly overlap.  Against the FP64 adjoint within the bound
the adjoint has everywhere, 2e-5 of the largest gradient; plans, kept states and the static scratch give the same bits."""
import ctypes as C

import numpy as np
import pytest

import lpaici
import oracle_bind as ob

pytestmark = pytest.mark.gpu

SIGMA, GAMMA = 0.1, 1.7


def make(kernels, D, S):
    """kernels: D * S square arrays of one odd size."""
    n = kernels[0].shape[0]
    w = np.stack([k / k.sum() for k in kernels]).astype(np.float32)
    off = np.arange(D * S, dtype=np.int32) * n * n
    rows = np.full(D * S, n, np.int32)
    return lpaici.KernelSet.from_dense(w.ravel(), off, rows, rows, D, S), ob.DenseKernels(D, S, w.ravel(), off, rows, rows)


def dense(n, m, seed):
    """n x n with random taps in the middle m x m."""
    k = np.zeros((n, n))
    a = (n - m) // 2
    k[a:a + m, a:a + m] = np.random.default_rng(seed).uniform(0.1, 1.0, (m, m))
    return k


def halves(n, seed):
    """Rows of half the width, left and right in turn."""
    k = np.random.default_rng(seed).uniform(0.1, 1.0, (n, n))
    k[0::2, (n + 1) // 2:] = 0.0
    k[1::2, :n // 2] = 0.0
    return k


SETS = {
    "dense89": lambda: make([dense(89, 89, 0)], 1, 1),
    "dense95": lambda: make([dense(95, 95, 1)], 1, 1),
    "dense91_three_scales": lambda: make([dense(91, m, 2 + m) for m in (1, 15, 91)], 1, 3),
    "dense89_two_scales": lambda: make([dense(89, m, 2 + m) for m in (33, 89)], 1, 2),
    "halves95_two_directions": lambda: make([halves(95, 5), halves(95, 6)], 2, 1),
    "halves105": lambda: make([halves(105, 7)], 1, 1),
}


def inputs(W, H):
    import torch

    rng = np.random.default_rng(W * 1000 + H)
    x = rng.uniform(0.0, 1.0, (H, W)).astype(np.float32)
    g = rng.standard_normal((H, W)).astype(np.float32)
    return x, g, torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda()


@pytest.mark.parametrize("name", SETS)
@pytest.mark.parametrize("W,H", [(1, 1), (64, 32), (150, 141), (33, 200)])
def test_adjoint_near_its_limit(name, W, H):
    import torch

    ks, ko = SETS[name]()
    x, g, xt, gt = inputs(W, H)
    got = lpaici.backward(ks, xt, gt, SIGMA, GAMMA)
    var = ks.variances(SIGMA)
    _, smap, _ = ob.oracle_forward_f32(x, ko, var, GAMMA, want_map=True)
    ref = ob.oracle_adjoint_f64(ko, var, smap, g.astype(np.float64))
    assert np.abs(got.cpu().numpy() - ref).max() <= 2e-5 * np.abs(ref).max() + 1e-6
    _, state = lpaici.forward_state(ks, xt, SIGMA, GAMMA)
    assert torch.equal(lpaici.backward_state(ks, state, gt, SIGMA), got)
    outs = [torch.empty_like(xt) for _ in range(2)]
    plan = lpaici.BackwardBatch(ks, [xt, xt], [gt, gt], outs, [SIGMA] * 2, [GAMMA] * 2)
    plan.run()
    assert torch.equal(outs[0], got) and torch.equal(outs[1], got)
    plan.close()
    out = torch.empty_like(xt)
    rc = lpaici.lib().lpaici_backward_noalloc(ks.handle, xt.data_ptr(), W, gt.data_ptr(), W, out.data_ptr(), W, W, H, SIGMA, GAMMA,
                                              C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == lpaici.OK and torch.equal(out, got)


def test_infinite_cotangent_near_the_limit():
    """The single dense kernel: exactly the pixels within its reach see the infinity."""
    import torch

    ks, _ = SETS["dense89"]()
    x, g, xt, gt = inputs(200, 150)
    gt[70, 90] = float("inf")
    got = lpaici.backward(ks, xt, gt, SIGMA, GAMMA)
    reach = torch.zeros_like(got, dtype=torch.bool)
    reach[70 - 44:70 + 45, 90 - 44:90 + 45] = True
    assert torch.equal(~torch.isfinite(got), reach)
