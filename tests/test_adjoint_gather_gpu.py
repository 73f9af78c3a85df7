"""The adjoint's gather at its edges: direction counts below, at and beside its eight chunks, one to sixteen
scales, kernel rows apart and of every remainder of the four-tap blocks, images at and beside the tiles' edges;
the same gradient however many CTAs a tile gets; infinities and NaNs in the cotangent reach exactly the pixels
whose kernels read them."""
import numpy as np
import pytest

import lpaici
import oracle_bind as ob
from test_tile_sweep_gpu import random_set

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,S", [(1, 1), (2, 16), (3, 4), (8, 2), (16, 3), (17, 2)])
@pytest.mark.parametrize("W,H", [(1, 1), (128, 64), (129, 65), (255, 33), (300, 140)])
def test_gather_edges(D, S, W, H):
    """Against the FP64 adjoint, within the bound the adjoint has everywhere: 2e-5 of the largest gradient."""
    import torch

    ks, ko = random_set(D, S, 100 * D + S)
    sigma, gamma = 0.1, 1.7
    rng = np.random.default_rng(W * 1000 + H)
    x = rng.uniform(0.0, 1.0, (H, W)).astype(np.float32)
    g = rng.standard_normal((H, W)).astype(np.float32)
    got = lpaici.backward(ks, torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda(), sigma, gamma).cpu().numpy()
    var = ks.variances(sigma)
    _, smap, _ = ob.oracle_forward_f32(x, ko, var, gamma, want_map=True)
    ref = ob.oracle_adjoint_f64(ko, var, smap, g.astype(np.float64))
    assert np.abs(got - ref).max() <= 2e-5 * np.abs(ref).max() + 1e-6


def test_same_gradient_however_a_tile_is_split():
    """One image alone (eight or four CTAs per tile) and in plans of more and more images (down to one)."""
    import torch

    ks, _ = random_set(16, 3, 5)
    rng = np.random.default_rng(1)
    x = torch.from_numpy(rng.uniform(0, 1, (200, 300)).astype(np.float32)).cuda()
    g = torch.from_numpy(rng.standard_normal((200, 300)).astype(np.float32)).cuda()
    ref = lpaici.backward(ks, x, g, 0.1, 1.7)
    for n in (2, 3, 8, 14):
        outs = [torch.empty_like(x) for _ in range(n)]
        b = lpaici.BackwardBatch(ks, [x] * n, [g] * n, outs, [0.1] * n, [1.7] * n, use_graph=False)
        b.run()
        for o in outs:
            assert torch.equal(o.view(torch.int32), ref.view(torch.int32)), n
        b.close()


def test_non_finite_cotangents_reach_only_their_kernels():
    import torch

    D, S, R = 5, 3, 7
    ks, ko = random_set(D, S, 7)
    H, W = 90, 150
    rng = np.random.default_rng(9)
    x = torch.from_numpy(rng.uniform(0, 1, (H, W)).astype(np.float32)).cuda()
    g = rng.standard_normal((H, W)).astype(np.float32)
    at = [(int(rng.integers(0, H)), int(rng.integers(0, W))) for _ in range(4)]
    for (y, c), v in zip(at, (np.inf, -np.inf, np.nan, np.inf)):
        g[y, c] = v
    out, state = lpaici.forward_state(ks, x, 0.1, 1.7)
    smap = state[:D * H * W].cpu().numpy().reshape(D, H, W)
    got = lpaici.backward_state(ks, state, torch.from_numpy(g).cuda(), 0.1).cpu().numpy()
    # gradient at q reads source q + t through the telescoped, mirrored kernels D_0 .. D_{s*(source)}, each row
    # from its first to its last nonzero tap: source p reaches p + (tap's offset)
    reach = np.zeros((H + 2 * R, W + 2 * R), bool)
    for d in range(D):
        for s in range(S):
            box = np.zeros((2 * R + 1, 2 * R + 1))
            for q, sign in ((s, 1.0), (s - 1, -1.0)):
                if q >= 0:
                    h = ko.kernel(d, q).astype(np.float64)
                    y0, c0 = R - h.shape[0] // 2, R - h.shape[1] // 2
                    box[y0:y0 + h.shape[0], c0:c0 + h.shape[1]] += sign * h
            box = box.astype(np.float32)
            for y in range(2 * R + 1):
                nz = np.nonzero(box[y])[0]
                if not nz.size:
                    continue
                for py, pc in at:
                    if smap[d, py, pc] >= s:
                        reach[py + y, pc + nz[0]:pc + nz[-1] + 1] = True
    reach = reach[R:R + H, R:R + W]
    assert reach.any() and not reach.all()
    assert np.array_equal(~np.isfinite(got), reach)


@pytest.mark.parametrize("R", [36, 40, 48, 55])
@pytest.mark.parametrize("W,H", [(64, 32), (150, 141), (33, 200)])
def test_gather_of_wide_kernels(R, W, H):
    """Radii past the usual 31: fields of more words than a thread holds, and the 64 x 32 tile."""
    import torch

    D, S, n = 2, 3, 2 * R + 1
    rng = np.random.default_rng(R)
    w = np.zeros((D * S, n, n), np.float32)
    for d in range(D):
        for y in range(n):
            m = int(rng.integers(1, 6))
            x = int(rng.integers(0, n - m + 1))
            w[d * S:(d + 1) * S, y, x:x + m] = rng.uniform(0.05, 1.0, (S, m))  # the scales' rows lie alike
    w /= w.sum((1, 2), keepdims=True)
    off = np.arange(D * S, dtype=np.int32) * n * n
    rows = np.full(D * S, n, np.int32)
    ks = lpaici.KernelSet.from_dense(w.ravel(), off, rows, rows, D, S)
    ko = ob.DenseKernels(D, S, w.ravel(), off, rows, rows)
    x = rng.uniform(0.0, 1.0, (H, W)).astype(np.float32)
    g = rng.standard_normal((H, W)).astype(np.float32)
    got = lpaici.backward(ks, torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda(), 0.1, 1.7).cpu().numpy()
    var = ks.variances(0.1)
    _, smap, _ = ob.oracle_forward_f32(x, ko, var, 1.7, want_map=True)
    ref = ob.oracle_adjoint_f64(ko, var, smap, g.astype(np.float64))
    assert np.abs(got - ref).max() <= 2e-5 * np.abs(ref).max() + 1e-6
