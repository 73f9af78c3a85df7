"""The adjoint of kernel sets whose neighbouring rows hardly overlap: rows apart, every other row, single rows and lines,
of every length up to eighteen and on odd and even rows, one direction to more than the gather's chunks, images at and
beside the tiles' edges.  Against the FP64 adjoint within the bound the adjoint has everywhere, 2e-5 of the largest
gradient; the same bits however a tile is split; infinities and NaNs reach exactly the pixels whose kernels read them."""
import numpy as np
import pytest

import lpaici
import oracle_bind as ob

SIGMA, GAMMA = 0.1, 1.7


def make(w, D, S):
    """w: D * S square kernels of one odd size; a kernel without taps stays empty."""
    n = w.shape[1]
    w = (w / np.maximum(w.sum((1, 2), keepdims=True), 1e-9)).astype(np.float32)
    off = np.arange(D * S, dtype=np.int32) * n * n
    rows = np.full(D * S, n, np.int32)
    return lpaici.KernelSet.from_dense(w.ravel(), off, rows, rows, D, S), ob.DenseKernels(D, S, w.ravel(), off, rows, rows)


def apart(D, S, n, longest, seed):
    """Row y: one run of 1 .. longest taps, left of the row before or right of it."""
    rng = np.random.default_rng(seed)
    w = np.zeros((D * S, n, n))
    for d in range(D):
        for y in range(n):
            m = int(rng.integers(1, min(longest, n // 2) + 1))
            x = int(rng.integers(0, n // 2 - m + 1)) + (n // 2 + 1) * (y % 2)
            w[d * S:(d + 1) * S, y, x:x + m] = rng.uniform(0.1, 1.0, (S, m))
    for k in range(D * S):  # scale s has the rows within its share of the radius
        r = max(1, n // 2 * (k % S + 1) // S)
        w[k, :n // 2 - r] = w[k, n // 2 + r + 1:] = 0.0
    return make(w, D, S)


def other_rows(D, S, n, odd, seed):
    w = np.random.default_rng(seed).uniform(0.1, 1.0, (D * S, n, n))
    w[:, 1 - odd::2] = 0.0
    return make(w, D, S)


def row_lengths():
    """One row of 1 .. 18 taps a direction, on odd and even rows, at both ends."""
    n, w = 37, np.zeros((18, 37, 37))
    for d in range(18):
        a = 0 if d % 4 < 2 else n - d - 1
        w[d, 17 + d % 3, a:a + d + 1] = np.arange(1, d + 2)
    return make(w, 18, 1)


SETS = {
    "one_direction": lambda: apart(1, 1, 33, 9, 1),
    "three_scales": lambda: apart(3, 3, 41, 20, 2),
    "seventeen": lambda: apart(17, 2, 21, 6, 3),
    "radius47": lambda: apart(4, 2, 95, 20, 4),   # 128 x 32 tiles
    "radius55": lambda: apart(2, 3, 111, 5, 5),   # 64 x 32 tiles
    "even_rows": lambda: other_rows(2, 2, 31, 0, 6),
    "odd_rows": lambda: other_rows(9, 1, 31, 1, 7),
    "row_lengths": row_lengths,
}


@pytest.mark.parametrize("name", SETS)
def test_a_tap_is_stored_once(name):
    """The blob is no larger than a weight per tap twice over and 16 bytes a run, as the support limit counts it."""
    ks, _ = SETS[name]()
    n = ks.runs()
    if ks.S == 1:
        words = ((ks.D + 1 + 3) & ~3) + 4 * len(n.run_len) + 2 * (16 + int(((n.run_len + 1) & ~1).sum()))
        assert ks.info.adjoint_blob_bytes <= 4 * ((words + 3) & ~3)
    else:  # telescoped rows span both scales' runs
        words = 4 * 2 * len(n.run_len) + 2 * 2 * 2 * int(((n.run_len + 1) & ~1).sum()) + 64 + 2 * ks.D * ks.S
        assert ks.info.adjoint_blob_bytes <= 4 * words


def inputs(W, H):
    import torch

    rng = np.random.default_rng(W * 1000 + H)
    x = rng.uniform(0.0, 1.0, (H, W)).astype(np.float32)
    g = rng.standard_normal((H, W)).astype(np.float32)
    return x, g, torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda()


@pytest.mark.gpu
@pytest.mark.parametrize("name", SETS)
@pytest.mark.parametrize("W,H", [(1, 1), (64, 32), (129, 65), (255, 33), (300, 140)])
def test_against_fp64(name, W, H):
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


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["seventeen", "radius47"])
def test_same_gradient_however_a_tile_is_split(name):
    import torch

    ks, _ = SETS[name]()
    _, _, x, g = inputs(300, 200)
    ref = lpaici.backward(ks, x, g, SIGMA, GAMMA)
    for n in (2, 3, 8, 14):
        outs = [torch.empty_like(x) for _ in range(n)]
        b = lpaici.BackwardBatch(ks, [x] * n, [g] * n, outs, [SIGMA] * n, [GAMMA] * n, use_graph=False)
        b.run()
        for o in outs:
            assert torch.equal(o.view(torch.int32), ref.view(torch.int32)), n
        b.close()


@pytest.mark.gpu
def test_non_finite_cotangents_reach_only_their_kernels():
    """One scale: the cotangent at p reaches p + t for the kernel's taps t, each row from its first to its last."""
    import torch

    ks, ko = SETS["odd_rows"]()
    _, _, x, g = inputs(150, 90)
    at = [(10, 20), (44, 45), (60, 149)]
    for (r, c), v in zip(at, (float("inf"), float("nan"), float("-inf"))):
        g[r, c] = v
    got = lpaici.backward(ks, x, g, SIGMA, GAMMA)
    R = 15
    reach = torch.zeros(90 + 2 * R, 150 + 2 * R, dtype=torch.bool, device="cuda")
    taps = torch.from_numpy(np.any([ko.kernel(d, 0) != 0 for d in range(9)], axis=0)).cuda()
    for r, c in at:
        reach[r:r + 2 * R + 1, c:c + 2 * R + 1] |= taps
    reach = reach[R:R + 90, R:R + 150]
    assert reach.any() and not reach.all()
    assert torch.equal(~torch.isfinite(got), reach)
