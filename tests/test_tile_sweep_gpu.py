"""The tile sweep's run loop and direction groups at their edges, bit for bit against the oracle: direction
counts below, at and beside the groups of a tile configuration, run lengths with every remainder of the
four-tap blocks (1 to 9 taps), one to sixteen scales, images at and beside the tiles' edges."""
import numpy as np
import pytest

import lpaici
import oracle_bind as ob
from conftest import SYM, kernel_file

pytestmark = pytest.mark.gpu


def random_set(D, S, seed):
    """Dense kernels of D x S: rows of 1 .. 9 taps at random offsets, some rows empty."""
    rng = np.random.default_rng(seed)
    w, off, rows, cols = [], [], [], []
    at = 0
    shapes = [(int(rng.integers(1, 8)), int(rng.integers(9, 14))) for _ in range(S)]
    for _ in range(D):
        for s in range(S):
            r, c = shapes[s]
            h = np.zeros((r, c), np.float32)
            for y in range(r):
                if y != r // 2 and rng.random() < 0.25:
                    continue
                n = int(rng.integers(1, 10))
                x = int(rng.integers(0, c - n + 1))
                h[y, x:x + n] = rng.uniform(0.05, 1.0, n).astype(np.float32)
            h /= h.sum()
            w.append(h.ravel())
            off.append(at)
            rows.append(r)
            cols.append(c)
            at += r * c
    w = np.concatenate(w).astype(np.float32)
    off, rows, cols = (np.array(v, np.int32) for v in (off, rows, cols))
    return (lpaici.KernelSet.from_dense(w, off, rows, cols, D, S), ob.DenseKernels(D, S, w, off, rows, cols))


@pytest.mark.parametrize("config", range(lpaici.lib().lpaici_num_tile_configs()))
@pytest.mark.parametrize("D,S", [(1, 1), (2, 16), (3, 4), (5, 2), (16, 3), (17, 2)])
def test_sweep_edges(config, D, S):
    import torch

    ks, ko = random_set(D, S, 100 * D + S)
    tw, th, _, _ = lpaici.tile_configs()[config]
    ks.set_tile_config(config)
    sigma, gamma = 0.1, 1.7
    var = ks.variances(sigma)
    for W, H in ((1, 1), (tw, th), (tw + 1, th // 2 + 1), (2 * tw - 1, th + 3)):
        rng = np.random.default_rng(W * 1000 + H)
        x = rng.uniform(0.0, 1.0, (H, W)).astype(np.float32)
        out, smap = lpaici.forward(ks, torch.from_numpy(x).cuda(), sigma, gamma, scale_map=True)
        ref, rmap, _ = ob.oracle_forward_f32(x, ko, var, gamma, want_map=True)
        assert np.array_equal(smap.cpu().numpy(), rmap), (W, H)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), ref.view(np.uint32)), (W, H)


def test_non_finite_pixels_reach_the_same_outputs():
    """Infinities and NaNs in the input: every tile configuration gives the same bits (no configuration
    multiplies a pixel by a padding weight)."""
    import torch

    ks, _ = random_set(5, 3, 7)
    rng = np.random.default_rng(3)
    x = rng.uniform(0.0, 1.0, (70, 90)).astype(np.float32)
    for v in (np.inf, -np.inf, np.nan):
        x[rng.integers(0, 70), rng.integers(0, 90)] = v
    t = torch.from_numpy(x).cuda()
    ref = None
    for config in range(lpaici.lib().lpaici_num_tile_configs()):
        ks.set_tile_config(config)
        out, smap = (v.cpu().numpy() for v in lpaici.forward(ks, t, 0.1, 1.7, scale_map=True))
        if ref is None:
            ref = (out, smap)
            reach = ~np.isfinite(out)
            assert reach.any() and not reach.all()
        assert np.array_equal(np.nan_to_num(out, nan=7.5).view(np.uint32),
                              np.nan_to_num(ref[0], nan=7.5).view(np.uint32)), config
        assert np.array_equal(smap, ref[1]), config


@pytest.mark.parametrize("D,S", [(3, 4), (16, 2), (17, 2)])
def test_few_tiles_shared_by_clusters(D, S):
    """Kernels of a few hundred taps on images of a few tiles: clusters of CTAs split the directions, with
    fewer directions than a round takes, as many, and one more."""
    import torch

    rng = np.random.default_rng(D)
    n = 25
    w = rng.uniform(0.0, 1.0, (D * S, n, n)).astype(np.float32)
    w[:, :, 0] = 0.0
    w[rng.random((D * S, n, n)) < 0.1] = 0.0
    w /= w.sum((1, 2), keepdims=True)
    off = np.arange(D * S, dtype=np.int32) * n * n
    rows = np.full(D * S, n, np.int32)
    ks = lpaici.KernelSet.from_dense(w.ravel(), off, rows, rows, D, S)
    ko = ob.DenseKernels(D, S, w.ravel(), off, rows, rows)
    var = ks.variances(0.1)
    for W, H in ((1, 1), (16, 16), (17, 33), (97, 64), (130, 127)):
        x = rng.uniform(0.0, 1.0, (H, W)).astype(np.float32)
        t = torch.from_numpy(x).cuda()
        out, smap = lpaici.forward(ks, t, 0.1, 0.6, scale_map=True)
        ref, rmap, _ = ob.oracle_forward_f32(x, ko, var, 0.6, want_map=True)
        assert np.array_equal(smap.cpu().numpy(), rmap), (W, H)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), ref.view(np.uint32)), (W, H)
        # through a state as well: 1 / den of the same sums
        state_out, _ = lpaici.forward_state(ks, t, 0.1, 0.6)
        assert torch.equal(state_out.view(torch.int32), out.view(torch.int32))


@pytest.mark.parametrize("D,sizes", [(5, (25,)), (18, (9, 25)), (4, (5, 21, 25)), (5, (3, 3, 27, 25, 23)), (16, (21, 9, 3))])
def test_cluster_helpers(D, sizes):
    """The last one or two scales of a direction swept by a second warp: one scale (none to hand over), two,
    the split before the last scale and before the last two, scales that shrink, more than one round of directions,
    and images whose warps partly lie outside."""
    rng = np.random.default_rng(D)
    S = len(sizes)
    rows = np.tile(np.array(sizes, np.int32), D)
    off = (np.cumsum(rows * rows) - rows * rows).astype(np.int32)
    w = []
    for n in rows:
        k = rng.uniform(0.1, 1.0, (n, n)).astype(np.float32)
        w.append((k / k.sum()).ravel())
    w = np.concatenate(w).astype(np.float32)
    ks = lpaici.KernelSet.from_dense(w, off, rows, rows, D, S)
    ko = ob.DenseKernels(D, S, w, off, rows, rows)
    var = ks.variances(0.1)
    for W, H in ((1, 1), (19, 33), (90, 64), (127, 70), (150, 120)):
        x = rng.uniform(0.0, 1.0, (H, W)).astype(np.float32)
        for gamma in (0.4, 3.0):
            out, smap = lpaici.forward(ks, torch_image(x), 0.1, gamma, scale_map=True)
            ref, rmap, _ = ob.oracle_forward_f32(x, ko, var, gamma, want_map=True)
            assert np.array_equal(smap.cpu().numpy(), rmap), (W, H, gamma)
            assert np.array_equal(out.cpu().numpy().view(np.uint32), ref.view(np.uint32)), (W, H, gamma)


def torch_image(x):
    import torch

    return torch.from_numpy(x).cuda()


@pytest.mark.parametrize("W,H", [(200, 150), (180, 190), (592, 64), (16, 2368), (145, 255), (593, 64)])
def test_one_round_per_tile(W, H):
    """Images of up to as many 16 x 16 tiles as there are SMs, ragged ones, and one tile column more."""
    import torch

    ks = lpaici.KernelSet.load(kernel_file(SYM))
    x = torch_image(np.random.default_rng(W).uniform(0.0, 1.0, (H, W)).astype(np.float32))
    out, smap = lpaici.forward(ks, x, 0.08, 2.0, scale_map=True)
    fused = lpaici.forward(ks, x, 0.08, 2.0, ffma=True)
    ks.set_tile_config(0)
    ref, rmap = lpaici.forward(ks, x, 0.08, 2.0, scale_map=True)
    fref = lpaici.forward(ks, x, 0.08, 2.0, ffma=True)
    assert torch.equal(out.view(torch.int32), ref.view(torch.int32)) and torch.equal(smap, rmap)
    assert torch.equal(fused.view(torch.int32), fref.view(torch.int32))
