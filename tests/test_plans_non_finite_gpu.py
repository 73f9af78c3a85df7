"""Infinities and NaNs in the input through every kind of plan (clusters of four, two and one CTAs with and without helper
warps, mixes, grid layers, queues, channels, bands): the same output bits and scale maps as one configuration gives, so
that they reach the same outputs."""
import numpy as np
import pytest

import lpaici
from conftest import SYM, kernel_file

pytestmark = pytest.mark.gpu

SIGMA, GAMMA = 0.08, 2.0


def image(W, H, seed):
    """Eight non-finite pixels, at the corners and beside the borders of 16-, 32- and 64-pixel tiles."""
    x = np.random.default_rng(W * 4096 + H + seed).uniform(0.0, 1.0, (H, W)).astype(np.float32)
    at = [(0, 0), (H - 1, W - 1), (0, W - 1), (15, 16), (H // 2, 31), (31, W // 2), (min(64, H - 1), min(63, W - 1)), (H // 3, W // 3)]
    for (r, c), v in zip(at, (np.inf, np.nan, -np.inf, np.inf, -np.inf, np.nan, np.inf, np.nan)):
        x[r, c] = v
    return x


def same(a, b):
    """Equal bits, any NaN equal to any other."""
    a, b = (v.cpu().numpy() if hasattr(v, "cpu") else v for v in (a, b))
    return np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(
        np.where(np.isnan(a), 0, a.view(np.uint32)), np.where(np.isnan(b), 0, b.view(np.uint32)))


def one_configuration():
    ks = lpaici.KernelSet.load(kernel_file(SYM))
    ks.set_tile_config(0)
    return ks


@pytest.mark.parametrize("W,H", [(60, 33), (97, 64), (128, 128), (150, 120), (200, 150), (512, 300), (1024, 700)])
@pytest.mark.parametrize("ffma", [False, True])
def test_one_image(W, H, ffma):
    import torch

    ks, ref = lpaici.KernelSet.load(kernel_file(SYM)), one_configuration()
    x = image(W, H, 0)
    t = torch.from_numpy(x).cuda()
    out, smap = lpaici.forward(ks, t, SIGMA, GAMMA, scale_map=True, ffma=ffma)
    want, wmap = lpaici.forward(ref, t, SIGMA, GAMMA, scale_map=True, ffma=ffma)
    reach = ~torch.isfinite(want)
    assert reach.any() and (W < 200 or not reach.all())
    assert same(out, want) and torch.equal(smap, wmap)
    if not ffma:
        assert same(lpaici.denoise_host(ks, x, SIGMA, GAMMA), want)
        state = lpaici.forward_state(ks, t, SIGMA, GAMMA)[0]
        assert same(state, want)
        # the adjoint's selection: of a finite cotangent and the pixels that see no such value
        grad = lpaici.backward(ks, t, torch.ones_like(t), SIGMA, GAMMA)
        assert same(grad, lpaici.backward(ref, t, torch.ones_like(t), SIGMA, GAMMA))


@pytest.mark.parametrize("sizes", [[(97, 64)] * 3, [(512, 300)] * 5, [(97, 64), (300, 200), (33, 150)], [(700, 500), (130, 90)]])
def test_several_images(sizes):
    import torch

    ks, ref = lpaici.KernelSet.load(kernel_file(SYM)), one_configuration()
    xs = [torch.from_numpy(image(W, H, i)).cuda() for i, (W, H) in enumerate(sizes)]
    for out, x in zip(lpaici.forward_batched(ks, xs, [SIGMA] * len(xs), [GAMMA] * len(xs)), xs):
        assert same(out, lpaici.forward(ref, x, SIGMA, GAMMA))
    if len(set(sizes)) == 1:
        got = lpaici.forward_channels(ks, torch.stack(xs, dim=2).contiguous(), SIGMA, GAMMA)
        for c, x in enumerate(xs):
            assert same(got[:, :, c].contiguous(), lpaici.forward(ref, x, SIGMA, GAMMA))
