"""Launches that mix two tile configurations (whole waves of big tiles, the rest in small ones) against one
configuration forced over the whole image, bit for bit: single images with scale maps, row bands, interleaved
channels, one-size and mixed-size plans, the adjoint's selection pass and the host-pointer engine.  The sizes
are around one to three waves of 128 x 64 and of 64 x 32 tiles, with ragged right and bottom strips."""
import numpy as np
import pytest

import lpaici
from conftest import SMALL, SYM, kernel_file

pytestmark = pytest.mark.gpu

SIGMA, GAMMA = 0.08, 2.0


def forced(ks, config, f):
    ks.set_tile_config(config)
    try:
        return f()
    finally:
        ks.set_tile_config(-1)


def image(W, H, seed=0):
    import torch

    g = torch.Generator("cuda")
    g.manual_seed(W * 8192 + H + seed)
    return torch.rand(H, W, device="cuda", generator=g)


@pytest.mark.parametrize("kernels", [SYM, SMALL])
@pytest.mark.parametrize("W,H", [(600, 601), (640, 640), (777, 333), (1281, 833), (1535, 1021), (129, 2100), (2049, 127)])
def test_mixed_equals_one_configuration(kernels, W, H):
    import torch

    ks = lpaici.KernelSet.load(kernel_file(kernels))
    x = image(W, H)
    out, smap = lpaici.forward(ks, x, SIGMA, GAMMA, scale_map=True)
    ref, rmap = forced(ks, 0, lambda: lpaici.forward(ks, x, SIGMA, GAMMA, scale_map=True))
    assert torch.equal(out.view(torch.int32), ref.view(torch.int32)) and torch.equal(smap, rmap)
    fused = lpaici.forward(ks, x, SIGMA, GAMMA, ffma=True)
    fref = forced(ks, 0, lambda: lpaici.forward(ks, x, SIGMA, GAMMA, ffma=True))
    assert torch.equal(fused.view(torch.int32), fref.view(torch.int32))
    r0, n = H // 5, H - H // 3
    band = lpaici.forward_rows(ks, x, r0, n, SIGMA, GAMMA)
    bref = forced(ks, 0, lambda: lpaici.forward_rows(ks, x, r0, n, SIGMA, GAMMA))
    assert torch.equal(band.view(torch.int32), bref.view(torch.int32))
    host = lpaici.denoise_host(ks, x.cpu().numpy(), SIGMA, GAMMA)
    assert np.array_equal(host.view(np.uint32), ref.cpu().numpy().view(np.uint32))


@pytest.mark.parametrize("W,H,C", [(300, 257, 3), (768, 513, 3), (129, 65, 4), (700, 200, 2)])
def test_channels_in_one_launch(W, H, C):
    import torch

    ks = lpaici.KernelSet.load(kernel_file(SYM))
    x = torch.stack([image(W, H, c) for c in range(C)], 2).contiguous()
    pad = torch.full((H, W + 3, C), 7.0, device="cuda")[:, :W]
    out = lpaici.forward_channels(ks, x, SIGMA, GAMMA)
    lpaici.forward_channels(ks, x, SIGMA, GAMMA, out=pad)
    assert torch.equal(out, pad)
    for c in range(C):
        ref = lpaici.forward(ks, x[:, :, c].contiguous(), SIGMA, GAMMA)
        assert torch.equal(out[:, :, c].contiguous().view(torch.int32), ref.view(torch.int32)), c


@pytest.mark.parametrize("sizes", [[(640, 640)] * 3, [(512, 300)] * 9, [(900, 700), (333, 801), (512, 512), (129, 65), (1000, 17)]])
def test_plans_mix(sizes):
    import torch

    ks = lpaici.KernelSet.load(kernel_file(SYM))
    one = len(set(sizes)) == 1
    sig = [SIGMA if one else SIGMA + 0.01 * i for i in range(len(sizes))]
    xs = [image(w, h, i) for i, (w, h) in enumerate(sizes)]
    outs = [torch.empty_like(x) for x in xs]
    b = lpaici.Batch(ks, xs, outs, sig, [GAMMA] * len(xs))
    b.run()
    for x, o, s in zip(xs, outs, sig):
        ref = forced(ks, 0, lambda: lpaici.forward(ks, x, s, GAMMA))
        assert torch.equal(o.view(torch.int32), ref.view(torch.int32)), tuple(x.shape)
    b.close()
    gs = [image(w, h, 50 + i) for i, (w, h) in enumerate(sizes)]
    gi = [torch.empty_like(x) for x in xs]
    bb = lpaici.BackwardBatch(ks, xs, gs, gi, sig, [GAMMA] * len(xs))
    bb.run()
    for x, g, o, s in zip(xs, gs, gi, sig):
        ref = forced(ks, 0, lambda: lpaici.backward(ks, x, g, s, GAMMA))
        assert torch.equal(o.view(torch.int32), ref.view(torch.int32)), tuple(x.shape)
    bb.close()
