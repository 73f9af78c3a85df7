"""Plans and host arrays of one image of a few tiles, which clusters sweep, with kernel sets that the largest tile
configuration does not fit: every entry point takes what lpaici_forward and lpaici_backward take, bit for bit."""
import numpy as np
import pytest

import lpaici

pytestmark = pytest.mark.gpu

SIGMA, GAMMA = 0.08, 2.0
# (directions, scales): radius 39 of sixteen directions, radius 47 of eight
WIDE = [(16, (1, 2, 4, 8, 16, 24, 40)), (8, (1, 48))]


def bits(t):
    import torch

    return t.view(torch.int32)


def image(W, H, seed=0):
    import torch

    g = torch.Generator("cuda")
    g.manual_seed(W * 8192 + H + seed)
    return torch.rand(H, W, device="cuda", generator=g)


@pytest.mark.parametrize("D,scales", WIDE)
@pytest.mark.parametrize("W,H", [(64, 64), (97, 64), (150, 120), (200, 150)])
@pytest.mark.parametrize("use_graph", [False, True])
def test_plan_of_one_small_image(D, scales, W, H, use_graph):
    import torch

    ks = lpaici.KernelSet.generate(D, list(scales), 1)
    x, g = image(W, H), image(W, H, 1)
    out, grad = torch.empty_like(x), torch.empty_like(x)
    plan = lpaici.Batch(ks, [x], [out], [SIGMA], [GAMMA], use_graph=use_graph)
    plan.run()
    assert torch.equal(bits(out), bits(lpaici.forward(ks, x, SIGMA, GAMMA)))
    plan.close()
    plan = lpaici.BackwardBatch(ks, [x], [g], [grad], [SIGMA], [GAMMA], use_graph=use_graph)
    plan.run()
    assert torch.equal(bits(grad), bits(lpaici.backward(ks, x, g, SIGMA, GAMMA)))
    plan.close()
    assert torch.equal(bits(lpaici.forward_batched(ks, [x], [SIGMA], [GAMMA])[0]), bits(out))


def test_forced_configuration_that_does_not_fit_is_refused():
    ks = lpaici.KernelSet.generate(16, list(WIDE[0][1]), 1)
    x = image(64, 64)
    with pytest.raises(lpaici.LpaIciError) as e:
        lpaici.Batch(ks, [x], [image(64, 64, 2)], [SIGMA], [GAMMA], tile_config=0)
    assert e.value.code == lpaici.ERR_UNSUPPORTED


@pytest.mark.parametrize("D,scales", WIDE + [(16, (1, 2, 4, 8, 16, 24, 32))])
@pytest.mark.parametrize("W,H", [(96, 193), (110, 200), (128, 256), (150, 200), (64, 500), (16, 2000)])
def test_host_array_of_a_few_tiles(D, scales, W, H):
    """Taller than three rows of the largest tile, where larger images are cut into bands."""
    ks = lpaici.KernelSet.generate(D, list(scales), 1)
    x = image(W, H, 3)
    ref = lpaici.forward(ks, x, SIGMA, GAMMA).cpu().numpy()
    got = lpaici.denoise_host(ks, x.cpu().numpy(), SIGMA, GAMMA)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("D,scales", [(8, (1,)), (8, (1, 2, 4, 8)), (16, (1, 2, 4, 8, 16, 24, 32))])
@pytest.mark.parametrize("W,H", [(200, 150), (275, 273), (390, 400), (1100, 130), (700, 500), (40, 9000), (900, 901), (1200, 1000),
                                 (1500, 1000), (1, 100000)])
def test_host_array_of_every_number_of_bands(D, scales, W, H):
    """One to six bands, with one configuration and with mixes."""
    ks = lpaici.KernelSet.generate(D, list(scales), 1)
    x = image(W, H, 4)
    ref = lpaici.forward(ks, x, SIGMA, GAMMA).cpu().numpy()
    got = lpaici.denoise_host(ks, x.cpu().numpy(), SIGMA, GAMMA)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))


def small_and_large_sets():
    return (lpaici.KernelSet.generate(16, [1, 2, 4, 8, 16, 24, 32], 1), lpaici.KernelSet.generate(8, [1, 2, 4], 1))


def test_plans_of_a_large_and_a_small_set_in_turn():
    """A plan keeps working after another set's plans, launches and adjoints have used the same kernels with less
    shared memory."""
    import torch

    sets = small_and_large_sets()
    xs = [image(300, 200), image(150, 260, 1), image(64, 64, 2)]
    gs = [image(300, 200, 5), image(150, 260, 6), image(64, 64, 7)]
    sig = [SIGMA, SIGMA + 0.01, SIGMA]
    for config in (-1, 0, 4):
        plans = []
        for ks in sets:
            outs, grads = [torch.empty_like(x) for x in xs], [torch.empty_like(x) for x in xs]
            plans.append((ks, outs, grads, lpaici.Batch(ks, xs, outs, sig, [GAMMA] * 3, use_graph=False, tile_config=config),
                          lpaici.BackwardBatch(ks, xs, gs, grads, sig, [GAMMA] * 3, use_graph=False, tile_config=config)))
        for _ in range(2):
            for ks, outs, grads, fwd, bwd in plans:
                fwd.run()
                bwd.run()
                for x, g, s, o, d in zip(xs, gs, sig, outs, grads):
                    assert torch.equal(bits(o), bits(lpaici.forward(ks, x, s, GAMMA)))
                    assert torch.equal(bits(d), bits(lpaici.backward(ks, x, g, s, GAMMA)))
        for _, _, _, fwd, bwd in plans:
            fwd.close()
            bwd.close()


def test_threads_with_a_large_and_a_small_set():
    """Two host threads launch the same kernels with different sets, each on a stream of its own."""
    import threading

    import torch

    x = image(128, 128)
    sets = small_and_large_sets()
    refs = []
    for ks in sets:
        ks.set_tile_config(3)
        refs.append(lpaici.forward(ks, x, SIGMA, GAMMA))
    torch.cuda.synchronize()
    wrong = []

    def work(ks, ref):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(300):
                    out = lpaici.forward(ks, x, SIGMA, GAMMA)
                torch.cuda.current_stream().synchronize()
                if not torch.equal(bits(out), bits(ref)):
                    wrong.append("bits")
        except lpaici.LpaIciError as e:
            wrong.append(str(e))

    threads = [threading.Thread(target=work, args=a) for a in zip(sets, refs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong


def set_filling_shared_memory(spare):
    """28 kernels of radius 31 whose set leaves `spare` bytes of an SM's 232,448 beside the 128 x 64 tile: rows of eight
    taps, the last ones of four (a row is a group of 16 bytes and one per four taps, a bit of the mask per group)."""
    D, S, n = 7, 4, 63
    tile = ((128 + 62 + 8) | 1) * (32 + 62) * 8
    words = (232448 - spare - tile) // 4 - ((3 * D * S + 3) & ~3) - ((D * S + 4) & ~3)
    groups = words // 4
    while groups + (((groups + 31) // 32 + 3) // 4) > words // 4:
        groups -= 1
    rows = (groups + 2) // 3
    short = 3 * rows - groups
    assert rows <= D * S * n
    w = np.zeros((D * S, n, n), np.float32)
    for r in range(rows):
        w[r // n, r % n, (r * 7) % 40:(r * 7) % 40 + (4 if r >= rows - short else 8)] = 1.0 + r % 5
    w /= np.maximum(w.sum((1, 2), keepdims=True), 1e-6)  # (the last kernel may be empty)
    off = np.arange(D * S, dtype=np.int32) * n * n
    rows_ = np.full(D * S, n, np.int32)
    return lpaici.KernelSet.from_dense(w.ravel(), off, rows_, rows_, D, S)


@pytest.mark.parametrize("spare", [0, 16, 32, 48, 64, 80, 96, 128, 144])
def test_tile_that_leaves_no_room_for_the_image_arguments(spare):
    """Plans of several images keep their arguments in static shared memory beside the tile."""
    import torch

    ks = set_filling_shared_memory(spare)
    xs = [image(900, 640), image(700, 500, 1)]
    outs = [torch.empty_like(x) for x in xs]
    plan = lpaici.Batch(ks, xs, outs, [SIGMA, SIGMA], [GAMMA, GAMMA], use_graph=False)
    plan.run()
    one = [torch.empty_like(xs[0]) for _ in range(3)]
    same = lpaici.Batch(ks, [xs[0]] * 3, one, [SIGMA] * 3, [GAMMA] * 3, use_graph=False)
    same.run()
    ks.set_tile_config(7)
    for x, o in zip(xs + [xs[0]], outs + [one[2]]):
        assert torch.equal(bits(o), bits(lpaici.forward(ks, x, SIGMA, GAMMA)))
    plan.close()
    same.close()


def check_rows(ks, x, out):
    """out against bands of x: its first and last rows, and those around the 65,535th 16-, 32- and 64-row tile."""
    import torch

    H, R = x.shape[0], ks.radius
    for at in (0, H - 100, 16 * 65535 - 50, 32 * 65535 - 50, 64 * 65535 - 50):
        if not 0 <= at <= H - 100:
            continue
        lo, hi = max(0, at - R), min(H, at + 100 + R)
        ref = lpaici.forward_rows(ks, x[lo:hi], at - lo, 100, SIGMA, GAMMA)
        assert torch.equal(bits(out[at:at + 100]), bits(ref)), at


@pytest.mark.parametrize("W,H", [(1, 1048561), (5, 1048700), (16, 2097121), (33, 2100000), (64, 4194241), (3, 8388480)])
def test_images_of_more_tile_rows_than_a_grid(W, H):
    import torch

    ks = lpaici.KernelSet.generate(8, [1, 2, 4], 1)
    x = image(W, H)
    check_rows(ks, x, lpaici.forward(ks, x, SIGMA, GAMMA))
    if W * H < 40_000_000:
        outs = [torch.empty_like(x) for _ in range(3)]
        xs = [x, image(W, H, 1), image(W, H, 2)]
        plan = lpaici.Batch(ks, xs, outs, [SIGMA] * 3, [GAMMA] * 3)
        plan.run()
        for a, o in zip(xs, outs):
            check_rows(ks, a, o)
        plan.close()
    ks.set_tile_config(6)
    check_rows(ks, x, lpaici.forward(ks, x, SIGMA, GAMMA))


def test_images_past_the_tallest_are_refused():
    ks = lpaici.KernelSet.generate(8, [1, 2, 4], 1)
    with pytest.raises(lpaici.LpaIciError) as e:
        lpaici.forward(ks, image(1, 8388481), SIGMA, GAMMA)
    assert e.value.code == lpaici.ERR_UNSUPPORTED and "too tall" in str(e.value)
