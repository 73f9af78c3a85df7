"""Performance cases of the LPA-ICI denoiser: the calls a program makes through the package's public
entry points, from a thumbnail to the 4096^2 benchmark image, forward and adjoint, single images, plans,
interleaved channels and host buffers.

A case is a dict: "op" names the entry point, "kernels" the kernel set (the fixtures under
tests/golden/kernels/taps), width and height in pixels, sigma in units of 1/255, gamma, and what the
entry point needs beside these.
"""
import math
import os
import sys

import numpy as np
import torch
import torch.nn.functional as F

sys.path.insert(0, os.path.join(os.getcwd(), "lpa-ici-cuda_b200"))
import lpaici  # noqa: E402

TAPS = os.path.join(os.getcwd(), "tests", "golden", "kernels", "taps")
KERNELS = {
    # the default set: 16 directions, 7 scales up to 32 pixels, uniform windows, order 1
    "sym": "lpa_kernels_m_1_0_d_16_h12_1_2_4_8_16_24_32_symmetric.taps",
    # the gaussian order-2 set of the large forward + adjoint configuration
    "gauss": "lpa_kernels_m_2_0_d_16_h12_1_2_4_8_16_24_32_gaussian.taps",
    # the small set: 8 directions, 4 scales up to 8 pixels
    "small": "lpa_kernels_m_1_0_d_8_h12_1_2_4_8.taps",
    # the tapered set, the one with the most taps but one
    "tapered": "lpa_kernels_python_16_tapered.taps",
}


def listed():
    return [
        # a patch cut out for one crop of a training loop, or a thumbnail: the smallest calls in earnest
        {"name": "patch", "op": "forward", "kernels": "sym", "width": 97, "height": 64, "sigma": 20.0, "gamma": 2.0},
        # the photograph size that the reference publishes its times for, command-line defaults
        {"name": "photo512", "op": "forward", "kernels": "sym", "width": 512, "height": 512, "sigma": 20.0, "gamma": 2.0},
        # the same size with the small kernel set, a preview quality
        {"name": "preview", "op": "forward", "kernels": "small", "width": 643, "height": 480, "sigma": 15.0, "gamma": 1.5},
        # a ragged camera frame with the gaussian set, the scale maps kept for inspection
        {"name": "frame_maps", "op": "forward_map", "kernels": "gauss", "width": 1535, "height": 1021, "sigma": 25.0,
         "gamma": 1.5},
        # the benchmark image
        {"name": "image4096", "op": "forward", "kernels": "sym", "width": 4096, "height": 4096, "sigma": 20.0,
         "gamma": 2.0},
        # the contracted mode on an ordinary photograph
        {"name": "contracted", "op": "ffma", "kernels": "sym", "width": 1600, "height": 1200, "sigma": 20.0, "gamma": 2.0},
        # an RGB photograph, channels interleaved
        {"name": "rgb", "op": "channels", "kernels": "sym", "width": 768, "height": 513, "channels": 3, "sigma": 20.0,
         "gamma": 2.0},
        # a plan of images of mixed sizes, sigmas and gammas, replayed from a graph
        {"name": "batch_mixed", "op": "batch", "kernels": "sym", "width": 900, "height": 700, "images": 10, "mixed": True},
        # host array in, host array out (pinned), as the command line's engine does it
        {"name": "host2048", "op": "host", "kernels": "sym", "width": 2048, "height": 2048, "sigma": 20.0, "gamma": 2.0},
        # one image of a training step that keeps nothing from the forward
        {"name": "backward1024", "op": "backward", "kernels": "sym", "width": 1024, "height": 1024, "sigma": 20.0,
         "gamma": 2.0},
        # a training step on a crop: forward with its state kept, and the adjoint from that state
        {"name": "step_crop", "op": "step", "kernels": "gauss", "width": 384, "height": 320, "sigma": 25.0, "gamma": 1.5},
        # the adjoint of a batch of equal crops, planned once and replayed
        {"name": "backward_batch", "op": "backward_batch", "kernels": "sym", "width": 640, "height": 640, "images": 8,
         "mixed": False},
    ]


def _size(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    op = rng.choice(["forward", "forward", "forward_map", "ffma", "channels", "batch", "host", "backward", "step",
                     "backward_batch"])
    case = {"op": op, "kernels": rng.choice(["sym", "sym", "gauss", "small", "tapered"])}
    if op in ("batch", "backward_batch"):
        case.update(width=_size(rng, 96, 1000), height=_size(rng, 96, 1000), images=rng.randint(2, 12),
                    mixed=rng.random() < 0.5)
        return case
    low, high = {"forward": (24, 3000), "channels": (64, 1200), "step": (64, 1200)}.get(op, (64, 2000))
    # a side of its own for each, the second within a factor of two of the first
    w = _size(rng, low, high)
    h = max(low // 2, min(high, int(round(w * math.exp(rng.uniform(-0.7, 0.7))))))
    case.update(width=w, height=h, sigma=float(rng.randint(10, 40)), gamma=round(rng.uniform(1.3, 2.5), 2))
    if op == "channels":
        case["channels"] = rng.choice([2, 3, 4])
    return case


def _images(case):
    """(width, height, sigma, gamma) of every image of the case; sigma in units of 1."""
    w, h = case["width"], case["height"]
    if "images" not in case:
        return [(w, h, case["sigma"] / 255.0, case["gamma"])]
    if not case["mixed"]:
        return [(w, h, 20.0 / 255.0, 2.0)] * case["images"]
    rng = np.random.default_rng(w * 65536 + h)  # sizes belong to the case, not to the seed of the inputs
    out = []
    for _ in range(case["images"]):
        f = rng.uniform(0.4, 1.5, 2)
        out.append((max(16, int(w * f[0])), max(16, int(h * f[1])), float(np.float32(rng.uniform(10, 40) / 255.0)),
                    float(np.float32(rng.uniform(1.5, 2.5)))))
    return out


def _noisy(w, h, sigma, gen):
    """A scene of flat cells, half of them striped, over a ramp, in [0, 1], plus gaussian noise."""
    dev = "cuda"
    yy = torch.arange(h, device=dev, dtype=torch.float32)[:, None].expand(h, w)
    xx = torch.arange(w, device=dev, dtype=torch.float32)[None, :].expand(h, w)
    pitch = 80.0
    ny, nx = int(h / pitch) + 3, int(w / pitch) + 3
    cells = torch.rand((6, ny, nx), device=dev, generator=gen)
    iy, ix = (yy / pitch).long() + 1, (xx / pitch).long() + 1
    best = torch.full((h, w), float("inf"), device=dev)
    at = torch.zeros((h, w), device=dev, dtype=torch.long)
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            k = (iy + dy) * nx + ix + dx
            sy = ((iy + dy - 1) + cells[0].flatten()[k]) * pitch
            sx = ((ix + dx - 1) + cells[1].flatten()[k]) * pitch
            dist = (yy - sy) ** 2 + (xx - sx) ** 2
            near = dist < best
            best = torch.where(near, dist, best)
            at = torch.where(near, k, at)
    level, kind, angle, period = (cells[i].flatten()[at] for i in (2, 3, 4, 5))
    wave = torch.sin((xx * torch.cos(math.pi * angle) + yy * torch.sin(math.pi * angle)) * (2 * math.pi)
                     / (4.0 + 12.0 * period))
    ramp = 0.2 * (xx / max(w, 1) - 0.5) + 0.1 * (yy / max(h, 1) - 0.5)
    clean = torch.clamp(level + ramp + torch.where(kind < 0.5, 0.15 * wave, 0.0 * wave), 0.0, 1.0)
    return (clean + sigma * torch.randn((h, w), device=dev, generator=gen)).contiguous()


def _inputs(case, seed):
    """The noisy images and cotangents of a case, from the seed alone."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["op"] == "channels":
        w, h, sigma, _ = _images(case)[0]
        return [torch.stack([_noisy(w, h, sigma, gen) for _ in range(case["channels"])], 2).contiguous()], []
    noisy = [_noisy(w, h, sigma, gen) for w, h, sigma, _ in _images(case)]
    grads = []
    if case["op"] in ("backward", "step", "backward_batch"):
        grads = [torch.randn(x.shape, device="cuda", generator=gen) for x in noisy]
    return noisy, grads


def prepare(case, seed):
    noisy, grads = _inputs(case, seed)
    ks = lpaici.KernelSet.load(os.path.join(TAPS, KERNELS[case["kernels"]]))
    images = _images(case)
    st = {"op": case["op"], "ks": ks, "noisy": noisy, "grads": grads, "sigma": images[0][2], "gamma": images[0][3]}
    op = case["op"]
    if op == "host":
        st["host_in"] = noisy[0].cpu().pin_memory().numpy()
        st["host_out"] = torch.empty(noisy[0].shape, dtype=torch.float32, pin_memory=True).numpy()
    elif op == "batch":
        st["outs"] = [torch.empty_like(x) for x in noisy]
        st["plan"] = lpaici.Batch(ks, noisy, st["outs"], [i[2] for i in images], [i[3] for i in images], use_graph=True)
    elif op == "backward_batch":
        st["outs"] = [torch.empty_like(x) for x in noisy]
        st["plan"] = lpaici.BackwardBatch(ks, noisy, grads, st["outs"], [i[2] for i in images], [i[3] for i in images],
                                          use_graph=True)
    return st


def run(st):
    op, ks, sigma, gamma = st["op"], st["ks"], st["sigma"], st["gamma"]
    if op == "forward":
        return lpaici.forward(ks, st["noisy"][0], sigma, gamma)
    if op == "forward_map":
        return lpaici.forward(ks, st["noisy"][0], sigma, gamma, scale_map=True)
    if op == "ffma":
        return lpaici.forward(ks, st["noisy"][0], sigma, gamma, ffma=True)
    if op == "channels":
        return lpaici.forward_channels(ks, st["noisy"][0], sigma, gamma)
    if op == "host":
        return lpaici.denoise_host(ks, st["host_in"], sigma, gamma, out=st["host_out"])
    if op == "backward":
        return lpaici.backward(ks, st["noisy"][0], st["grads"][0], sigma, gamma)
    if op == "step":
        out, state = lpaici.forward_state(ks, st["noisy"][0], sigma, gamma)
        return out, lpaici.backward_state(ks, state, st["grads"][0], sigma)
    st["plan"].run()
    return st["outs"]


def _taps(name):
    """A tap-list file: (D, S, per kernel the list of (dy, dx, weight) in row-major order)."""
    with open(os.path.join(TAPS, KERNELS[name]), "rb") as f:
        data = f.read()
    D, S = np.frombuffer(data, np.int32, 2, 8)
    nk = int(D) * int(S)
    n_runs, n_taps = (int(v) for v in np.frombuffer(data, np.int32, 2, 16 + 8 * nk))
    at = 24 + 8 * nk
    first = np.frombuffer(data, np.int32, nk + 1, at)
    at += 4 * (nk + 1)
    dy, dx0, length = (np.frombuffer(data, np.int32, n_runs, at + 4 * n_runs * i) for i in range(3))
    w = np.frombuffer(data, np.float32, n_taps, at + 12 * n_runs)
    start = np.concatenate([[0], np.cumsum(length)])
    out = []
    for k in range(nk):
        taps = []
        for r in range(first[k], first[k + 1]):
            taps += [(int(dy[r]), int(dx0[r]) + j, w[start[r] + j]) for j in range(length[r])]
        out.append(taps)
    return int(D), int(S), out


def work(case):
    D, S, kernels = _taps(case["kernels"])
    taps = sum(sum(1 for t in k if t[2] != 0) for k in kernels)
    px = sum(w * h for w, h, _, _ in _images(case)) * case.get("channels", 1)
    op = case["op"]
    # the forward: every nonzero tap of every kernel a product and a sum (what noise leaves of the early
    # stop is a few per cent); the adjoint: the selected kernels' taps, half of the sweep's on such images
    flops = {"step": 3, "backward": 3, "backward_batch": 3}.get(op, 2) * taps * px
    bytes_ = {"forward_map": 8 + D, "step": 16, "backward": 12, "backward_batch": 12}.get(op, 8) * px
    return {"bytes": bytes_, "flops": flops}


def _select(kernels, D, S, x, sigma, gamma, visit):
    """The interval-intersection rule for every direction and pixel.  A selected scale is a whole number
    that the method's own 32-bit arithmetic defines, so the interval test repeats that arithmetic (taps in
    row-major order, each product and sum rounded); visit(d, chosen, taps of the direction's kernels, the
    variances) then works in 64 bits."""
    h, w = x.shape
    r = max(max(abs(t[0]), abs(t[1])) for k in kernels for t in k)
    pad = F.pad(x, (r, r, r, r))
    s2 = np.float32(sigma) * np.float32(sigma)
    for d in range(D):
        lo = torch.full_like(x, -math.inf)
        hi = torch.full_like(x, math.inf)
        chosen = torch.zeros(x.shape, dtype=torch.long, device=x.device)
        alive = torch.ones(x.shape, dtype=torch.bool, device=x.device)
        variances = []
        for s in range(S):
            taps = kernels[d * S + s]
            conv = torch.zeros_like(x)
            prod = torch.empty_like(x)
            norm = np.float32(0)
            for dy, dx, wt in taps:
                torch.mul(pad[r + dy:r + dy + h, r + dx:r + dx + w], float(wt), out=prod)
                conv.add_(prod)
                norm = np.float32(norm + np.float32(wt * wt))
            var = np.float32(s2 * norm)
            thr = float(np.float32(np.float32(gamma) * np.sqrt(var)))
            lo = torch.maximum(lo, conv - thr)
            hi = torch.minimum(hi, conv + thr)
            alive &= hi >= lo
            chosen = torch.where(alive, s, chosen)
            variances.append(float(var))
        visit(d, chosen, kernels[d * S:(d + 1) * S], torch.tensor(variances, dtype=torch.float64, device=x.device))


def _forward64(kernels, D, S, x, sigma, gamma):
    h, w = x.shape
    r = max(max(abs(t[0]), abs(t[1])) for k in kernels for t in k)
    pad = F.pad(x.double(), (r, r, r, r))
    num, den = torch.zeros_like(x, dtype=torch.float64), torch.zeros_like(x, dtype=torch.float64)

    def visit(d, chosen, taps, var):
        for s, k in enumerate(taps):
            conv = torch.zeros_like(num)
            for dy, dx, wt in k:
                conv.add_(pad[r + dy:r + dy + h, r + dx:r + dx + w], alpha=float(wt))
            mask = chosen == s
            num.add_(torch.where(mask, conv / var[s], 0.0))
            den.add_(torch.where(mask, 1.0 / var[s], 0.0))

    _select(kernels, D, S, x, sigma, gamma, visit)
    return num / den


def _backward64(kernels, D, S, x, g, sigma, gamma):
    h, w = x.shape
    r = max(max(abs(t[0]), abs(t[1])) for k in kernels for t in k)
    selected = []
    _select(kernels, D, S, x, sigma, gamma, lambda d, chosen, taps, var: selected.append((chosen, taps, var)))
    den = sum(1.0 / var[chosen] for chosen, _, var in selected)
    u = g.double() / den
    grad = torch.zeros((h + 2 * r, w + 2 * r), dtype=torch.float64, device=x.device)
    for chosen, taps, var in selected:
        for s, k in enumerate(taps):
            field = torch.where(chosen == s, u / var[s], 0.0)
            for dy, dx, wt in k:
                grad[r + dy:r + dy + h, r + dx:r + dx + w].add_(field, alpha=float(wt))
    return grad[r:r + h, r:r + w].contiguous()


def exact(case, seed):
    noisy, grads = _inputs(case, seed)
    D, S, kernels = _taps(case["kernels"])
    images = _images(case)
    op, sigma, gamma = case["op"], images[0][2], images[0][3]
    if op == "channels":
        x = noisy[0]
        return torch.stack([_forward64(kernels, D, S, x[:, :, c].contiguous(), sigma, gamma)
                            for c in range(x.shape[2])], 2)
    if op == "batch":
        return [_forward64(kernels, D, S, x, i[2], i[3]) for x, i in zip(noisy, images)]
    if op == "backward_batch":
        return [_backward64(kernels, D, S, x, g, i[2], i[3]) for x, g, i in zip(noisy, grads, images)]
    if op == "backward":
        return _backward64(kernels, D, S, noisy[0], grads[0], sigma, gamma)
    out = _forward64(kernels, D, S, noisy[0], sigma, gamma)
    if op == "forward_map":
        return out, None
    if op == "step":
        return out, _backward64(kernels, D, S, noisy[0], grads[0], sigma, gamma)
    return out.cpu().numpy() if op == "host" else out
