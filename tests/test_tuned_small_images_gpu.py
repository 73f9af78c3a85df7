"""Images of a few tiles after lpaici_autotune, on a large image and on a small one: still swept by clusters, as with a set
that is not tuned.  The same bits, and less than twice its time (without clusters it is 1.3 to 2.4 times; the best of
five loops of twenty calls each)."""
import pytest

import lpaici
from conftest import SYM, kernel_file

pytestmark = pytest.mark.gpu

SIGMA, GAMMA = 0.08, 2.0


def best_ms(ks, x, out):
    import torch

    best = 1e9
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(20):
            lpaici.forward(ks, x, SIGMA, GAMMA, out=out)
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) / 20)
    return best


@pytest.mark.parametrize("on", [(1024, 1024), (97, 64)])
def test_clusters_after_tuning(on):
    import torch

    plain, tuned = (lpaici.KernelSet.load(kernel_file(SYM)) for _ in range(2))
    tuned.autotune(*on, SIGMA, GAMMA)
    ratio = {}
    for W, H in ((33, 20), (97, 64), (128, 128), (200, 150)):
        gen = torch.Generator("cuda")
        gen.manual_seed(W)
        x = torch.rand(H, W, device="cuda", generator=gen)
        a, b = lpaici.forward(plain, x, SIGMA, GAMMA), lpaici.forward(tuned, x, SIGMA, GAMMA)
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
        ratio[W, H] = best_ms(tuned, x, b) / best_ms(plain, x, a)
    print({k: round(v, 2) for k, v in ratio.items()})
    assert ratio[97, 64] < 2.0 and ratio[33, 20] < 2.0, ratio
