"""The 3x3 convolution and its three gradients where the tiles of 8 x 16
pixels, the steps of 64 channels and the 64 outputs of a CTA end: against
float64 on the same bf16 operands.

Tolerances: FP32 sums of at most 9 * 264 (weights: 2 * 33 * 24) products, relative to the result's
norm well under 1e-5 for random operands; a bf16 result (8 bits) rounds by at
most 2**-8."""
import pytest
import torch
import torch.nn.functional as F

from tests._util import rel

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("n,h,w,c,co", [
    (1, 1, 1, 8, 8), (2, 16, 8, 64, 64), (1, 17, 9, 72, 80), (3, 5, 50, 136, 72), (2, 33, 24, 24, 8),
    (1, 16, 64, 128, 200), (5, 20, 12, 264, 16), (2, 9, 23, 56, 136)])
def test_conv3x3_matches_float64(n, h, w, c, co):
    from sweep_b200 import unet
    gen = torch.Generator().manual_seed(n + 3 * h + 7 * w + c + co)
    x = torch.randn((n, h, w, c), generator=gen).to(torch.bfloat16)
    wt = (torch.randn((co, 3, 3, c), generator=gen) * 0.1).to(torch.bfloat16).float()
    b = torch.randn(co, generator=gen)
    g = torch.randn((n, h, w, co), generator=gen).to(torch.bfloat16).float()
    leaves = [t.to(DEV).requires_grad_(True) for t in (x, wt, b)]
    y = unet.conv3x3(*leaves)
    y.backward(g.to(DEV))
    unet.check()
    ref = [t.double().requires_grad_(True) for t in (x, wt, b)]
    yr = F.conv2d(ref[0].permute(0, 3, 1, 2), ref[1].permute(0, 3, 1, 2), ref[2], padding=1).permute(0, 2, 3, 1)
    yr.backward(g.double())
    errs = [rel(y.detach().cpu(), yr.detach())] + [rel(a.grad.float().cpu(), r.grad) for a, r in zip(leaves, ref)]
    print(f"{(n, h, w, c, co)}: y {errs[0]:.1e}, dx {errs[1]:.1e}, dw {errs[2]:.1e}, db {errs[3]:.1e}")
    assert errs[0] < 1e-5 and errs[2] < 1e-5 and errs[3] < 1e-5
    assert errs[1] < 2.0 ** -8 + 1e-5


def test_weight_gradient_keeps_an_infinity_to_its_taps():
    """Infinite inputs in the last row and column of an image that ends inside a
    tile: the taps that do not read them keep a finite gradient."""
    from sweep_b200 import unet
    gen = torch.Generator().manual_seed(3)
    x = torch.randn((2, 17, 12, 16), generator=gen).to(torch.bfloat16)
    x[0, 16, 5, 3], x[1, 4, 11, 9] = float("inf"), float("-inf")
    g = torch.randn((2, 17, 12, 8), generator=gen).to(torch.bfloat16).float()
    w = torch.zeros((8, 3, 3, 16), device=DEV, requires_grad=True)
    y = unet.conv3x3(x.to(DEV), w, torch.zeros(8, device=DEV))
    y.backward(g.to(DEV))
    unet.check()
    want = torch.zeros((8, 3, 3, 16), dtype=torch.float64)
    for dy in range(3):
        for dx in range(3):
            h, v = slice(max(0, 1 - dy), 17 - max(0, dy - 1)), slice(max(0, 1 - dx), 12 - max(0, dx - 1))
            hx, vx = slice(max(0, dy - 1), 17 - max(0, 1 - dy)), slice(max(0, dx - 1), 12 - max(0, 1 - dx))
            want[:, dy, dx] = torch.einsum("nhwo,nhwc->oc", g[:, h, v].double(), x[:, hx, vx].double())
    got = w.grad.double().cpu()
    assert want[:, 0, :, 3].isfinite().all() and not want[:, 1:, :, 3].isfinite().any()
    assert want[:, :, 0, 9].isfinite().all() and not want[:, :, 1:, 9].isfinite().any()
    assert torch.equal(got.isfinite(), want.isfinite())
    assert rel(got[want.isfinite()], want[want.isfinite()]) < 1e-5


def test_saved_tensors_of_another_order():
    """Saved-tensor hooks may hand the operands back in another memory order."""
    from sweep_b200 import unet
    gen = torch.Generator().manual_seed(4)
    grads = []
    for hooked in (False, True):
        gen.manual_seed(4)
        leaves = [torch.randn(s, generator=gen).to(DEV) for s in ((2, 9, 12, 24), (16, 3, 3, 24), (16,))]
        leaves[0] = leaves[0].to(torch.bfloat16)
        for t in leaves:
            t.requires_grad_(True)
        swap = (lambda t: t.transpose(0, -1).contiguous()), (lambda t: t.transpose(0, -1))
        with torch.autograd.graph.saved_tensors_hooks(*swap) if hooked else torch.enable_grad():
            y = unet.conv3x3(*leaves)
        (y * y.detach().cos()).sum().backward()
        unet.check()
        grads.append([t.grad for t in leaves])
    for a, b in zip(*grads):
        assert rel(b.float().cpu(), a.float().cpu()) < 1e-5      # the weight gradient's atomics
