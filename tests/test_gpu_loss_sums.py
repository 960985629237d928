"""GPU: how far the two sums of the L1 + SSIM loss go in float32 before they enter the double sum: over 32x16
values, four rows of a column by a thread, 32 columns by a tree, four such strips in turn.  Replayed bit for bit,
on images whose edges cut the 32x16 blocks and the 32x32 tiles of the kernels: |x - y| of every pixel is formed in
float32 here, an SSIM value is read from the kernel as the sum of an 11x11 crop, which has one."""
import pytest
import torch

from filtergs_b200._C import _ptr, _stream
from filtergs_b200._lib import call, lib

pytestmark = pytest.mark.gpu


def _sums(x, y):
    _, H, W = x.shape
    g = torch.empty_like(x)
    sums = torch.zeros(2, dtype=torch.float64, device=x.device)
    scratch = torch.empty(int(lib().fgs_loss_scratch_bytes(W, H)) // 4 + 1, device=x.device)
    call("fgs_loss_l1_ssim", W, H, _ptr(x), _ptr(y), _ptr(g), 1e-3, 2e-3, _ptr(sums), _ptr(scratch), _stream())
    return sums


def _replay(v):
    """The sum of a [C, h, w] array of float32 values as the loss forms it."""
    C, h, w = v.shape
    full = v.new_zeros(C, (h + 15) // 16 * 16, (w + 31) // 32 * 32)
    full[:, :h, :w] = v
    b = full.view(C, full.shape[1] // 16, 4, 4, full.shape[2] // 32, 32)  # channel, block, strip, row, block, lane
    s = torch.zeros_like(b[:, :, :, 0])
    for r in range(4):
        s = s + b[:, :, :, r]
    for o in (16, 8, 4, 2, 1):
        s = s + s[..., torch.arange(32, device=v.device) ^ o]
    s = s[..., 0]
    t = torch.zeros_like(s[:, :, 0])
    for k in range(4):
        t = t + s[:, :, k]
    return t.double().sum()


@pytest.mark.parametrize("W,H", [(33, 17), (74, 59), (97, 130)])
def test_l1_sum(cuda, W, H):
    g = torch.Generator(device="cuda").manual_seed(W)
    x, y = (torch.rand(3, H, W, device="cuda", generator=g) for _ in range(2))
    # (doubles hold a sum of a few dozen float32 values of like size exactly: their order does not show)
    assert float(_sums(x, y)[0]) == float(_replay((x - y).abs()))


def test_ssim_sum(cuda):
    W, H = 49, 37
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.rand(3, H, W, device="cuda", generator=g)
    y = (x + 0.2 * torch.rand(3, H, W, device="cuda", generator=g)).clamp(max=1)
    ss = torch.empty(3, H - 10, W - 10, device="cuda")
    one = torch.zeros(2, 3, 11, 11, device="cuda")  # black channels: an SSIM of exactly 1 each
    for c in range(3):
        for i in range(H - 10):
            vals = []
            for j in range(W - 10):
                one[0, 0], one[1, 0] = x[c, i:i + 11, j:j + 11], y[c, i:i + 11, j:j + 11]
                vals.append(_sums(one[0], one[1])[1] - 2)
            ss[c, i] = torch.stack(vals).float()
    assert float(ss.min()) > 0.02
    assert float(_sums(x, y)[1]) == float(_replay(ss))
