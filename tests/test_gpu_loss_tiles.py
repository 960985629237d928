"""GPU: the L1 + SSIM kernels where their tiling can go wrong.  A pixel's arithmetic does not depend on the
32x32 tile it falls in or on how the tile was staged (16-byte copies for rows that allow them, 4-byte ones
otherwise), so these change no bit: the image embedded at another offset of a larger image, and the image in
storage that does not start on 16 bytes.  (The values themselves are checked against torch in
test_gpu_train.py.)"""
import pytest
import torch

from filtergs_b200._C import _ptr, _stream
from filtergs_b200._lib import call, lib

pytestmark = pytest.mark.gpu


def _grad(x, y):
    """dL/dx with fixed scales (not those of the image's size), and the two sums."""
    _, H, W = x.shape
    g = torch.full_like(x, float("nan"))
    sums = torch.zeros(2, dtype=torch.float64, device=x.device)
    scratch = torch.full((int(lib().fgs_loss_scratch_bytes(W, H)) // 4 + 1,), float("nan"), device=x.device)
    call("fgs_loss_l1_ssim", W, H, _ptr(x), _ptr(y), _ptr(g), 1e-3, 2e-3, _ptr(sums), _ptr(scratch), _stream())
    return g, sums


@pytest.mark.parametrize("W,H", [(21, 21), (32, 43), (42, 42), (43, 74), (64, 33), (108, 97)])
@pytest.mark.parametrize("dx,dy", [(1, 3), (4, 0), (32, 32), (39, 21)])
def test_gradient_does_not_depend_on_the_tile(cuda, W, H, dx, dy):
    g = torch.Generator(device="cuda").manual_seed(W * H + dx)
    big = [torch.rand(3, H + dy + 2, W + dx + 5, device="cuda", generator=g) for _ in range(2)]
    small = [t[:, dy:dy + H, dx:dx + W].contiguous() for t in big]
    a, _ = _grad(*small)
    b, _ = _grad(*big)
    assert torch.isfinite(a).all() and torch.isfinite(b).all()
    # the pixels all of whose windows lie in the small image
    inner = (slice(None), slice(10, H - 10), slice(10, W - 10))
    assert torch.equal(a[inner], b[:, dy:dy + H, dx:dx + W][inner])


@pytest.mark.parametrize("W,H", [(12, 11), (44, 42), (64, 75), (96, 40)])
@pytest.mark.parametrize("off", [1, 2, 3])
def test_storage_off_16_bytes(cuda, W, H, off):
    g = torch.Generator(device="cuda").manual_seed(W + H)
    x, y = (torch.rand(3, H, W, device="cuda", generator=g) for _ in range(2))
    shift = lambda t: torch.cat([t.new_zeros(off), t.reshape(-1)])[off:].view(t.shape)  # noqa: E731
    a, sa = _grad(x, y)
    for u, v in ((shift(x), y), (x, shift(y)), (shift(x), shift(y))):
        b, sb = _grad(u, v)
        assert torch.equal(a, b) and torch.equal(sa, sb)
