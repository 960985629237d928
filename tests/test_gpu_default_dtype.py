"""GPU: the operator under another default dtype of torch.  All its tensors are float32 whatever the default
is, also the image gradient that it makes itself for a loss that does not use the image."""
import pytest
import torch

from _helpers import small_case
from filtergs_b200.diff_gaussian_rasterization_wodilate import GaussianRasterizationSettings, GaussianRasterizer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("use_image", [False, True])
def test_backward_under_a_default_dtype(cuda, dtype, use_image):
    case = small_case(P=500, seed=43, W=64, H=48)
    a = case.torch_inputs()
    rs = GaussianRasterizationSettings(case.cam.H, case.cam.W, case.cam.tanfovx, case.cam.tanfovy, a["background"], 1.0,
                                       a["viewmatrix"], a["projmatrix"], case.scene["sh_degree"], a["campos"], False,
                                       False)
    x = {k: a[k].clone().requires_grad_(True) for k in ("means3D", "opacity", "sh", "scales", "rotations")}
    was = torch.get_default_dtype()
    torch.set_default_dtype(dtype)
    try:
        color, _, _, pw_pixel, _ = GaussianRasterizer(rs)(
            x["means3D"], torch.zeros_like(x["means3D"]), x["opacity"], shs=x["sh"], scales=x["scales"],
            rotations=x["rotations"], ogfs_enable_stats=False)
        assert color.dtype == torch.float32
        (pw_pixel.sum() + (color.sum() if use_image else 0) + x["opacity"].sum()).backward()
    finally:
        torch.set_default_dtype(was)
    for k, t in x.items():
        assert t.grad.dtype == torch.float32 and torch.isfinite(t.grad).all(), k
    assert (float(x["means3D"].grad.abs().sum()) > 0) == use_image
    if not use_image:
        assert torch.equal(x["opacity"].grad, torch.ones_like(x["opacity"]))
