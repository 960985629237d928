"""GPU: the paths around the kernels that one view takes through autograd and with statistics: images of
few and of many tiles (the statistics' device memory comes from different buffers), gradient buffers that
are zeroed inside the backward launch (every row of a Gaussian no tile lists, at lengths that are not whole
16-byte items), a loss that does not use the image, and a call after one whose kernels are still running."""
import pytest
import torch

from _helpers import O, ours, run_backward, run_forward, small_case
from filtergs_b200.diff_gaussian_rasterization_wodilate import GaussianRasterizationSettings, GaussianRasterizer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(16, 16), (30, 17), (48, 48), (160, 16), (250, 130)])
def test_statistics_vs_oracle(cuda, W, H):
    case = small_case(P=1500, seed=31, W=W, H=H)
    got = run_forward(ours, case, stats=True)[9]
    f = O.forward(case.oracle_scene(), stats=True)
    want = O.kpc_stats(f["kv_sum"], f["kv_cnt"], f["ranges"])
    T = ((W + 15) // 16) * ((H + 15) // 16)
    assert got.numel() == 9 + 128 + 2 * T
    assert got[3] == f["num_rendered"] and got[4] == T and got[5] == 1500 and got[8] == 11
    # a pair whose weight lies within rounding of a bin's edge may fall on either side
    for i, k in ((6, "used_kv_pairs"), (7, "unused_kv_pairs")):
        assert abs(float(got[i]) - want[k]) <= 2, k
    assert torch.allclose(got[9 + 128 + T:], torch.from_numpy(want["tile_total_kv"]))
    assert (got[9 + 64:9 + 75] - torch.from_numpy(want["kpc_hist"])).abs().sum() <= 8
    assert (got[9 + 128:9 + 128 + T] - torch.from_numpy(want["tile_ratio"])).abs().max() <= 0.05
    assert float((got[9 + 11:9 + 64]).abs().sum()) == 0 and float(got[9 + 75:9 + 128].abs().sum()) == 0


@pytest.mark.parametrize("P,M", [(1, 1), (7, 4), (333, 9), (1021, 16)])
def test_gradients_of_unlisted_gaussians_are_zero(cuda, P, M):
    degree = {1: 0, 4: 1, 9: 2, 16: 3}[M]
    case = small_case(P=P, seed=41, W=70, H=50)
    case.scene["shs"], case.scene["sh_degree"] = case.scene["shs"][:, :M], degree
    case.scene["means3D"][::3, 2] = -1.0    # behind the camera
    fwd = run_forward(ours, case)
    junk = [torch.full((P + 5, 64), float("nan"), device="cuda") for _ in range(20)]  # what new buffers may hold
    del junk
    grads = run_backward(ours, case, fwd, torch.ones(3, 50, 70, device="cuda"))
    gone = fwd[5] == 0
    assert gone[::3].all()
    for g in grads:
        assert torch.isfinite(g).all() and float(g[gone].abs().sum()) == 0
    if P > 100:
        assert float(grads[3][~gone].abs().sum()) > 0


def _module(case):
    a = case.torch_inputs()
    rs = GaussianRasterizationSettings(case.cam.H, case.cam.W, case.cam.tanfovx, case.cam.tanfovy, a["background"], 1.0,
                                       a["viewmatrix"], a["projmatrix"], case.scene["sh_degree"], a["campos"], False, False)
    x = {k: a[k].clone().requires_grad_(True) for k in ("means3D", "opacity", "sh", "scales", "rotations")}
    r = GaussianRasterizer(rs)
    return x, lambda: r(x["means3D"], torch.zeros_like(x["means3D"]), x["opacity"], shs=x["sh"], scales=x["scales"],
                        rotations=x["rotations"], ogfs_enable_stats=False)


def test_loss_without_the_image(cuda):
    x, render = _module(small_case(P=500, seed=43, W=64, H=48))
    color, _, _, pw_pixel, _ = render()
    (pw_pixel.sum() + x["opacity"].sum()).backward()
    assert torch.equal(x["opacity"].grad, torch.ones_like(x["opacity"]))   # the weights carry no gradient
    assert float(x["means3D"].grad.abs().sum()) == 0


def test_calls_queue_behind_one_another(cuda):
    """A forward while the previous backward still runs gives what it gives alone."""
    x, render = _module(small_case(P=20000, seed=44, W=320, H=240))
    want = [t.clone() for t in render()]
    torch.cuda.synchronize()
    for _ in range(5):
        got = render()
        torch.autograd.grad(got[0].sum(), list(x.values()))
    for a, b in zip(render(), want):
        assert torch.equal(a, b)
