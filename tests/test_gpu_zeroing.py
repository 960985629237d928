"""GPU: where the backward zeroes its gradient buffers.  Inside the compositing launch each tile's block stores a
share, which is free while the shares are small; buffers that would give a tile's block too much are zeroed by a
launch of their own, at the memory's rate.  Every row that no tile lists is zero either way."""
import pytest
import torch

from _helpers import ours, run_backward, run_forward, small_case
from filtergs_b200 import _lib
from filtergs_b200.batched import BatchedRasterizer, Camera

pytestmark = pytest.mark.gpu

# Gaussians (59 + 9 + 4 floats of gradients each) and an image: one tile block with megabytes to store, and
# tiles whose shares are a few KB
FEW, MANY = (60_000, 16, 16), (3_000, 256, 192)


def _case(P, W, H):
    case = small_case(P=P, seed=61, W=W, H=H)
    case.scene["means3D"][::3, 2] = -1.0  # behind the camera: no tile lists them
    return case


def _backward(case):
    fwd = run_forward(ours, case)
    junk = [torch.full((case.P, 64), float("nan"), device="cuda") for _ in range(4)]  # what new buffers may hold
    del junk
    n = _lib.launch_count()
    grads = run_backward(ours, case, fwd, torch.ones(3, case.cam.H, case.cam.W, device="cuda"))
    n = _lib.launch_count() - n
    gone = fwd[5] == 0
    assert gone[::3].all() and not gone.all()
    for g in grads:
        assert torch.isfinite(g).all() and float(g[gone].abs().sum()) == 0
    assert float(grads[3][~gone].abs().sum()) > 0
    return n


def test_one_view(cuda):
    assert _backward(_case(*FEW)) == _backward(_case(*MANY)) + 1


def _batched_backward(P, W, H, views=2):
    case = _case(P, W, H)
    a = case.torch_inputs()
    cams = [Camera(W, H, case.cam.tanfovx, case.cam.tanfovy, a["viewmatrix"], a["projmatrix"], a["campos"])] * views
    br = BatchedRasterizer(a["means3D"], a["opacity"], a["scales"], a["rotations"], cams, shs=a["sh"],
                           sh_degree=a["degree"], graph=False)
    for d in br.dL:
        d.fill_(1.0)
    for g in br.grad.values():
        if g is not None:
            g.fill_(float("nan"))
    br.forward()
    n = _lib.launch_count()
    br.backward()
    n = _lib.launch_count() - n
    br.check()
    gone = br.radii[0] == 0
    assert gone[::3].all() and not gone.all()
    for k, g in br.grad.items():
        if g is not None:
            assert torch.isfinite(g).all() and float(g[gone].abs().sum()) == 0, k
    return n


def test_batch(cuda):
    assert _batched_backward(*FEW) == _batched_backward(*MANY) + 1
