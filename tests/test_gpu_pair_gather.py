"""GPU: the sums of the per-pair gradient rows, at the numbers of Gaussians and of rows where the kernel
changes: runs of four ranks and blocks of sixteen, no rows at all, groups of 32 rows, more rows than a
block stages at once (512), and several such Gaussians side by side; against the oracle's backward at the
tolerance the other comparisons with it use."""
import numpy as np
import pytest
import torch

from _helpers import Case, O, S, norm_rel, ours, run_backward, run_forward

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,large", [(1, 0), (1, 1), (3, 2), (16, 0), (17, 5), (65, 1), (400, 12)])
def test_gradient_sums(cuda, P, large):
    sc, cam = S.small_scene(P=P, seed=91, W=512, H=400)
    sc["opacities"] = (0.3 * sc["opacities"]).astype(np.float32)
    sc["scales"][:large] = 2.0                      # every tile of the view
    sc["means3D"][:large, 2] = 2.0 + 0.1 * np.arange(large)
    case = Case(sc, cam)
    dL = np.random.default_rng(3).standard_normal((3, cam.H, cam.W)).astype(np.float32)
    fwd = run_forward(ours, case)
    tiles = ours.preprocess_outputs(fwd[6], P)["tiles_touched"]
    assert int((tiles > 512).sum()) == large and (P < 10 or int((tiles < 32).sum()) > 0)
    mine = run_backward(ours, case, fwd, torch.from_numpy(dL).cuda())
    scene = case.oracle_scene()
    want = O.backward(scene, O.forward(scene), dL)
    for n, a in zip(["means2D", "colors", "opacity", "means3D", "cov3D", "sh", "scales", "rotations"], mine):
        assert norm_rel(a.cpu(), torch.from_numpy(want[n]).reshape(a.shape)) <= 1e-3, n
