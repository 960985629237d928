"""GPU: the pair list's order -- (tile, depth bits), ties in the order of the Gaussians' indices -- at the
sizes where the sort passes change: one element, the edges of the smallest chunk (2048), more elements than
the resident blocks' smallest chunks hold (longer chunks), and more than their largest ones do (several
chunks per block).  Depths take 64 values, so that most keys have ties."""
import numpy as np
import pytest
import torch

from _helpers import Case, S, ours, run_forward

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,scale,pairs", [(1, 1e-4, 1), (2047, 1e-4, 2047), (2048, 1e-4, 2048), (2049, 1e-4, 2049),
                                           (40_961, 1e-4, 40_000), (700_001, 1e-4, 650_000),
                                           (150_000, 0.08, 2_600_000)])
def test_pair_order(cuda, P, scale, pairs):
    sc, cam = S.small_scene(P=P, seed=61, W=512, H=384)
    rng = np.random.default_rng(61)
    z = (2.0 + 0.05 * rng.integers(0, 64, P)).astype(np.float32)
    x = rng.uniform(-0.9, 0.9, (P, 2)).astype(np.float32)
    sc["means3D"] = np.concatenate([x * z[:, None] * np.float32([cam.tanfovx, cam.tanfovy]), z[:, None]], 1)
    sc["scales"] = np.full((P, 3), scale, np.float32)
    sc["opacities"] = np.full((P, 1), 0.5, np.float32)
    fwd = run_forward(ours, Case(sc, cam))
    K = fwd[0]
    assert K >= pairs
    keys, vals = ours.sorted_pairs(fwd[6], fwd[7], P, K)
    vals = vals.long()
    po = ours.preprocess_outputs(fwd[6], P)
    assert torch.equal(keys & 0xffffffff, po["depths"].view(torch.int32)[vals].long())
    up, same = keys[1:] > keys[:-1], keys[1:] == keys[:-1]
    assert (up | (same & (vals[1:] > vals[:-1]))).all()
    assert torch.equal(torch.bincount(vals, minlength=P), po["tiles_touched"].long())
    assert same.any() or K < 40_000
