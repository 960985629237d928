"""GPU: what a batched backward does around its compositing: every gradient row written on each step,
whatever the buffers held (they are zeroed in shares after single tiles, rows of Gaussians no view saw
included), and the list of the seen Gaussians at lengths around its blocks of 2048, for one word of
visibility bits and for two."""
import pytest
import torch

from filtergs_b200.batched import BatchedRasterizer
from test_gpu_batched import _cams, _plain, _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,views", [(1, 1), (2047, 2), (2049, 1), (10_000, 33), (60_001, 3)])
def test_gradient_rows_are_written(cuda, P, views):
    sc = _scene(P=P)
    cams = _cams(views)
    bg = torch.zeros(3, device="cuda")
    br = BatchedRasterizer(sc["means3D"], sc["opacities"], sc["scales"], sc["rotations"], cams, shs=sc["shs"],
                           sh_degree=3, bg=bg)
    gen = torch.Generator(device="cuda").manual_seed(7)
    for v in range(views):
        br.dL[v].copy_(torch.randn(br.dL[v].shape, device="cuda", generator=gen))
    for _ in range(2):
        for g in br.grad.values():
            g.fill_(float("nan"))
        br.step()
    br.check()
    want, seen = None, torch.zeros(P, dtype=torch.bool, device="cuda")
    for v in range(views):
        f, g = _plain(sc, cams[v], br.dL[v], bg)
        rows = dict(means3D=g[3], opacity=g[2], sh=g[5], scales=g[6], rotations=g[7])
        want = rows if want is None else {k: want[k] + rows[k] for k in rows}
        seen |= f[5] > 0
    for k, g in br.grad.items():
        assert torch.equal(g.reshape(want[k].shape), want[k]), k
        assert float(g[~seen].abs().sum()) == 0, k
