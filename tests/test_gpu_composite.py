"""GPU: the compositing kernels where their record masks and their packed pixel pairs can go wrong.

* against the same arithmetic in torch, one record at a time and without masks, bit for bit:
  needles, opacities around 1/255 and images whose edges cut tiles and quads.
* colours, positions and upstream gradients that are huge or not finite, which take the
  kernels' branching form: the packed shapes (2 and 4 pixels per lane) against the scalar one
  (1 pixel per lane), bit for bit forward, non-finite values in the same places backward.
"""
import numpy as np
import pytest
import torch

from _helpers import Case, S, norm_rel, ours, run_backward, run_forward
from filtergs_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture
def shapes():
    cfg, split = _lib.get_render_config(), _lib.get_render_split()
    yield lambda p, b: _lib.set_render_config(p, b, p, b)
    _lib.set_render_config(*cfg)
    _lib.set_render_split(*split)


def _case(W, H, aspect, opacity, seed=51, P=4000, **kw):
    sc, cam = S.small_scene(P=P, seed=seed, W=W, H=H)
    rng = np.random.default_rng(seed)
    sc["scales"][:, 0] *= np.exp(rng.uniform(0, np.log(aspect), P)).astype(np.float32)
    sc["opacities"] = (sc["opacities"] * opacity).astype(np.float32)
    return Case(sc, cam, **kw)


def _fma(a, b, c):
    """fmaf of float32 tensors: the product is exact in float64."""
    return (a.double() * b.double() + c.double()).float()


def _composite(case, fwd):
    """The image, final T and n_contrib from a forward's own per-Gaussian state and sorted pairs, one
    record of every tile at a time, in float32 with the kernels' operation order and fused products."""
    W, H, P = case.cam.W, case.cam.H, case.P
    gx, gy = (W + 15) // 16, (H + 15) // 16
    po = ours.preprocess_outputs(fwd[6], P)
    vals = ours.sorted_pairs(fwd[6], fwd[7], P, fwd[0])[1].long()
    rg = ours.image_outputs(fwd[8], W, H)["ranges"].long()
    tile = torch.arange(gx * gy, device="cuda")
    k = torch.arange(256, device="cuda")
    px = ((tile % gx) * 16)[:, None] + (k % 16)[None]
    py = (torch.div(tile, gx, rounding_mode="floor") * 16)[:, None] + torch.div(k, 16, rounding_mode="floor")[None]
    T = torch.ones(gx * gy, 256, device="cuda")
    C = [torch.zeros_like(T) for _ in range(3)]
    last = torch.zeros_like(T, dtype=torch.int32)
    done = torch.zeros_like(T, dtype=torch.bool)
    n = rg[:, 1] - rg[:, 0]
    for j in range(int(n.max())):
        have = (j < n)[:, None]
        g = vals[(rg[:, 0] + j).clamp(max=vals.numel() - 1)]
        e = lambda t: t[g][:, None].expand_as(T)  # noqa: E731
        m, co = po["means2D"], po["conic_opacity"]
        dx, dy = e(m[:, 0]) - px, e(m[:, 1]) - py
        q = _fma(e(co[:, 0]) * dx, dx, e(co[:, 2]) * dy * dy)
        power = _fma(torch.full_like(T, -0.5), q, -(e(co[:, 1]) * dx * dy))
        alpha = torch.clamp(e(co[:, 3]) * torch.exp(power), max=0.99)
        on = have & ~done & ~(power > 0) & ~(alpha < np.float32(1 / 255))
        test = T * (1 - alpha)
        end = on & (test < 1e-4)
        done |= end
        on &= ~end
        for c in range(3):
            C[c] = torch.where(on, _fma(e(po["rgb"][:, c]) * alpha, T, C[c]), C[c])
        T = torch.where(on, test, T)
        last = torch.where(on, j + 1, last)
    img = lambda t: t.reshape(gy, gx, 16, 16).permute(0, 2, 1, 3).reshape(gy * 16, gx * 16)[:H, :W]  # noqa: E731
    return [img(c) for c in C], img(T), img(last)


@pytest.mark.parametrize("W,H", [(256, 192), (129, 75), (23, 41)])
@pytest.mark.parametrize("aspect,opacity", [(1, 1.0), (100, 1.0), (10, 0.012)])
def test_forward_bits(cuda, shapes, W, H, aspect, opacity):
    case = _case(W, H, aspect, opacity, use_filter=aspect != 100)
    for p, b in ((1, 256), (2, 128), (4, 64)):
        shapes(p, b)
        got = run_forward(ours, case)
        im = ours.image_outputs(got[8], W, H)
        C, T, last = _composite(case, got)
        off = (im["n_contrib"].reshape(H, W) != last) | (im["final_T"].reshape(H, W) != T)
        for c in range(3):
            off |= got[1][c] != C[c]
        # (float64 rounds a fused sum twice: about one in 2^29 differs, times 256 records at most)
        assert int(off.sum()) <= 2, (p, int(off.sum()))


@pytest.mark.parametrize("which", ["colors", "means", "gradient", "background"])
def test_values_too_large_for_the_packed_form(cuda, shapes, which):
    case = _case(150, 90, 3, 1.0, colors_precomp=True)
    dL = torch.randn(3, 90, 150, generator=torch.Generator().manual_seed(9)).cuda()
    if which == "colors":
        case.colors[::97, 0], case.colors[5::97, 1], case.colors[9::97] = np.inf, np.nan, 3e20
    elif which == "means":
        # a precomputed covariance lets a Gaussian with any mean through: far outside, on the axis
        case.scene["means3D"][::50, 0] = 1e9
    elif which == "gradient":
        dL[0, 40, 70], dL[1, 3, 3], dL[2, 80, 140] = float("inf"), float("nan"), 1e25
    else:
        case.bg = np.array([1e31, 0, np.inf], np.float32)
    outs = []
    for p, b in ((1, 64), (2, 64), (4, 64)):
        shapes(p, b)
        fwd = run_forward(ours, case)
        outs.append((fwd, run_backward(ours, case, fwd, dL)))
    f0, g0 = outs[0]
    for f, g in outs[1:]:
        for i in (1, 2, 3, 4, 5):
            assert torch.equal(f[i].nan_to_num(7.0) if f[i].is_floating_point() else f[i],
                               f0[i].nan_to_num(7.0) if f0[i].is_floating_point() else f0[i]), i
        for x, y in zip(g, g0):
            fine = torch.isfinite(y)
            assert torch.equal(fine, torch.isfinite(x))
            # the finite part without what overflow makes of the rest: rows whose values stay ordinary
            keep = fine & (y.abs() < 1e12)
            if keep.any():
                assert norm_rel(torch.where(keep, x, 0), torch.where(keep, y, 0)) <= 2e-5


_RULE = """
import sys
import numpy as np, torch
sys.path[:0] = {path!r}
from _helpers import Case, S, ours, run_forward
from filtergs_b200 import _lib
from filtergs_b200.batched import BatchedRasterizer, Camera

def case(P, scale, squeeze, W, H):
    sc, cam = S.small_scene(P=P, seed=77, W=W, H=H)
    sc["scales"] = (sc["scales"] * scale).astype(np.float32)
    sc["means3D"][: P // 2, :2] *= squeeze
    return Case(sc, cam)

small = case(30000, 0.05, 0.05, 250, 190)   # K <= 2 V: bands from 256 records on
large = case(9000, 1.0, 0.1, 333, 140)      # K > 2 V, one tile past 1024 records
plain = case(3000, 1.0, 1.0, 147, 133)      # no long tile
runs = [(c, st) for c in (small, large, plain) for st in (False, True)]
rule = [run_forward(ours, c, stats=st) for c, st in runs]

def batch(c):
    a = c.torch_inputs()
    cams = [Camera(c.cam.W, c.cam.H, c.cam.tanfovx, c.cam.tanfovy, a["viewmatrix"], a["projmatrix"], a["campos"])] * 3
    br = BatchedRasterizer(a["means3D"], a["opacity"], a["scales"], a["rotations"], cams, shs=a["sh"],
                           sh_degree=a["degree"], full_outputs=True)
    br.step()
    br.check()
    return [(br.images[v].clone(), br.point_id[v], br.point_weight_pixel[v], br.point_weight[v]) for v in (0, 2)]

batches = [batch(c) for c in (small, large)]
lengths = []
_lib.set_render_config(1, 64, 1, 64)
_lib.set_render_split(0, 0)
for (c, st), got in zip(runs, rule):
    want = run_forward(ours, c, stats=st)
    rg = ours.image_outputs(want[8], c.cam.W, c.cam.H)["ranges"]
    lengths.append((int((rg[:, 1] - rg[:, 0]).max()), int(want[0]), int((want[5] > 0).sum())))
    assert torch.equal(ours.image_outputs(got[8], c.cam.W, c.cam.H)["ranges"], rg)
    for i in (1, 2, 3, 4, 5):
        assert torch.equal(got[i], want[i]), i
    if st:
        assert np.allclose(got[9].numpy(), want[9].numpy(), rtol=1e-4, atol=1e-6)
for c, views in zip((small, large), batches):
    want = run_forward(ours, c)
    for view in views:
        for x, i in zip(view, (1, 2, 3, 4)):
            assert torch.equal(x, want[i]), i
n, K, V = lengths[0]
assert K <= 2 * V and n >= 256, lengths
n, K, V = lengths[2]
assert K > 2 * V and n >= max(1024, K // 592), lengths
assert lengths[4][0] < 1024, lengths
print("rule ok", lengths)
"""


def _own_process(code):
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", code.format(path=[here, os.path.dirname(here)])], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "rule ok" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]


def test_launch_rule_gives_the_same_bits(cuda):
    """The shapes and the long tiles the launch rule picks (before any set_render_* call, so in a process
    of its own) against one pixel per lane without bands: one view and batched, with and without
    statistics, with long tiles of small splats, of large ones, and without any."""
    _own_process(_RULE)


_BWD = """
import sys
import numpy as np, torch
sys.path[:0] = {path!r}
from _helpers import Case, S, ours, run_backward, run_forward
from filtergs_b200 import _lib

def case(P, W, H, **kw):
    sc, cam = S.small_scene(P=P, seed=78, W=W, H=H)
    sc["means3D"][: P // 2, :2] *= 0.1
    return Case(sc, cam, **kw)

cases = [case(1, 16, 16), case(60, 16, 16), case(9000, 333, 140, bg=np.array([0.2, 0.5, 0.9], np.float32)),
         case(3000, 147, 133)]
dL = [torch.randn(3, c.cam.H, c.cam.W, device="cuda", generator=torch.Generator("cuda").manual_seed(3)) for c in cases]
runs = [(c, d, m) for c, d in zip(cases, dL) for m in ("ref_compat", "consistent")]
grads = lambda: [run_backward(ours, c, run_forward(ours, c), d, backward_mode=m) for c, d, m in runs]  # noqa: E731
want = grads()
assert all(float(g[3].abs().sum()) > 0 for g in want)
for ppt, batch in ((2, 64), (2, 256), (4, 64), (4, 128)):
    _lib.set_render_config(2, 128, ppt, batch)
    for x, y in zip(grads(), want):
        for k, (u, v) in enumerate(zip(x, y)):
            assert torch.equal(u, v), (ppt, batch, k)
print("rule ok")
"""


def test_backward_has_the_same_bits_in_every_shape(cuda):
    """Gradients of the default backward shape and of others of 2 and 4 pixels per lane: one record, a
    last batch that is not full, lists of many batches, images whose edges cut tiles, either mode."""
    _own_process(_BWD)
