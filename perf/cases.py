"""The workloads this framework's speed is measured on, through its public entry points.

  raster      GaussianRasterizer, one view: the forward alone (a viewer, an evaluation) or the
              forward and the backward through autograd (a training view)
  batched     BatchedRasterizer.step: forward + backward of many cameras of one Gaussian set
  lod         per-view selection from a Gaussian tree and the render of what it selects
  train_step  BatchedTrainer.step: render, loss, backward, Adam, densification statistics
  loss        Loss: L1 + SSIM and their gradient, and the loss value
  adam        TrainState.adam: one optimizer step on the rows that were visible

Scenes are synthetic: a cube of Gaussians in front of the camera, and an aerial town (ground plane
and building faces) of surfels whose sizes spread over a factor of 40, with 2 Gaussians per square
metre as in an aerial capture of 1 km^2 with 2,000,000 Gaussians; the larger a scene, the larger its
area.  A surfel's two in-plane axes are of similar length and its normal axis is a quarter of them:
needles of 100:1 would make the scale and rotation gradients differences of nearly equal terms, in
which float32 keeps three digits whatever sums them.
"""
import math

import numpy as np
import torch

from filtergs_b200 import lod, synthetic, train
from filtergs_b200.batched import BatchedRasterizer, Camera
from filtergs_b200.diff_gaussian_rasterization_wodilate import GaussianRasterizationSettings, GaussianRasterizer

DENSITY = 2.0                      # aerial Gaussians per square metre
SH_C0, SH_C1 = 0.28209479177387814, 0.4886025119029199
ACTIVE = 0.3                       # share of the rows an optimizer step finds visible (adam)


def listed():
    return [
        # the smallest view: a thumbnail or a unit-test scene, bounded by launches and host work;
        # statistics are on by default
        dict(name="raster_fwd_10k_256", kind="raster", scene="cube", P=10_000, W=256, H=256, D=3, stats=True,
             grad=False, use_filter=True, mode="ref_compat"),
        # the same size as a training view
        dict(name="raster_train_10k_256", kind="raster", scene="cube", P=10_000, W=256, H=256, D=3, stats=False,
             grad=True, use_filter=True, mode="ref_compat"),
        # a ragged image with precomputed colours, no dilation and the exact-gradient backward
        dict(name="raster_train_300k_ragged", kind="raster", scene="aerial", P=300_007, W=1237, H=823, D=-1,
             stats=False, grad=True, use_filter=False, mode="consistent"),
        # a viewer's frame and a training view of a large scene at full HD
        dict(name="raster_fwd_2M_1080p", kind="raster", scene="aerial", P=2_000_000, W=1920, H=1080, D=3,
             stats=False, grad=False, use_filter=True, mode="ref_compat"),
        dict(name="raster_train_2M_1080p", kind="raster", scene="aerial", P=2_000_000, W=1920, H=1080, D=3,
             stats=False, grad=True, use_filter=True, mode="ref_compat"),
        # many cameras a step: full HD throughout, and a mixture of smaller sizes
        dict(name="batched_2M_16x1080p", kind="batched", P=2_000_000, V=16, W=1920, H=1080, mixed=False, D=3),
        dict(name="batched_500k_6_mixed", kind="batched", P=500_000, V=6, W=1600, H=900, mixed=True, D=2),
        # a frame of a level-of-detail scene by either selection rule
        dict(name="lod_filtergs_8M_1080p", kind="lod", rule="filtergs", P=8_000_000, W=1920, H=1080),
        dict(name="lod_logcut_1M_720p", kind="lod", rule="logcut", P=1_000_000, W=1280, H=720),
        # one iteration of training, and its two dense parts by themselves
        dict(name="train_step_4M_4x900p", kind="train_step", P=4_000_000, V=4, W=1600, H=900),
        dict(name="loss_1080p", kind="loss", W=1920, H=1080, V=1),
        dict(name="adam_1M", kind="adam", P=1_000_000, M=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["raster", "raster", "raster", "batched", "batched", "lod", "train_step", "loss", "adam"])
    if kind == "raster":
        grad = rng.random() < 0.6
        scene = rng.choice(["cube", "aerial", "aerial"])
        P = _log(rng, 5_000, 60_000) if scene == "cube" else _log(rng, 20_000, 2_000_000)
        W = _log(rng, 96, 640) if scene == "cube" else _log(rng, 320, 1920)
        return dict(kind=kind, scene=scene, P=P, W=W, H=max(64, int(W * rng.uniform(0.5, 1.0))),
                    D=rng.choice([-1, 0, 1, 2, 3, 3, 3]), stats=(not grad) and rng.random() < 0.3, grad=grad,
                    use_filter=rng.random() < 0.8, mode=rng.choice(["ref_compat", "ref_compat", "consistent"]))
    if kind == "batched":
        W = _log(rng, 480, 1920)
        return dict(kind=kind, P=_log(rng, 100_000, 2_000_000), V=rng.randint(2, 10), W=W, H=int(W * 0.5625),
                    mixed=rng.random() < 0.5, D=rng.choice([1, 2, 3, 3]))
    if kind == "lod":
        W = _log(rng, 640, 1920)
        return dict(kind=kind, rule=rng.choice(["filtergs", "logcut"]), P=_log(rng, 300_000, 8_000_000), W=W,
                    H=int(W * rng.uniform(0.5, 0.75)))
    if kind == "train_step":
        W = _log(rng, 400, 1600)
        return dict(kind=kind, P=_log(rng, 200_000, 4_000_000), V=rng.randint(1, 4), W=W, H=int(W * 0.5625))
    if kind == "loss":
        W = _log(rng, 100, 1920)
        return dict(kind=kind, W=W, H=max(48, int(W * rng.uniform(0.5, 1.0))), V=rng.randint(1, 4))
    return dict(kind=kind, P=_log(rng, 50_000, 4_000_000), M=rng.choice([1, 4, 9, 16, 16]))


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 13)


def _uniform(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, device="cuda", generator=g)


def _normal(g, *n):
    return torch.randn(*n, device="cuda", generator=g)


def _quat_mul(a, b):
    w1, x1, y1, z1 = a.unbind(-1)
    w2, x2, y2, z2 = b.unbind(-1)
    return torch.stack([w1 * w2 - x1 * x2 - y1 * y2 - z1 * z2, w1 * x2 + x1 * w2 + y1 * z2 - z1 * y2,
                        w1 * y2 - x1 * z2 + y1 * w2 + z1 * x2, w1 * z2 + x1 * y2 - y1 * x2 + z1 * w2], -1)


def _sh(g, P, D):
    """SH rows for degree D, or precomputed colours (D = -1)."""
    if D < 0:
        return None, torch.rand(P, 3, device="cuda", generator=g)
    sh = 0.1 * _normal(g, P, (D + 1) ** 2, 3)
    sh[:, 0] = 0.5 * _normal(g, P, 3)
    return sh, None


def _cube(g, P, D):
    means = torch.stack([_uniform(g, P, -1, 1), _uniform(g, P, -1, 1), _uniform(g, P, 2, 6)], 1)
    rots = torch.nn.functional.normalize(_normal(g, P, 4))
    sh, colors = _sh(g, P, D)
    return dict(means=means, scales=torch.exp(-4 + 0.5 * _normal(g, P, 3)), rots=rots,
                opac=torch.sigmoid(_normal(g, P, 1)), sh=sh, colors=colors)


def _aerial(g, P, D):
    """Ground plane (70%) and the faces of boxes (30%) on a square of P / DENSITY square metres."""
    half = 0.5 * math.sqrt(P / DENSITY)
    nb = max(4, int(P / 5000))
    ground = torch.rand(P, device="cuda", generator=g) < 0.7
    means = torch.stack([_uniform(g, P, -half, half), _uniform(g, P, -half, half), 0.2 * _normal(g, P)], 1)
    b = torch.randint(nb, (P,), device="cuda", generator=g)
    c = _uniform(g, nb, -half, half)[b], _uniform(g, nb, -half, half)[b]
    s = _uniform(g, nb, 10, 60)[b], _uniform(g, nb, 10, 60)[b]
    h = _uniform(g, nb, 10, 120)[b]
    face = torch.randint(5, (P,), device="cuda", generator=g)
    u, v = _uniform(g, P, -0.5, 0.5), _uniform(g, P, 0, 1)
    roof = torch.stack([c[0] + u * s[0], c[1] + (v - 0.5) * s[1], h], 1)
    sx = torch.where(face == 1, 0.5, -0.5)
    sy = torch.where(face == 3, 0.5, -0.5)
    side_x = torch.stack([c[0] + sx * s[0], c[1] + u * s[1], v * h], 1)
    side_y = torch.stack([c[0] + u * s[0], c[1] + sy * s[1], v * h], 1)
    f = face[:, None]
    box = torch.where(f == 0, roof, torch.where(f <= 2, side_x, side_y))
    means = torch.where(ground[:, None], means, box)
    face = torch.where(ground, torch.zeros_like(face), face)
    r2 = math.sqrt(0.5)
    face_q = torch.tensor([[1, 0, 0, 0], [r2, 0, r2, 0], [r2, 0, -r2, 0], [r2, -r2, 0, 0], [r2, r2, 0, 0]],
                          device="cuda")
    yaw = _uniform(g, P, 0, math.pi)
    zero = torch.zeros_like(yaw)
    rots = _quat_mul(face_q[face], torch.stack([yaw.cos(), zero, zero, yaw.sin()], 1))
    ls = _uniform(g, P, math.log(0.1), math.log(4.0))[:, None] + 0.2 * _normal(g, P, 3)
    ls[:, 2] += math.log(0.25)
    sh, colors = _sh(g, P, D)
    return dict(means=means.contiguous(), scales=torch.exp(ls), rots=rots.contiguous(),
                opac=torch.sigmoid(1 + _normal(g, P, 1)), sh=sh, colors=colors)


def _camera(c):
    """A synthetic.Camera with its matrices on the GPU."""
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    return Camera(c.W, c.H, c.tanfovx, c.tanfovy, t(c.viewmatrix), t(c.projmatrix), t(c.campos))


def _aerial_cameras(seed, n, P, W, H, mixed=False):
    """Cameras over the town that look down at 30 to 75 degrees from 80 to 300 m (45 degrees and 150 m
    unless mixed); mixed sizes are W x H times 1, 0.83, 0.67 or 0.33."""
    rng = np.random.default_rng(int(seed) + 31)
    half = 0.5 * math.sqrt(P / DENSITY)
    cams = []
    for i in range(n):
        k = (1.0, 0.83, 0.67, 0.33)[i % 4] if mixed else 1.0
        w, h = max(64, int(W * k)), max(64, int(H * k))
        alt, pitch = (rng.uniform(80, 300), math.radians(rng.uniform(30, 75))) if mixed else (150.0, math.radians(45))
        yaw = rng.uniform(0, 2 * math.pi)
        at = np.array([rng.uniform(-0.5, 0.5) * half, rng.uniform(-0.5, 0.5) * half, 0.0])
        away = alt / math.tan(pitch)
        eye = at + np.array([-away * math.cos(yaw), -away * math.sin(yaw), alt])
        cams.append(_camera(synthetic.look_at_camera(eye, at, W=w, H=h, fx=1600.0 * w / 1920)))
    return cams


def _raster_inputs(case, seed):
    g = _gen(seed)
    P, W, H = case["P"], case["W"], case["H"]
    if case["scene"] == "cube":
        gs = _cube(g, P, case["D"])
        f = 300.0 * max(W, H) / 256
        cam = _camera(synthetic.identity_camera(W, H, fx=f, fy=f))
    else:
        gs = _aerial(g, P, case["D"])
        cam = _aerial_cameras(seed, 1, P, W, H)[0]
    return gs, cam, _normal(g, 3, H, W)


def _batched_inputs(case, seed):
    g = _gen(seed)
    gs = _aerial(g, case["P"], case["D"])
    cams = _aerial_cameras(seed, case["V"], case["P"], case["W"], case["H"], case["mixed"])
    return gs, cams, [_normal(g, 3, c.H, c.W) for c in cams]


def _tree(g, P):
    """A Gaussian tree in breadth-first order: branching min(Poisson(3) + 1, 8) up to 12 levels, child
    mean = parent + N(0, parent scale), child scale = half the parent's, the last level cut at P nodes."""
    half, roots, depth = 250.0 * math.sqrt(P / 8e6), 2, 12
    dev = "cuda"
    xyz = [torch.stack([_uniform(g, roots, -half, half), _uniform(g, roots, -half, half), _uniform(g, roots, 0, 20)], 1)]
    ls = [_uniform(g, roots, math.log(20), math.log(80))[:, None].expand(roots, 3)]
    parent, counts, total = [torch.full((roots,), -1, dtype=torch.long, device=dev)], [], roots
    anc = [torch.full((roots, depth + 1), -1, dtype=torch.int32, device=dev)]
    while total < P and len(counts) < depth:
        n = xyz[-1].shape[0]
        c = (torch.poisson(torch.full((n,), 3.0, device=dev), generator=g) + 1).clamp(max=8).long()
        end = c.cumsum(0)
        c = torch.minimum(c, (P - total - (end - c)).clamp(min=0))
        kids = int(c.sum())
        if kids == 0:
            break
        at = torch.repeat_interleave(torch.arange(n, device=dev), c)
        parent.append(at + (total - n))
        counts.append(c)
        xyz.append(xyz[-1][at] + _normal(g, kids, 3) * torch.exp(ls[-1][at]))
        ls.append(ls[-1][at] - math.log(2.0))
        a = anc[-1][at].clone()
        a[:, len(counts) - 1] = parent[-1].int()
        anc.append(a)
        total += kids
    parent, nc = torch.cat(parent), torch.cat(counts)
    nc = torch.cat([nc, torch.zeros(total - nc.numel(), dtype=torch.long, device=dev)])
    inner = nc > 0
    node_index = torch.where(inner, inner.long().cumsum(0) - 1, torch.full_like(nc, -1)).int()
    tree = torch.full((int(inner.sum()), 8), -1, dtype=torch.int32, device=dev)
    ids = torch.arange(roots, total, device=dev)
    first = (nc.cumsum(0) - nc + roots)[parent[roots:]]
    tree[node_index[parent[roots:]].long(), ids - first] = ids.int()
    return dict(xyz=torch.cat(xyz).contiguous(), log_scales=torch.cat(ls).contiguous(), rotations=_normal(g, total, 4),
                opacity_raw=1 + _normal(g, total, 1), features_dc=0.5 * _normal(g, total, 3),
                shs_rest=0.1 * _normal(g, total, 3, 3), node_index=node_index,
                ancestor_path=torch.cat(anc)[:, :len(counts) + 1].contiguous(), tree=tree,
                roots=torch.arange(roots, dtype=torch.int32, device=dev))


def _lod_inputs(case, seed):
    d = _tree(_gen(seed), case["P"])
    at = d["xyz"][0].double().cpu().numpy()
    at[2] = 0.0
    cam = synthetic.look_at_camera(at + np.array([150.0, 0.0, 150.0]), at, W=case["W"], H=case["H"],
                                   fx=1600.0 * case["W"] / 1920)
    return d, _camera(cam)


def _train_inputs(case, seed):
    """Raw parameters, the moments of an optimizer in mid-training, cameras and target images (renders of
    a perturbed copy)."""
    g = _gen(seed)
    P = case["P"]
    gs = _aerial(g, P, 3)
    raw = dict(xyz=gs["means"], log_scale=gs["scales"].log(), rot_raw=gs["rots"] * _uniform(g, P, 0.8, 1.2)[:, None],
               opac_logit=torch.logit(gs["opac"].clamp(1e-6, 1 - 1e-6)), shs=gs["sh"])
    shape = dict(xyz=(P, 3), shs=(P, 16, 3), opacity=(P, 1), scale=(P, 3), rotation=(P, 4))
    size = dict(xyz=1e-6, shs=1e-6, opacity=1e-5, scale=1e-5, rotation=1e-5)
    m = {k: size[k] * _normal(g, *s) for k, s in shape.items()}
    v = {k: (size[k] * (0.5 + torch.rand(*s, device="cuda", generator=g))).square() for k, s in shape.items()}
    cams = _aerial_cameras(seed, case["V"], P, case["W"], case["H"])
    targets = []
    moved = gs["means"] + 0.05 * _normal(g, P, 3)
    sh = gs["sh"].clone()
    sh[:, 0] += 0.1 * _normal(g, P, 3)
    with torch.no_grad():
        for c in cams:
            targets.append(_rasterizer(c, 3, "ref_compat")(moved, torch.zeros_like(moved), gs["opac"], shs=sh,
                                                           scales=gs["scales"], rotations=gs["rots"])[0])
    return raw, m, v, cams, targets


LATE_LR = tuple(0.01 * x for x in train.DEFAULT_LR)  # the end of the learning-rate schedule
STEP0 = 5000


def _train_state(raw, m, v):
    st = train.TrainState(raw["xyz"], raw["log_scale"], raw["rot_raw"], raw["opac_logit"], raw["shs"], lr=LATE_LR)
    for k in m:
        st.m[k].copy_(m[k])
        st.v[k].copy_(v[k])
    st.step.fill_(STEP0)
    return st


def _adam_inputs(case, seed):
    """Raw parameters, moments and gradients; the visible rows lie in runs, as the points of a capture do."""
    g = _gen(seed)
    P, M = case["P"], case["M"]
    raw = dict(xyz=100 * _normal(g, P, 3), log_scale=-3 + _normal(g, P, 3), rot_raw=_normal(g, P, 4),
               opac_logit=_normal(g, P, 1), shs=0.1 * _normal(g, P, M, 3))
    shape = dict(xyz=(P, 3), shs=(P, M, 3), opacity=(P, 1), scale=(P, 3), rotation=(P, 4))
    m = {k: 1e-4 * _normal(g, *s) for k, s in shape.items()}
    v = {k: (1e-4 * (0.5 + torch.rand(*s, device="cuda", generator=g))).square() for k, s in shape.items()}
    grad = {k: 1e-4 * _normal(g, *s) for k, s in shape.items()}
    run = torch.rand((P + 63) // 64, device="cuda", generator=g) < 0.5
    flag = run.repeat_interleave(64)[:P] & (torch.rand(P, device="cuda", generator=g) < 2 * ACTIVE)
    return raw, m, v, grad, flag.to(torch.uint8)


def _loss_inputs(case, seed):
    g = _gen(seed)
    W, H = case["W"], case["H"]
    targets, preds = [], []
    for _ in range(case["V"]):
        coarse = torch.rand(1, 3, H // 16 + 2, W // 16 + 2, device="cuda", generator=g)
        t = torch.nn.functional.interpolate(coarse, size=(H, W), mode="bilinear")[0]
        t = (t + 0.05 * _normal(g, 3, H, W)).clamp(0, 1).contiguous()
        targets.append(t)
        preds.append((t + 0.05 * _normal(g, 3, H, W)).contiguous())
    return preds, targets


def _rasterizer(cam, D, mode, stats=False):
    return GaussianRasterizer(GaussianRasterizationSettings(
        image_height=cam.H, image_width=cam.W, tanfovx=cam.tanfovx, tanfovy=cam.tanfovy,
        bg=torch.zeros(3, device="cuda"), scale_modifier=1.0, viewmatrix=cam.viewmatrix, projmatrix=cam.projmatrix,
        sh_degree=max(D, 0), campos=cam.campos, prefiltered=False, debug=False, ogfs_enable_stats=stats,
        backward_mode=mode))


# ---------------------------------------------------------------- prepare and run
def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "raster":
        gs, cam, dL = _raster_inputs(case, seed)
        leaf = {k: t for k, t in gs.items() if t is not None}
        leaf["means2D"] = torch.zeros_like(gs["means"])
        if case["grad"]:
            leaf = {k: t.requires_grad_(True) for k, t in leaf.items()}
        s.update(leaf=leaf, dL=dL, rasterizer=_rasterizer(cam, case["D"], case["mode"], case["stats"]))
    elif kind == "batched":
        gs, cams, dLs = _batched_inputs(case, seed)
        s["br"] = BatchedRasterizer(gs["means"], gs["opac"], gs["scales"], gs["rots"], cams, shs=gs["sh"],
                                    sh_degree=case["D"])
        s["br"].set_io_many(list(range(len(cams))), list(s["br"].images), dLs)
    elif kind == "lod":
        d, cam = _lod_inputs(case, seed)
        s.update(scene=lod.TreeScene.from_arrays(d), cam=cam, bg=torch.zeros(3, device="cuda"))
    elif kind == "train_step":
        raw, m, v, cams, targets = _train_inputs(case, seed)
        s["state"] = _train_state(raw, m, v)
        s["trainer"] = train.BatchedTrainer(s["state"], cams, targets)
    elif kind == "loss":
        s["preds"], s["targets"] = _loss_inputs(case, seed)
        s["grads"] = [torch.empty_like(p) for p in s["preds"]]
        s["loss"] = train.Loss([(case["W"], case["H"])] * case["V"], "cuda")
    else:
        raw, m, v, grad, flag = _adam_inputs(case, seed)
        s["state"] = _train_state(raw, m, v)
        s["state"].flag.copy_(flag)
        s["grad"] = grad
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "raster":
        t = s["leaf"]
        with torch.set_grad_enabled(case["grad"]):
            color, radii, pid, pwp, pw = s["rasterizer"](t["means"], t["means2D"], t["opac"], shs=t.get("sh"),
                                                         colors_precomp=t.get("colors"), scales=t["scales"],
                                                         rotations=t["rots"], use_filter=case["use_filter"])
        out = dict(color=color, radii=radii, point_id=pid, point_weight_pixel=pwp, point_weight=pw)
        if case["grad"]:
            names = list(t)
            out["grad"] = dict(zip(names, torch.autograd.grad(color, [t[k] for k in names], s["dL"])))
        return out
    if kind == "batched":
        s["br"].step()
        return dict(images=s["br"].images, radii=s["br"].radii, grad=s["br"].grad)
    if kind == "lod":
        sc, cam = s["scene"], s["cam"]
        nodes = {}
        if case["rule"] == "filtergs":
            idx, cnt, mask, radius, depth = lod.select_filtergs(sc, cam.viewmatrix, cam.projmatrix, cam, 1.5, 0.1, 700.0)
            nodes = dict(mask=mask, radius=radius, depth=depth)
        else:
            idx, cnt = lod.select_logcut(sc, cam.viewmatrix, cam.projmatrix, cam, 1.5, 1.0)
        # (the outputs with a row per selected node are as long as the selection: not the same for other inputs)
        K, color, pid, pwp = lod.render_selected(sc, idx, cnt, cam.viewmatrix, cam.projmatrix, cam.campos, cam,
                                                 s["bg"])[:4]
        return dict(pairs=K, selected=cnt, color=color, point_id=pid, point_weight_pixel=pwp, **nodes)
    st = s.get("state")
    if kind == "train_step":
        s["trainer"].step()
        return dict(grad=s["trainer"].br.grad, images=s["trainer"].br.images, raw=st.raw(), m=st.m, v=st.v,
                    scale=st.scale, rot=st.rot, opac=st.opac, grad_sum=st.grad_sum, vis_count=st.vis_count,
                    flag=st.flag)
    if kind == "loss":
        s["loss"](s["preds"], s["targets"], s["grads"])
        return dict(grads=s["grads"], value=s["loss"].value())
    g = s["grad"]
    st.adam(g["xyz"], g["shs"], g["opacity"], g["scale"], g["rotation"])
    return dict(raw=st.raw(), m=st.m, v=st.v, scale=st.scale, rot=st.rot, opac=st.opac)


def work(case):
    """Inputs read once and outputs written once; for compositing about 1.2 (tile, Gaussian) pairs per
    pixel of an aerial view, and of a pair's 256 pixels about 100 evaluated, at 40 operations forward and
    60 more backward."""
    kind = case["kind"]
    n = case.get("W", 0) * case.get("H", 0)
    P = case.get("P", 0)
    D = case.get("D", 3)
    sh = 4 * 3 * (D + 1) ** 2 if D >= 0 else 12
    if kind == "raster":
        pairs = 1.2 * n if case["scene"] == "aerial" else 6.0 * P
        seen = min(P, 0.06 * n) if case["scene"] == "aerial" else P
        b = 44 * P + 8 * P + sh * seen + 20 * n
        f = pairs * 100 * 40
        if case["grad"]:
            b += 12 * n + P * (12 + 12 + 12 + 16 + 4 + sh)
            f += pairs * 100 * 60
        return dict(bytes=b, flops=f)
    if kind == "batched":
        V, k = case["V"], (0.55 if case["mixed"] else 1.0)
        return dict(bytes=44 * P + P * (4 * V + 36 + 2 * sh) + 24 * n * V * k, flops=1.2 * n * V * k * 100 * 100)
    if kind == "lod":
        # the parameters, ancestors and node outputs of every node, or the nodes above the cut; about 0.4 P rows selected
        return dict(bytes=(80 if case["rule"] == "filtergs" else 60) * P + 0.4 * P * 80 + 20 * n,
                    flops=1.0 * P * 100 * 40)
    if kind == "train_step":
        V = case["V"]
        seen = min(P, 0.06 * n * V)
        return dict(bytes=44 * P + seen * 59 * 4 * 7 + P * 59 * 4 + n * V * 12 * 4, flops=1.2 * n * V * 100 * 100)
    if kind == "loss":
        return dict(bytes=36 * n * case["V"], flops=3 * n * case["V"] * 2 * 22 * 8)
    floats = 11 + 3 * case["M"]
    return dict(bytes=P + ACTIVE * P * (floats * 4 * 7 + 32), flops=ACTIVE * P * floats * 12)


# ---------------------------------------------------------------- the same values in 64 bits
def _cov3d(scales, rots):
    r, x, y, z = rots.unbind(-1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - r * z), 2 * (x * z + r * y),
                     2 * (x * y + r * z), 1 - 2 * (x * x + z * z), 2 * (y * z - r * x),
                     2 * (x * z - r * y), 2 * (y * z + r * x), 1 - 2 * (x * x + y * y)], -1).reshape(-1, 3, 3)
    M = R * scales[:, None, :]
    return M @ M.transpose(1, 2)


def _hom(means, m):
    return torch.cat([means, torch.ones_like(means[:, :1])], 1) @ m.double().reshape(4, 4)


def _cov2d(means, cov3d, cam, exact_clamp):
    """The projected covariance (a, b, c) without dilation.  exact_clamp: a clamped x / z keeps its
    dependence on z (the exact derivative); otherwise it is a constant, as in the reference's backward."""
    t = _hom(means, cam.viewmatrix)
    fx, fy = cam.W / (2 * cam.tanfovx), cam.H / (2 * cam.tanfovy)
    z = t[:, 2]

    def clamped(u, tan):
        lim = 1.3 * tan
        over = (u / z).abs() > lim
        at = torch.sign(u / z).detach() * lim * z
        return torch.where(over, at if exact_clamp else at.detach(), u)

    tx, ty = clamped(t[:, 0], cam.tanfovx), clamped(t[:, 1], cam.tanfovy)
    o = torch.zeros_like(z)
    J = torch.stack([fx / z, o, -fx * tx / (z * z), o, fy / z, -fy * ty / (z * z)], -1).reshape(-1, 2, 3)
    A = J @ cam.viewmatrix.double().reshape(4, 4)[:3, :3].T
    S = A @ cov3d @ A.transpose(1, 2)
    return torch.stack([S[:, 0, 0], S[:, 0, 1], S[:, 1, 1]], -1)


def _conic(abc):
    a, b, c = abc.unbind(-1)
    return torch.stack([c, -b, a], -1) / (a * c - b * b)[:, None]


def _sh_color(sh, D, means, campos):
    res = SH_C0 * sh[:, 0]
    if D > 0:
        d = torch.nn.functional.normalize(means - campos.double()[None], dim=-1)
        x, y, z = d[:, 0:1], d[:, 1:2], d[:, 2:3]
        res = res - SH_C1 * y * sh[:, 1] + SH_C1 * z * sh[:, 2] - SH_C1 * x * sh[:, 3]
        if D > 1:
            c = (1.0925484305920792, 0.31539156525252005, 0.5462742152960396)
            xx, yy, zz = x * x, y * y, z * z
            res = (res + c[0] * x * y * sh[:, 4] - c[0] * y * z * sh[:, 5] + c[1] * (2 * zz - xx - yy) * sh[:, 6] -
                   c[0] * x * z * sh[:, 7] + c[2] * (xx - yy) * sh[:, 8])
            if D > 2:
                res = (res - 0.5900435899266435 * y * (3 * xx - yy) * sh[:, 9] +
                       2.890611442640554 * x * y * z * sh[:, 10] -
                       0.4570457994644658 * y * (4 * zz - xx - yy) * sh[:, 11] +
                       0.3731763325901154 * z * (2 * zz - 3 * xx - 3 * yy) * sh[:, 12] -
                       0.4570457994644658 * x * (4 * zz - xx - yy) * sh[:, 13] +
                       1.445305721320277 * z * (xx - yy) * sh[:, 14] -
                       0.5900435899266435 * x * (xx - 3 * yy) * sh[:, 15])
    return (res + 0.5).clamp(min=0)


def _lists(px, radius, depth, vis, W, H):
    """Per tile the ids of the Gaussians that reach it, front to back: (ids of all pairs, begin [T + 1])."""
    gx, gy = (W + 15) // 16, (H + 15) // 16
    lo = lambda v, n: torch.trunc(v / 16).clamp(0, n).long()  # noqa: E731
    x0, x1 = lo(px[:, 0] - radius, gx), lo(px[:, 0] + radius + 15, gx)
    y0, y1 = lo(px[:, 1] - radius, gy), lo(px[:, 1] + radius + 15, gy)
    n = torch.where(vis, (x1 - x0) * (y1 - y0), 0)
    ids = torch.nonzero(n > 0)[:, 0]
    ids = ids[torch.sort(depth[ids].float(), stable=True)[1]]
    n = n[ids]
    rep = torch.repeat_interleave(torch.arange(ids.numel(), device=px.device), n)
    k = torch.arange(rep.numel(), device=px.device) - (n.cumsum(0) - n)[rep]
    w = (x1 - x0)[ids][rep]
    tile = (y0[ids][rep] + k // w) * gx + x0[ids][rep] + k % w
    tile, order = torch.sort(tile, stable=True)
    begin = torch.searchsorted(tile, torch.arange(gx * gy + 1, device=px.device))
    return ids[rep][order], begin


def _composite(px, conic, opac, color, ids, begin, W, H, dL, clamp_grad):
    """Image, largest weight per pixel and per Gaussian, and the gradients w.r.t. px, conic, opac, color."""
    dev = px.device
    P, gx, gy = px.shape[0], (W + 15) // 16, (H + 15) // 16
    feat = torch.cat([px, conic, opac, color], 1)
    image = torch.zeros(gy * 16, gx * 16, 3, dtype=torch.float64, device=dev)
    best = torch.zeros(gy * 16, gx * 16, dtype=torch.float64, device=dev)
    weight = torch.zeros(P, dtype=torch.float64, device=dev)
    grad = torch.zeros_like(feat) if dL is not None else None
    if dL is not None:
        up = torch.zeros_like(image)
        up[:H, :W] = dL.double().permute(1, 2, 0)
    length = begin[1:] - begin[:-1]
    order = torch.argsort(length)
    sizes = length[order].tolist()
    at = next((i for i, v in enumerate(sizes) if v > 0), len(sizes))
    iy, ix = torch.meshgrid(torch.arange(16, device=dev), torch.arange(16, device=dev), indexing="ij")
    while at < len(sizes):
        end = at + 1
        while end < len(sizes) and (end + 1 - at) * sizes[end] * 256 <= 32_000_000:
            end += 1
        tiles, L = order[at:end], sizes[end - 1]
        at = end
        k = torch.arange(L, device=dev)[None]
        have = k < length[tiles][:, None]
        gid = torch.where(have, ids[(begin[tiles][:, None] + k).clamp(max=ids.numel() - 1)], 0)
        f = feat[gid].requires_grad_(dL is not None)
        ty, tx = (tiles // gx * 16)[:, None] + iy.reshape(1, -1), (tiles % gx * 16)[:, None] + ix.reshape(1, -1)
        with torch.set_grad_enabled(dL is not None):
            q = f[:, None]                                   # [tiles, 1, L, 9]
            dx, dy = q[..., 0] - tx[..., None], q[..., 1] - ty[..., None]
            power = -0.5 * (q[..., 2] * dx * dx + q[..., 4] * dy * dy) - q[..., 3] * dx * dy
            full = q[..., 5] * torch.exp(power)
            alpha = full.clamp(max=0.99)
            if not clamp_grad:
                alpha = full + (alpha - full).detach()
            ok = have[:, None] & (power <= 0) & (alpha >= 1 / 255)
            alpha = torch.where(ok, alpha, 0.0)
            ok = ok & (torch.cumprod(1 - alpha.detach(), -1) >= 1e-4)
            alpha = torch.where(ok, alpha, 0.0)
            T = torch.cumprod(1 - alpha, -1)
            w = alpha * torch.cat([torch.ones_like(T[..., :1]), T[..., :-1]], -1)
            out = w @ f[:, :, 6:9]
        image[ty, tx] = out.detach()
        wd = torch.where(((ty < H) & (tx < W))[..., None], w.detach(), 0.0)
        best[ty, tx] = wd.amax(-1)
        weight.scatter_reduce_(0, gid.reshape(-1), torch.where(have, wd.amax(1), 0.0).reshape(-1), "amax")
        if dL is not None:
            gf, = torch.autograd.grad(out, f, up[ty, tx])
            grad.index_add_(0, gid.reshape(-1), gf.reshape(-1, 9))
    return image[:H, :W].permute(2, 0, 1), best[:H, :W], weight, grad


def _exact_view(gs, cam, D, use_filter, mode, dL):
    """One view of Gaussians given in float64, and with dL the gradients w.r.t. the inputs."""
    x = {k: t.detach().double().requires_grad_(dL is not None) for k, t in gs.items() if t is not None}
    W, H, consistent = cam.W, cam.H, mode == "consistent"
    with torch.set_grad_enabled(dL is not None):
        z = _hom(x["means"], cam.viewmatrix)[:, 2]
        hom = _hom(x["means"], cam.projmatrix)
        ndc = hom[:, :2] / (hom[:, 3:] + 1e-7)
        px = torch.stack([((ndc[:, 0] + 1) * W - 1) / 2, ((ndc[:, 1] + 1) * H - 1) / 2], -1)
        cov = _cov2d(x["means"], _cov3d(x["scales"], x["rots"]), cam, consistent)
        dil = torch.stack([cov[:, 0].clamp(min=0.3), cov[:, 1], cov[:, 2].clamp(min=0.3)], -1) if use_filter else cov
        color = x["colors"] if "colors" in x else _sh_color(x["sh"], D, x["means"], cam.campos)
    with torch.no_grad():
        a, b, c = dil.unbind(-1)
        det = a * c - b * b
        vis = (z > 0.2) & (det != 0)
        lg = math.log(min(max(1 / 255 + 0.2 * ((1 - (254 / 255) ** 256) - 1 / 255), 1 / 255), 0.2))
        mid = 0.5 * (a + c)
        lam = (mid + (mid * mid - det).clamp(min=0).sqrt()).clamp(min=1e-6)
        base = 3 * lam.sqrt()
        opac = x["opac"][:, 0].clamp(min=1e-6)
        r = torch.maximum(torch.minimum((2 * (opac.log() - lg).clamp(min=0.05) * lam).sqrt(), base), 0.7 * base)
        r = torch.ceil(r + 1).clamp(min=1)
        ids, begin = _lists(px, r, z, vis, W, H)
        conic = torch.where(vis[:, None], _conic(dil), 0.0)
    image, best, weight, grad = _composite(px.detach(), conic, opac[:, None].detach(), color.detach(), ids, begin, W,
                                           H, dL, consistent)
    if dL is None:
        return image, best, weight, None
    seen = torch.zeros(z.shape[0], dtype=torch.bool, device=z.device)
    seen[ids] = True
    # the covariance's gradient: of the forward as it is, or the reference's (+0.3, 1 / (det^2 + 1e-7))
    abc = (dil if consistent else cov + torch.tensor([0.3, 0.0, 0.3], device=z.device)).detach()
    abc = torch.where(seen[:, None], abc, torch.tensor([1.0, 0.0, 1.0], dtype=torch.float64, device=z.device))
    leaf = abc.requires_grad_(True)
    g_abc, = torch.autograd.grad(_conic(leaf), leaf, grad[:, 2:5])
    if not consistent:
        d2 = (abc[:, 0] * abc[:, 2] - abc[:, 1] ** 2).detach().square()
        g_abc = g_abc * (d2 / (d2 + 1e-7))[:, None]
    keep = torch.nonzero(seen)[:, 0]
    names = [k for k in x if k != "opac"]
    g = torch.autograd.grad([px[keep], (dil if consistent else cov)[keep], color[keep]], [x[k] for k in names],
                            [grad[keep, 0:2], g_abc[keep], grad[keep, 6:9]], allow_unused=True)
    g = {k: torch.nan_to_num(t) for k, t in zip(names, g)}
    g["opac"] = grad[:, 5:6]
    g["means2D"] = torch.cat([grad[:, 0:2] * torch.tensor([0.5 * W, 0.5 * H], device=z.device),
                              torch.zeros_like(grad[:, :1])], 1)
    return image, best, weight, g


def _select(d, cam, rule):
    """The node ids a selection rule keeps and every node's radius and depth, from values in float64."""
    x = {k: t.double() for k, t in d.items() if t.is_floating_point()}
    hom = _hom(x["xyz"], cam.projmatrix)
    ndc = hom[:, :3] / (hom[:, 3:] + 1e-7)
    scales, rots = torch.exp(x["log_scales"]), torch.nn.functional.normalize(x["rotations"])
    a, b, c = _cov2d(x["xyz"], _cov3d(scales, rots), cam, False).unbind(-1)
    a, c = a.clamp(min=0.3), c.clamp(min=0.3)
    det, mid = a * c - b * b, 0.5 * (a + c)
    radius = 3 * (mid + (mid * mid - det).clamp(min=0.1).sqrt()).sqrt()
    leaf = d["node_index"] == -1
    if rule == "filtergs":
        seen = (ndc[:, 2] > 0) & (ndc[:, 2] < 1) & (ndc[:, :2].abs() < 1.1).all(1)
        radius = torch.where(seen & (det > 0), radius, 0.0)
        small = (~leaf) & (radius > 0) & (radius <= 1.5)
        anc = d["ancestor_path"].long()
        under = (small[anc.clamp(min=0)] & (anc >= 0)).any(1)
        keep = seen & torch.where(leaf, ~under, radius <= 1.5) & (radius <= 700)
        return torch.nonzero(keep)[:, 0], radius, ndc[:, 2]
    radius = torch.where((ndc[:, :2].abs() <= 1.3).all(1) & (det != 0), radius, 0.0)
    out, front = [], d["roots"].long()
    while front.numel():
        stop = (radius[front] < 1.5) | leaf[front]
        out.append(front[stop])
        kids = d["tree"][d["node_index"][front[~stop]].long()].reshape(-1).long()
        front = kids[kids >= 0]
    ids = torch.cat(out)
    return ids[(radius[ids] >= 1) & (torch.sigmoid(x["opacity_raw"][ids, 0]) >= 1 / 255)], radius, ndc[:, 2]


def _exact_lod(d, cam, rule):
    ids, radius, depth = _select(d, cam, rule)
    x = {k: d[k][ids].double() for k in ("xyz", "log_scales", "rotations", "opacity_raw", "features_dc", "shs_rest")}
    v = torch.nn.functional.normalize(x["xyz"] - cam.campos.double()[None], dim=-1)
    rest = x["shs_rest"]
    color = (x["features_dc"] * SH_C0 + 0.5 - SH_C1 * v[:, 1:2] * rest[:, 0] + SH_C1 * v[:, 2:3] * rest[:, 1] -
             SH_C1 * v[:, 0:1] * rest[:, 2])
    gs = dict(means=x["xyz"], scales=torch.exp(x["log_scales"]), rots=torch.nn.functional.normalize(x["rotations"]),
              opac=torch.sigmoid(x["opacity_raw"]), colors=color)
    image, best, _, _ = _exact_view(gs, cam, -1, True, "ref_compat", None)
    return image, best, radius, depth


def _exact_loss(preds, targets):
    """(value, gradient per image) of 0.8 L1 + 0.2 (1 - SSIM) over all images."""
    t = torch.arange(11, dtype=torch.float64, device=preds[0].device) - 5
    w = torch.exp(-t * t / 4.5).float().double()
    w = w / w.sum()
    k = (w[:, None] * w[None]).expand(3, 1, 11, 11).contiguous()
    l1 = sum(p.numel() for p in preds)
    ns = sum(3 * (p.shape[1] - 10) * (p.shape[2] - 10) for p in preds)
    value, grads = 0.2, []
    mean = lambda v: torch.nn.functional.conv2d(v[None], k, groups=3)  # noqa: E731
    for p, y in zip(preds, targets):
        x, y = p.detach().double().requires_grad_(True), y.double()
        with torch.enable_grad():
            m1, m2 = mean(x), mean(y)
            s11, s22, s12 = mean(x * x) - m1 * m1, mean(y * y) - m2 * m2, mean(x * y) - m1 * m2
            ssim = ((2 * m1 * m2 + 1e-4) * (2 * s12 + 9e-4)) / ((m1 * m1 + m2 * m2 + 1e-4) * (s11 + s22 + 9e-4))
            part = 0.8 * (x - y).abs().sum() / l1 - 0.2 * ssim.sum() / ns
            grads.append(torch.autograd.grad(part, x)[0])
        value = value + float(part.detach())
    return value, grads


def _exact_adam(raw, m, v, grad, rows):
    """The state after one step on the given rows; grad is w.r.t. the activated values."""
    p = dict(xyz=raw["xyz"], shs=raw["shs"], opacity=raw["opac_logit"], scale=raw["log_scale"],
             rotation=raw["rot_raw"])
    p = {k: t.detach().double() for k, t in p.items()}
    q = p["rotation"]
    n = q.norm(dim=-1, keepdim=True)
    s = torch.sigmoid(p["opacity"])
    g = {k: t.double() for k, t in grad.items()}
    g["opacity"] = g["opacity"] * s * (1 - s)
    g["scale"] = g["scale"] * torch.exp(p["scale"])
    g["rotation"] = (g["rotation"] - q / n * ((q / n) * g["rotation"]).sum(-1, keepdim=True)) / n
    t, out = STEP0 + 1, dict(raw={}, m={}, v={})
    for lr, k in zip(LATE_LR, ("xyz", "shs", "opacity", "scale", "rotation")):
        on = rows.reshape([-1] + [1] * (p[k].dim() - 1))
        m1 = 0.9 * m[k].double() + 0.1 * g[k]
        v1 = 0.999 * v[k].double() + 0.001 * g[k] ** 2
        to = p[k] - lr / (1 - 0.9 ** t) * m1 / (v1.sqrt() / math.sqrt(1 - 0.999 ** t) + 1e-15)
        for name, new, old in (("raw", to, p[k]), ("m", m1, m[k].double()), ("v", v1, v[k].double())):
            out[name][k] = torch.where(on, new, old)
    r = out["raw"]
    out.update(scale=torch.exp(r["scale"]), rot=torch.nn.functional.normalize(r["rotation"]),
               opac=torch.sigmoid(r["opacity"]))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "raster":
        gs, cam, dL = _raster_inputs(case, seed)
        image, best, weight, g = _exact_view(gs, cam, case["D"], case["use_filter"], case["mode"],
                                             dL if case["grad"] else None)
        out = dict(color=image, radii=None, point_id=None, point_weight_pixel=best, point_weight=weight)
        if case["grad"]:
            out["grad"] = g
        return out
    if kind == "batched":
        if case["V"] * case["W"] * case["H"] > 40_000_000:
            return None
        gs, cams, dLs = _batched_inputs(case, seed)
        images, total = [], None
        for cam, dL in zip(cams, dLs):
            image, _, _, g = _exact_view(gs, cam, case["D"], True, "ref_compat", dL)
            images.append(image)
            total = g if total is None else {k: total[k] + g[k] for k in g}
        return dict(images=images, radii=None, grad=dict(means3D=total["means"], opacity=total["opac"],
                                                         sh=total["sh"], scales=total["scales"],
                                                         rotations=total["rots"]))
    if kind == "lod":
        d, cam = _lod_inputs(case, seed)
        image, best, radius, depth = _exact_lod(d, cam, case["rule"])
        nodes = dict(mask=None, radius=radius, depth=depth) if case["rule"] == "filtergs" else {}
        return dict(pairs=None, selected=None, color=image, point_id=None, point_weight_pixel=best, **nodes)
    if kind == "train_step":
        raw, m, v, cams, targets = _train_inputs(case, seed)
        gs = dict(means=raw["xyz"].double(), scales=torch.exp(raw["log_scale"].double()),
                  rots=torch.nn.functional.normalize(raw["rot_raw"].double()),
                  opac=torch.sigmoid(raw["opac_logit"].double()), sh=raw["shs"].double())
        images = [_exact_view(gs, c, 3, True, "ref_compat", None)[0] for c in cams]
        dLs = _exact_loss(images, targets)[1]
        total, seen, moved = None, 0, 0.0
        for c, dL in zip(cams, dLs):
            _, _, weight, g = _exact_view(gs, c, 3, True, "ref_compat", dL)
            size = g.pop("means2D")[:, :2].norm(dim=-1)
            moved = moved + size
            seen = seen + (weight > 0).long()
            total = g if total is None else {k: total[k] + g[k] for k in g}
        # rows no view composites have zero gradients but may count as visible: their moments decay, which
        # only the framework's own visibility tells, so only the gradients and images have a value here
        return dict(grad=dict(means3D=total["means"], opacity=total["opac"], sh=total["sh"], scales=total["scales"],
                              rotations=total["rots"]), images=images, raw=None, m=None, v=None, scale=None, rot=None,
                    opac=None, grad_sum=moved, vis_count=None, flag=None)
    if kind == "loss":
        preds, targets = _loss_inputs(case, seed)
        value, grads = _exact_loss(preds, targets)
        return dict(grads=grads, value=value)
    raw, m, v, grad, flag = _adam_inputs(case, seed)
    return _exact_adam(raw, m, v, grad, flag.bool())
