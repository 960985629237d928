"""GPU: the Adam step's row lists and item widths: SH rows whose length allows 16-byte items and ones
whose length does not, arrays that start off a 16-byte boundary, row counts around the block size, and
none, one, some or all rows visible -- against torch in float64.  The update's float32 arithmetic is a
handful of rounded operations per value (p, m and v; the activations one exponential or root more), so
values agree to 1e-5 of the step or of the value, and rows that were not visible keep their bits.
"""
import pytest
import torch
import torch.nn.functional as F

from filtergs_b200 import train as T

pytestmark = pytest.mark.gpu


def _off(t):
    """The same values in storage that starts 4 bytes past a 16-byte boundary."""
    o = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape)
    o.copy_(t)
    return o


@pytest.mark.parametrize("P,M,shift,share", [(257, 16, False, 0.3), (1, 16, False, 1.0), (256, 9, False, 1.0),
                                             (1000, 1, False, 0.5), (700, 4, True, 0.5), (513, 16, True, 0.02),
                                             (300, 4, False, 0.0)])
def test_adam_rows(cuda, P, M, shift, share):
    g = torch.Generator(device="cuda").manual_seed(P + M)
    n = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    st = T.TrainState(n(P, 3), n(P, 3) - 3, n(P, 4), n(P, 1), 0.1 * n(P, M, 3))
    keys = dict(xyz=(P, 3), shs=(P, M, 3), opacity=(P, 1), scale=(P, 3), rotation=(P, 4))
    st.m = {k: 0.1 * n(*s) for k, s in keys.items()}
    st.v = {k: n(*s).square() * 0.01 + 1e-4 for k, s in keys.items()}
    grad = {k: n(*s) for k, s in keys.items()}
    if shift:
        for name in ("xyz", "log_scale", "rot_raw", "opac_logit", "shs", "scale", "rot", "opac"):
            setattr(st, name, _off(getattr(st, name)))
        st.m, st.v, grad = ({k: _off(t) for k, t in d.items()} for d in (st.m, st.v, grad))
    st.step.fill_(41)
    vis = torch.rand(P, device="cuda", generator=g) < share
    st.flag.copy_(vis.to(torch.uint8))
    was = {k: t.clone() for k, t in st.raw().items()}
    act = dict(scale=st.scale.clone(), rot=st.rot.clone(), opac=st.opac.clone())
    want = {}
    d = {k: t.double() for k, t in grad.items()}
    s, q = act["opac"].double(), was["rotation"].double()
    nq, qh = q.norm(dim=-1, keepdim=True), act["rot"].double()
    d["opacity"] = d["opacity"] * s * (1 - s)
    d["scale"] = d["scale"] * act["scale"].double()
    d["rotation"] = (d["rotation"] - qh * (qh * d["rotation"]).sum(-1, keepdim=True)) / nq
    for lr, k in zip(st.lr, keys):
        m = 0.9 * st.m[k].double() + 0.1 * d[k]
        v = 0.999 * st.v[k].double() + 0.001 * d[k] ** 2
        p = was[k].double() - lr / (1 - 0.9 ** 42) * m / (v.sqrt() / (1 - 0.999 ** 42) ** 0.5 + 1e-15)
        on = vis.reshape([P] + [1] * (p.dim() - 1))
        want[k] = [torch.where(on, a, b.double()) for a, b in ((p, was[k]), (m, st.m[k]), (v, st.v[k]))]
    st.adam(grad["xyz"], grad["shs"], grad["opacity"], grad["scale"], grad["rotation"])
    assert int(st.step) == 42
    for k, p in st.raw().items():
        for got, w in zip((p, st.m[k], st.v[k]), want[k]):
            assert torch.allclose(got.double(), w, rtol=1e-5, atol=1e-6), k
        assert torch.equal(p[~vis], was[k][~vis]), k
    r = st.raw()
    for got, f, old in ((st.scale, torch.exp(r["scale"].double()), act["scale"]),
                        (st.rot, F.normalize(r["rotation"].double()), act["rot"]),
                        (st.opac, torch.sigmoid(r["opacity"].double()), act["opac"])):
        assert torch.allclose(got[vis].double(), f[vis], rtol=1e-5, atol=1e-7)
        assert torch.equal(got[~vis], old[~vis])
