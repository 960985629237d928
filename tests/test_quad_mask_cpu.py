"""The compositing's record masks and warp sums, replayed on the CPU from their definitions in
csrc/fgs_common.cuh (quad_mask) and csrc/render.cu (warp_column_sum9).

* quad_mask against every pixel of a tile: a quad outside the mask must have no pixel whose
  alpha, evaluated in float32 as the compositing does, reaches 1/255 -- over round, elongated
  (up to 1000:1) and degenerate conics, opacities down to 1/255 and means inside and around the
  tile.  It must also leave out most of the quads that are not reached.
* warp_column_sum9: every stored component lands once, on the lane its table names, with the
  warp's total.
"""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "filtergs_b200", "csrc")
F = np.float32


def quad_mask(mx, my, a, b, c, o, tx0=F(0), ty0=F(0)):
    """quad_mask of tame records, in float32 (arrays of one value per record)."""
    with np.errstate(all="ignore"):
        ac = a * c
        det = ac - b * b
        t = F(1.02) * (F(2) * np.log(F(255) * o)) + F(0.1)
        s, ra = t / det, F(1) / a
        xmax, ymax = np.sqrt(s * c), np.sqrt(s * a)
        general = ~((a > 0) & (c > 0) & (det >= F(2.5e-4) * ac) & (xmax < 1e7) & (ymax < 1e7) & (ra < 1e30) &
                    (a * t < 1e30))
        ytop = -(b * xmax) / c
        X, at = tx0 - mx, a * t
        m = np.zeros(mx.shape, np.uint32)
        for r in range(2):
            lo, hi = np.maximum(ty0 + F(8 * r) - my, -ymax), np.minimum(ty0 + F(8 * r + 7) - my, ymax)
            yr, yl = np.minimum(np.maximum(ytop, lo), hi), np.minimum(np.maximum(-ytop, lo), hi)
            xr = (np.sqrt(np.maximum(at - det * yr * yr, F(0))) - b * yr) * ra + F(0.01)
            xl = -(np.sqrt(np.maximum(at - det * yl * yl, F(0))) + b * yl) * ra - F(0.01)
            rows = lo <= hi + F(0.01)
            for q in range(2):
                m |= np.where(rows & (xr >= X + F(8 * q)) & (xl <= X + F(8 * q + 7)), 1 << (2 * r + q), 0).astype(
                    np.uint32)
    return np.where(o >= F(1) / F(255), np.where(general, 15, m), 0)


def reached(mx, my, a, b, c, o):
    """The quads with a pixel of alpha >= 1/255, from the per-pixel evaluation in float32 (with
    its products rounded one by one: a fused product rounds less)."""
    y, x = np.meshgrid(np.arange(16, dtype=F), np.arange(16, dtype=F), indexing="ij")
    dx, dy = mx[:, None, None] - x, my[:, None, None] - y
    e = lambda v: v[:, None, None]  # noqa: E731
    with np.errstate(all="ignore"):
        power = F(-0.5) * (e(a) * dx * dx + e(c) * dy * dy) - e(b) * dx * dy
        ok = (power <= 0) & (np.minimum(F(0.99), e(o) * np.exp(power)) >= F(1) / F(255))
    q = ok.reshape(-1, 2, 8, 2, 8).any(axis=(2, 4))
    return sum(q[:, r, k].astype(np.uint32) << (2 * r + k) for r in range(2) for k in range(2))


def conics(n, aspect, seed):
    rng = np.random.default_rng(seed)
    s1 = np.exp(rng.uniform(np.log(0.3), np.log(40), n))
    s2 = np.maximum(s1 / np.exp(rng.uniform(0, np.log(aspect), n)), 0.02)
    th = rng.uniform(0, np.pi, n)
    u, v = np.cos(th), np.sin(th)
    ca, cb, cc = u * u * s1**2 + v * v * s2**2, u * v * (s1**2 - s2**2), v * v * s1**2 + u * u * s2**2
    det = ca * cc - cb * cb
    reach = 3.5 * s1
    return [np.asarray(z, F) for z in (rng.uniform(-1, 1, n) * reach + rng.uniform(0, 16, n),
                                       rng.uniform(-1, 1, n) * reach + rng.uniform(0, 16, n), cc / det, -cb / det,
                                       ca / det, np.exp(rng.uniform(np.log(1 / 255), 0, n)))]


@pytest.mark.parametrize("aspect", [1.2, 8, 60, 1000])
def test_quad_mask_covers_every_reached_pixel(aspect):
    rec = conics(60000, aspect, int(aspect * 10))
    m, r = quad_mask(*rec), reached(*rec)
    assert not np.any(r & ~m), int(np.count_nonzero(r & ~m))
    if aspect < 60:  # beyond, the degenerate conics keep every quad
        extra = sum(int(np.count_nonzero((m & ~r) >> k & 1)) for k in range(4))
        total = sum(int(np.count_nonzero(r >> k & 1)) for k in range(4))
        assert extra <= 0.15 * total, (extra, total)


def test_quad_mask_degenerate_conics():
    one = lambda v: np.full(6, v, F)  # noqa: E731
    a = np.array([1, -1, 0, np.nan, np.inf, 1], F)
    m = quad_mask(one(8), one(8), a, np.array([1, 0, 0, 0, 0, 2], F), one(1), one(0.5))
    assert np.all(m == 15)
    assert np.all(quad_mask(one(8), one(8), one(1), one(0), one(1), one(0.003)) == 0)  # below 1/255
    # the source states the constants replayed here
    src = open(os.path.join(CSRC, "fgs_common.cuh")).read()
    body = src[src.index("uint32_t quad_mask("):]
    for k in ("1.02f * (2.f * __logf(255.f * o)) + 0.1f", "det >= 2.5e-4f * ac", "+ 0.01f;", "lo <= hi + 0.01f"):
        assert k in body, k


def test_warp_column_sum9_places_every_total():
    rng = np.random.default_rng(5)
    lanes = np.arange(32)
    c, s = rng.standard_normal((3, 32)), rng.standard_normal((3, 32))
    dx = rng.standard_normal(8)[lanes & 7]          # one value per column of lanes
    want = [*c.sum(1), (s[0] * dx).sum(), s[1].sum(), (s[0] * dx * dx).sum(), (s[1] * dx).sum(), s[2].sum(),
            s[0].sum()]
    bit = lambda o: (lanes & o) != 0  # noqa: E731
    x = lambda v, o: v[lanes ^ o]  # noqa: E731
    v = [np.where(bit(16), s[i], c[i]) + x(np.where(bit(16), c[i], s[i]), 16) for i in range(3)]
    v = [t + x(t, 8) for t in v]
    e = bit(16) & bit(8)
    v = [np.where(e, v[0] * dx, v[0]), np.where(e, v[0] * dx * dx, v[1]), np.where(e, v[1] * dx, v[2])]
    r0 = np.where(bit(4), v[2], v[0]) + x(np.where(bit(4), v[0], v[2]), 4)
    r1 = v[1] + x(v[1], 4)
    t = np.where(bit(2), r1, r0) + x(np.where(bit(2), r0, r1), 2)
    t = t + x(t, 1)
    src = open(os.path.join(CSRC, "render.cu")).read()
    table = int(re.search(r"column_sum9_component.*?\(0x([0-9a-f]+)ull", src, re.S).group(1), 16)
    seen = []
    for lane in range(32):
        part, pick = (lane >> 3) & 3, 1 if lane & 2 else (2 if lane & 4 else 0)
        if lane & 1 or part == 1 or (lane & 2 and lane & 4):
            continue
        q = (table >> (4 * (3 * part + pick))) & 15
        seen.append(q)
        assert np.isclose(t[lane], want[q], rtol=1e-12), (lane, q)
    assert sorted(seen) == list(range(9))
