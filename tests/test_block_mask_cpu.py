"""The compositing's record masks and warp sums, replayed on the CPU from their definitions in
csrc/fgs_common.cuh (block_mask) and csrc/render.cu (add_step_sums).

* block_mask against every pixel of a tile: an 8x4 block outside the mask must have no pixel whose
  alpha, evaluated in float32 as the compositing does, reaches 1/255 -- over round, elongated
  (up to 1000:1) and degenerate conics, opacities down to 1/255 and means inside and around the
  tile.  It must also leave out most of the blocks that are not reached.
* add_step_sums: the totals of four steps, each with the bits of warp_transpose_sum9.
"""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "filtergs_b200", "csrc")
F = np.float32


def block_mask(mx, my, a, b, c, o, tx0=F(0), ty0=F(0)):
    """block_mask of tame records, in float32 (arrays of one value per record)."""
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
        for r in range(4):
            lo, hi = np.maximum(ty0 + F(4 * r) - my, -ymax), np.minimum(ty0 + F(4 * r + 3) - my, ymax)
            yr, yl = np.minimum(np.maximum(ytop, lo), hi), np.minimum(np.maximum(-ytop, lo), hi)
            xr = (np.sqrt(np.maximum(at - det * yr * yr, F(0))) - b * yr) * ra + F(0.01)
            xl = -(np.sqrt(np.maximum(at - det * yl * yl, F(0))) + b * yl) * ra - F(0.01)
            rows = lo <= hi + F(0.01)
            for q in range(2):
                m |= np.where(rows & (xr >= X + F(8 * q)) & (xl <= X + F(8 * q + 7)), 1 << (2 * r + q), 0).astype(
                    np.uint32)
    return np.where(o >= F(1) / F(255), np.where(general, 255, m), 0)


def reached(mx, my, a, b, c, o):
    """The blocks with a pixel of alpha >= 1/255, from the per-pixel evaluation in float32 (with
    its products rounded one by one: a fused product rounds less)."""
    y, x = np.meshgrid(np.arange(16, dtype=F), np.arange(16, dtype=F), indexing="ij")
    dx, dy = mx[:, None, None] - x, my[:, None, None] - y
    e = lambda v: v[:, None, None]  # noqa: E731
    with np.errstate(all="ignore"):
        power = F(-0.5) * (e(a) * dx * dx + e(c) * dy * dy) - e(b) * dx * dy
        ok = (power <= 0) & (np.minimum(F(0.99), e(o) * np.exp(power)) >= F(1) / F(255))
    q = ok.reshape(-1, 4, 4, 2, 8).any(axis=(2, 4))
    return sum(q[:, r, k].astype(np.uint32) << (2 * r + k) for r in range(4) for k in range(2))


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
def test_block_mask_covers_every_reached_pixel(aspect):
    rec = conics(60000, aspect, int(aspect * 10))
    m, r = block_mask(*rec), reached(*rec)
    assert not np.any(r & ~m), int(np.count_nonzero(r & ~m))
    if aspect < 60:  # beyond, the degenerate conics keep every block
        extra = sum(int(np.count_nonzero((m & ~r) >> k & 1)) for k in range(8))
        total = sum(int(np.count_nonzero(r >> k & 1)) for k in range(8))
        assert extra <= 0.15 * total, (extra, total)


def test_block_mask_degenerate_conics():
    one = lambda v: np.full(6, v, F)  # noqa: E731
    a = np.array([1, -1, 0, np.nan, np.inf, 1], F)
    m = block_mask(one(8), one(8), a, np.array([1, 0, 0, 0, 0, 2], F), one(1), one(0.5))
    assert np.all(m == 255)
    assert np.all(block_mask(one(8), one(8), one(1), one(0), one(1), one(0.003)) == 0)  # below 1/255
    # the source states the constants replayed here
    src = open(os.path.join(CSRC, "fgs_common.cuh")).read()
    body = src[src.index("uint32_t block_mask("):]
    for k in ("1.02f * (2.f * __logf(255.f * o)) + 0.1f", "det >= 2.5e-4f * ac", "+ 0.01f;", "lo <= hi + 0.01f"):
        assert k in body, k


def _level(v, m, o):
    """sum9_level: m of the values a lane holds go on, the others to the lane `o` away."""
    lanes = np.arange(32)
    hi = (lanes & o) != 0
    out = []
    for i in range(m):
        up = v[i + m] if i + m < len(v) else np.zeros(32, F)
        out.append(np.where(hi, up, v[i]) + np.where(hi, v[i], up)[lanes ^ o])
    return out


def _sum9(v):
    for m, o in ((5, 16), (3, 8), (2, 4), (1, 2)):
        v = _level(v, m, o)
    return v[0] + v[0][np.arange(32) ^ 1]


def test_add_step_sums_has_the_bits_of_warp_transpose_sum9():
    rng = np.random.default_rng(5)
    g = rng.standard_normal((4, 9, 32)).astype(F)    # four steps' sums of every lane
    lanes = np.arange(32)
    step, r, x = lanes >> 3, lanes & 3, lanes & 4
    # the staged sums: a[step][half][place][i] holds sum 4 half + i of lane place ^ (4 half)
    a = np.stack([np.stack([g[s, 4 * h:4 * h + 4, lanes ^ (4 * h)] for h in (0, 1)]) for s in range(4)])
    at = lambda k: a[step, x >> 2, (r + 4 * k) ^ x]  # noqa: E731
    v = [at(k) + at(k + 4) for k in range(4)]
    v = (v[0] + v[2]) + (v[1] + v[3])
    hi2, hi1 = (r & 2) != 0, (r & 1) != 0
    s = [np.where(hi2, v[:, 2 + i], v[:, i]) + np.where(hi2, v[:, i], v[:, 2 + i])[lanes ^ 2] for i in (0, 1)]
    tot = np.where(hi1, s[1], s[0]) + np.where(hi1, s[0], s[1])[lanes ^ 1]
    b = lambda k: g[step, 8, (lanes & 7) + 8 * k]  # noqa: E731
    z = (b(0) + b(2)) + (b(1) + b(3))
    for o in (4, 2, 1):
        z = z + z[lanes ^ o]
    src = open(os.path.join(CSRC, "fgs_common.cuh")).read()
    table = int(re.search(r"int sum9_component\(unsigned lane\).*?\(0x([0-9a-f]+)ull", src, re.S).group(1), 16)
    place = {(table >> (4 * i)) & 15: 2 * i for i in range(16)}
    for k in range(4):
        want = _sum9(list(g[k]))
        for q in range(8):
            assert tot[8 * k + q] == want[place[q]], (k, q)
        assert z[8 * k] == want[place[8]], k
        assert np.allclose(want[[place[q] for q in range(9)]], g[k].sum(1, dtype=np.float64), rtol=1e-5, atol=1e-5)
