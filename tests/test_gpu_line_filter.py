"""The line walk against the oracle's, bit for bit, where its line filter and
its slab test could differ from the plain test: uniform, tapered and thick
lines, lines far longer than the rest, tiny and huge units, geometry far from
the origin, boxes that are not ordered, leaves of more than 32 lines, caps on
and off, directions of any length and rays whose slab products are NaN."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle as O  # noqa: E402
from surface_b200 import scenes as S  # noqa: E402
from surface_b200.lines import LineAccel, LineBuildOptions, Lines  # noqa: E402

from conftest import bits  # noqa: E402

pytestmark = pytest.mark.gpu


def _rays(pos, n, seed):
    rng = np.random.default_rng(seed)
    lo, hi = pos.min(0).astype(np.float64), pos.max(0).astype(np.float64)
    c, e = (lo + hi) / 2, (hi - lo).max() + 1e-30
    o = c + e * rng.normal(size=(n, 3))
    d = c + 0.3 * e * rng.normal(size=(n, 3)) - o
    k = rng.integers(0, 10, size=n)
    on = pos[rng.integers(0, len(pos), n)].astype(np.float64)
    o[k == 1, 1:] = on[k == 1, 1:]  # along an axis through a vertex
    o[k == 2] = on[k == 2]          # from a vertex
    d[k >= 3] = on[k >= 3] - o[k >= 3]  # at a vertex
    d[k == 0, 0] = 0.0
    d[k == 1, 1:] = 0.0
    q = k >= 7  # directions of any length
    d[q] *= np.exp(rng.uniform(-5, 5, size=(n, 1)))[q]
    q = rng.random(n) < 0.5
    d[q] /= np.maximum(np.linalg.norm(d[q], axis=1, keepdims=True), 1e-30)
    r = S.make_rays(o, d)
    r["dir"][5] = np.nan
    r["org"][6, 1] = np.inf
    r["dir"][7] = 0.0
    r["dir"][8] = (3e25, 1e25, -2e25)
    r["dir"][9] = (1e-25, 0.0, -2e-25)
    r["dir"][10, 1] = -0.0
    return r


def _lines(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind == "uniform":
        return S.line_strands(n // 8, 8, seed=seed, radius=0.01, taper=False)
    pos = rng.uniform(-1, 1, size=(2 * n, 3))
    pos[1::2] = pos[::2] + rng.normal(size=(n, 3)) * 0.05
    rad = rng.uniform(0.0, 0.03, size=2 * n)
    if kind == "taper":  # radii that the boxes do not cover
        rad[::2] = 0.0
        rad[1::2] *= 8
    elif kind == "thin":
        pos[:16:2] *= 20.0
        rad[:] = 1e-4
    elif kind == "grid":  # on a lattice, many equal distances and box planes
        pos = np.round(pos * 4) / 4
        rad[:] = 0.125
    elif kind == "turned":  # boxes whose padding turns them around
        pos -= 100.0
        rad[:] = 0.0
        pos[1::2, 1:] = pos[::2, 1:]
    elif kind == "far":
        pos += 3000.0
    elif kind in ("tiny", "huge"):
        s = 1e-9 if kind == "tiny" else 1e9
        pos, rad = pos * s, rad * s
    seg = np.arange(2 * n, dtype=np.uint32).reshape(n, 2)
    return pos.astype(np.float32), seg, rad.astype(np.float32)


@pytest.mark.parametrize("kind", ["uniform", "random", "taper", "thin", "grid", "turned", "far",
                                  "tiny", "huge"])
@pytest.mark.parametrize("opts", [dict(cap=True), dict(cap=False), dict(max_depth=6),
                                  dict(min_leaf=1)])
def test_against_oracle(kind, opts):
    pos, seg, rad = _lines(kind, 4000, seed=3)
    rays = _rays(pos, 6000, seed=4)
    acc = LineAccel()
    acc.Build(Lines(pos, seg, rad),
              LineBuildOptions(minLeafPrimitives=opts.get("min_leaf", 4),
                               maxTreeDepth=opts.get("max_depth", 512),
                               cap=opts.get("cap", True)))
    want, wn = O.OracleLines(pos, seg, rad, 0.0, **opts).trace(rays)
    got, gn = acc.Traverse(rays, want_normal=True)
    assert np.array_equal(bits(got.view(np.float32).reshape(-1, 4)),
                          bits(want.view(np.float32).reshape(-1, 4)))
    assert np.array_equal(np.isnan(gn), np.isnan(wn))
    assert np.array_equal(bits(np.nan_to_num(gn)), bits(np.nan_to_num(wn)))
