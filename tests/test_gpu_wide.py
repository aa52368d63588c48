"""The four-lanes-per-ray walk over the wide nodes against the two-child walk
(grid_launch=True runs it): identical hits, bit for bit, at leaf and tile
edges, on rays whose slab products are NaN, on boxes that are not ordered and
on both sides of the size rule."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import surface_b200 as sb  # noqa: E402
from surface_b200 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a)).cuda()


def _rays(kind, n, seed):
    rng = np.random.default_rng(seed)
    c = np.zeros(3) if kind == "tri" else np.full(3, 0.5)
    o = c + rng.normal(size=(n, 3)) * 1.5
    d = c + 0.6 * rng.normal(size=(n, 3)) - o
    k = rng.integers(0, 8, size=n)
    d[k == 0, 0] = 0.0  # zero components: infinite reciprocals
    d[k == 1, 1:] = 0.0
    o[k == 1] = np.round(o[k == 1] * 4) / 4  # on box planes of grid-like scenes
    d[k == 2, 2] = -0.0
    r = S.make_rays(o, d)
    if n > 64:
        r["dir"][5] = np.nan
        r["org"][6, 1] = np.inf
        r["dir"][7] = 0.0
    return r


def _accel(kind, n, seed, special=None):
    if kind == "tri":
        v, f = S.octasphere_for_count(n, seed)
        if special == "flat":
            v = v.copy()
            v[:, 2] = 0.25
        if special == "same":
            f = np.tile(f[:1], (n, 1))
        if special == "nan":
            v = v.copy()
            v[f[0, 0]] = np.nan
        acc = sb.TriangleAccel()
        acc.Build32(sb.Mesh(_dev(v), _dev(f.astype(np.int32))))
        return acc
    p, r = S.particles(n, seed=seed, median_radius=0.3 / n ** (1 / 3))
    if special == "same":
        p[:] = p[:1]
    if special == "nan":
        p[0] = np.nan
    acc = sb.ParticleAccel()
    acc.Build32(sb.Particles(_dev(p), _dev(r)))
    return acc


def _same(acc, rays, **kw):
    r = _dev(rays.view(np.float32).reshape(-1, 8))
    a = acc.Traverse(r, want_normal=True, **kw)
    b = acc.Traverse(r, want_normal=True, grid_launch=True, **kw)
    acc.ctx.use_torch_stream()
    acc.ctx.synchronize()
    for x, y in ((a.hits, b.hits), (a.normal, b.normal)):
        assert torch.equal(x.view(torch.int32), y.view(torch.int32))
    return a.hits


@pytest.mark.parametrize("kind", ["tri", "sph"])
@pytest.mark.parametrize("n", [2, 17, 18, 19, 35, 1024, 4097, 40000])
def test_wide_matches_two_child_walk(kind, n):
    acc = _accel(kind, n, seed=n)
    hit = 0
    for m in (1, 31, 33, 5000):
        h = _same(acc, _rays(kind, m, seed=m + n))
        hit += int((h[:, 3].view(torch.int32) != -1).sum())
    assert hit > 0


@pytest.mark.parametrize("kind", ["tri", "sph"])
@pytest.mark.parametrize("special", ["flat", "same", "nan"])
def test_wide_special_trees(kind, special):
    if kind == "sph" and special == "flat":
        special = "same"
    _same(_accel(kind, 3000, 3, special), _rays(kind, 4000, 9))


@pytest.mark.parametrize("kind", ["tri", "sph"])
def test_wide_secondary_and_sorted(kind):
    acc = _accel(kind, 20000, 4)
    rays = _rays(kind, 20000, 5)
    h = _same(acc, rays)
    r = _dev(rays.view(np.float32).reshape(-1, 8))
    res = acc.Traverse(r, want_normal=True)
    more, nrm = sb.spawn_secondary(r, res.hits, res.normal, 3)
    sec = more.cpu().numpy().view(S.RAY_DTYPE).reshape(-1)
    _same(acc, sec, prev_normals=nrm)
    s = acc.Traverse(r, sort_rays=True)
    assert torch.equal(s.view(torch.int32), h.view(torch.int32))


@pytest.mark.parametrize("n", [(1 << 15) - 1, 1 << 15])
def test_wide_rule_edges(n):
    acc = _accel("tri", n, 6)
    for m in ((1 << 19) - 1, 1 << 19):
        _same(acc, _rays("tri", m, 7))
