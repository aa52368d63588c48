"""Axis-parallel rays, whose zero components make infinite reciprocals: the
four-lane walk, the two-child walk, the batch and the single pass in the
reference's own order agree bit for bit, for origins between the box planes
(where the packed slab test holds) and on them (where products are NaN), for
+0 and -0, denormal and infinite components."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import surface_b200 as sb  # noqa: E402
from surface_b200 import scenes as S  # noqa: E402
from surface_b200.batch import TriangleBatch  # noqa: E402

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a)).cuda()


def _rays(points, lo, hi, n, seed):
    """Rays along the axes and in the coordinate planes; half of the origins
    have a coordinate of a primitive's corner."""
    rng = np.random.default_rng(seed)
    o = rng.uniform(lo, hi, size=(n, 3)).astype(np.float32)
    at = points[rng.integers(0, points.shape[0], n)]
    on = rng.uniform(size=(n, 3)) < 0.5
    o = np.where(on, at, o).astype(np.float32)
    a = rng.integers(0, 3, n)
    k = np.arange(n)
    d = np.zeros((n, 3), np.float32)
    flat = rng.uniform(size=n) < 0.3  # in a plane: one zero component
    d[flat] = rng.normal(size=(int(flat.sum()), 3))
    d[k, (a + 1) % 3] = 0.0
    side = np.where(rng.uniform(size=n) < 0.5, -1.0, 1.0)
    d[k, a] = side
    o[k, a] -= np.float32(2.0 * (hi - lo)) * side.astype(np.float32)
    zero = rng.choice(5, n, p=[0.6, 0.2, 0.1, 0.05, 0.05])
    b = (a + 1) % 3
    d[k[zero == 1], b[zero == 1]] = -0.0
    d[k[zero == 2], b[zero == 2]] = np.float32(1e-42)
    d[k[zero == 3], b[zero == 3]] = np.float32(-1e-42)
    d[k[zero == 4], a[zero == 4]] *= np.float32(np.inf)
    return S.make_rays(o, d).view(np.float32).reshape(-1, 8)


def _tri(grid):
    if grid:  # corners on a coarse lattice: many box planes at the same places
        v, f, _ = S.tet_grid(8, seed=3, jitter=0.0)
        f = np.concatenate([f[:, :3], f[:, 1:]])
        return v, f.astype(np.int32), 0.0, 1.0
    v, f = S.displaced_octasphere(6, seed=3)
    return v, f.astype(np.int32), -1.2, 1.2


@pytest.mark.parametrize("kind", ["tri", "grid", "sph"])
@pytest.mark.parametrize("n", [3000, (1 << 19) + 77])
def test_axis_parallel_rays(kind, n):
    if kind == "sph":
        p, r = S.particles(30000, seed=3, median_radius=8e-3)
        pts, lo, hi = np.concatenate([p, p + r[:, None], p - r[:, None]]), 0.0, 1.0
        acc = sb.ParticleAccel()
        acc.Build32(sb.Particles(_dev(p), _dev(r)))
    else:
        v, f, lo, hi = _tri(kind == "grid")
        pts = v
        acc = sb.TriangleAccel()
        acc.Build32(sb.Mesh(_dev(v), _dev(f)))
    rays = _dev(_rays(pts, lo, hi, n, seed=n))
    want = acc.Traverse(rays, single_pass=True)
    assert (want[:, 3].view(torch.int32) != -1).float().mean() > 0.1
    for kw in (dict(), dict(grid_launch=True), dict(sort_rays=True)):
        got = acc.Traverse(rays, **kw)
        assert torch.equal(got.view(torch.int32), want.view(torch.int32)), kw
    if kind != "sph":
        b = TriangleBatch()
        b.set_tuning()
        got = b.build_trace(_dev(v), _dev(f), [0, f.shape[0]], rays, [0, n])
        torch.cuda.synchronize()
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))
