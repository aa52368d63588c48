"""Replays on both sides of the count that parts warps from threads: exactly as
many rays with a tied nearest hit (every primitive is there several times, and
every ray hits one), in leaves of more primitives than a warp has lanes among
them.  The hits equal the single pass in the reference's own order, bit for
bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import surface_b200 as sb  # noqa: E402
from surface_b200 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu

EDGE = {"tri": 1 << 16, "sph": 1 << 16, "tet": 1 << 13}


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a)).cuda()


def _accel(kind, copies):
    """The accel and the points of its primitives to aim at."""
    keep = None if copies == 2 else 40
    if kind == "tri":
        v, f = S.displaced_octasphere(4, seed=8)
        f = f[:keep]
        acc = sb.TriangleAccel()
        acc.Build32(sb.Mesh(_dev(v), _dev(np.tile(f, (copies, 1)).astype(np.int32))))
        return acc, v[f.astype(np.int64)].mean(1)
    if kind == "tet":
        v, f, _ = S.tet_grid(6, seed=8)
        f = f[:keep]
        acc = sb.TetraAccel()
        acc.Build32(sb.Tetrahedron(_dev(v), _dev(np.tile(f, (copies, 1)).astype(np.int32))))
        return acc, v[f.astype(np.int64)].mean(1)
    p, r = S.particles(2000, seed=8, median_radius=0.03)
    p, r = p[:keep], r[:keep]
    acc = sb.ParticleAccel()
    acc.Build32(sb.Particles(_dev(np.tile(p, (copies, 1))), _dev(np.tile(r, copies))))
    return acc, p


@pytest.mark.parametrize("kind", ["tri", "sph", "tet"])
@pytest.mark.parametrize("copies", [2, 50])
@pytest.mark.parametrize("extra", [-1, 0, 1])
def test_replay_on_both_sides_of_the_count(kind, copies, extra):
    acc, aim = _accel(kind, copies)
    n = EDGE[kind] + extra
    rng = np.random.default_rng(n)
    to = aim[rng.integers(0, aim.shape[0], 2 * n)] + 1e-3 * rng.normal(size=(2 * n, 3))
    o = to + 3.0 * S._normalize(rng.normal(size=(2 * n, 3)))
    rays = S.make_rays(o, to - o)
    rt = _dev(rays.view(np.float32).reshape(-1, 8))
    want = acc.Traverse(rt, single_pass=True)
    hit = (want[:, 3].view(torch.int32) != -1).nonzero()[:, 0]
    assert hit.numel() >= n
    rt, want = rt[hit[:n]].contiguous(), want[hit[:n]].contiguous()
    got = acc.Traverse(rt)
    acc.ctx.use_torch_stream()
    acc.ctx.synchronize()
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
