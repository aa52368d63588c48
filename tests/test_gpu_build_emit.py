"""The wide nodes are emitted with the two-child nodes of a build and made in a
kernel of their own for a loaded tree: the build launches no kernel for them,
and both accels find the same hits by their wide nodes, for trees of one branch
up, with coinciding primitives and with NaN (whose boxes are out of order)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import surface_b200 as sb  # noqa: E402
from surface_b200 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu

KERNELS = 10  # box, codes, three sort passes, Karras, levels, cache, refit, emission


def _data(kind, n, special):
    if kind == "tri":
        v, f = S.octasphere_for_count(n, n)
        v = v.copy()
        if special == "same":
            f = np.tile(f[:1], (n, 1))
        if special == "nan":
            v[f[0, 0]] = np.nan
        return sb.Mesh(torch.as_tensor(v).cuda(), torch.as_tensor(f.astype(np.int32)).cuda())
    p, r = S.particles(n, seed=n, median_radius=0.3 / n ** (1 / 3))
    if special == "same":
        p[:] = p[:1]
    if special == "nan":
        p[0] = np.nan
    return sb.Particles(torch.as_tensor(p).cuda(), torch.as_tensor(r).cuda())


@pytest.mark.parametrize("kind", ["tri", "sph"])
@pytest.mark.parametrize("special", [None, "same", "nan"])
@pytest.mark.parametrize("n", [2, 18, 35, 300, 5000, 70001])
def test_built_and_loaded(kind, special, n, tmp_path):
    make = sb.TriangleAccel if kind == "tri" else sb.ParticleAccel
    c = 0.0 if kind == "tri" else 0.5
    data = _data(kind, n, special)
    acc = make()
    before = acc.L.srt_ctx_launch_count(acc.ctx.h)
    acc.Build32(data)
    assert acc.L.srt_ctx_launch_count(acc.ctx.h) - before == KERNELS
    path = str(tmp_path / "a.bin")
    acc.Dump(path)
    loaded = make()
    loaded.Load(path, data)
    rng = np.random.default_rng(n)
    o = c + 2.5 * S._normalize(rng.normal(size=(6000, 3)))
    rays = S.make_rays(o, c + 0.5 * rng.uniform(-1, 1, size=o.shape) - o)
    r = torch.as_tensor(rays.view(np.float32).reshape(-1, 8)).cuda()
    a, b = acc.Traverse(r), loaded.Traverse(r)
    w = acc.Traverse(r, grid_launch=True)
    torch.cuda.synchronize()
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    assert torch.equal(a.view(torch.int32), w.view(torch.int32))
