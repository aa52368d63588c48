"""Both sides of every line of the rule that picks the wide or the two-child
walk: the hits of the single pass, from srt_trace_closest and, up to its limit
of 262,144 rays, srt_trace_closest_noalloc."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import surface_b200 as sb  # noqa: E402
from surface_b200 import _lib  # noqa: E402
from surface_b200 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["tri", "sph"])
@pytest.mark.parametrize("prims", [(1 << 13) - 1, 1 << 13, (1 << 15) - 1, 1 << 15])
def test_rule_edges(kind, prims):
    if kind == "tri":
        v, f = S.octasphere_for_count(prims, 5)
        acc, c = sb.TriangleAccel(), 0.0
        acc.Build32(sb.Mesh(torch.as_tensor(v).cuda(), torch.as_tensor(f.astype(np.int32)).cuda()))
    else:
        p, r = S.particles(prims, seed=5, median_radius=0.3 / prims ** (1 / 3))
        acc, c = sb.ParticleAccel(), 0.5
        acc.Build32(sb.Particles(torch.as_tensor(p).cuda(), torch.as_tensor(r).cuda()))
    most = 1 << 19
    rng = np.random.default_rng(prims)
    o = c + 2.5 * S._normalize(rng.normal(size=(most, 3)))
    rays = S.make_rays(o, c + 0.5 * rng.uniform(-1, 1, size=(most, 3)) - o)
    rays = torch.as_tensor(rays.view(np.float32).reshape(-1, 8)).cuda()
    want = acc.Traverse(rays, single_pass=True)
    assert (want[:, 3].view(torch.int32) != -1).float().mean() > 0.2
    for edge in (1 << 18, 3 << 17, 1 << 19):
        for n in (edge - 1, edge):
            got = [acc.Traverse(rays[:n].contiguous())]
            if n <= 262144:
                got.append(torch.full((n, 4), float("nan"), device="cuda"))
                _lib.check(acc.L.srt_trace_closest_noalloc(
                    acc.h, C.c_void_p(rays.data_ptr()), n, C.c_void_p(got[1].data_ptr())))
            acc.ctx.synchronize()
            for h in got:
                assert torch.equal(h.view(torch.int32), want[:n].view(torch.int32)), n
