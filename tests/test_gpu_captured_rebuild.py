"""Traces in a CUDA graph stay valid while the accel is rebuilt in place to
other counts that fit its buffers, on the device arrays that it had: a replay
finds the hits of the tree that is there then."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import surface_b200 as sb  # noqa: E402
from surface_b200 import _lib  # noqa: E402
from surface_b200 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu


def _data(kind, n):
    if kind == "tri":
        v, f = S.octasphere_for_count(n, n)
        return sb.Mesh(torch.as_tensor(v).cuda(), torch.as_tensor(f.astype(np.int32)).cuda())
    p, r = S.particles(n, seed=n, median_radius=0.3 / n ** (1 / 3))
    return sb.Particles(torch.as_tensor(p).cuda(), torch.as_tensor(r).cuda())


@pytest.mark.parametrize("kind", ["tri", "sph"])
@pytest.mark.parametrize("counts", [(40_000, 9_000, 25_001, 17, 40_000),
                                    (400_000, 30_000, 300_000, 400_000)])
def test_replays_after_rebuilds(kind, counts):
    acc = sb.TriangleAccel() if kind == "tri" else sb.ParticleAccel()
    c = 0.0 if kind == "tri" else 0.5
    rng = np.random.default_rng(3)
    o = c + 2.5 * S._normalize(rng.normal(size=(20_000, 3)))
    rays = S.make_rays(o, c + 0.5 * rng.uniform(-1, 1, size=o.shape) - o)
    rays = torch.as_tensor(rays.view(np.float32).reshape(-1, 8)).cuda()
    acc.Build32(_data(kind, counts[0]))
    acc.Traverse(rays)
    # captured with the second count, whose buffers are the first's
    acc.Build32(_data(kind, counts[1]))
    hits = [torch.empty((rays.shape[0], 4), device="cuda") for _ in range(2)]
    acc.Traverse(rays, hits=hits[0])
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        acc.Traverse(rays, hits=hits[0])
        acc.ctx.use_torch_stream()
        _lib.check(acc.L.srt_trace_closest_noalloc(acc.h, C.c_void_p(rays.data_ptr()),
                                                   rays.shape[0],
                                                   C.c_void_p(hits[1].data_ptr())))
    for n in counts[1:] + counts[:1]:
        acc.Build32(_data(kind, n))
        want = acc.Traverse(rays, single_pass=True)
        for h in hits:
            h.fill_(float("nan"))
        g.replay()
        torch.cuda.synchronize()
        assert (want[:, 3].view(torch.int32) != -1).float().mean() > 0.2
        for h in hits:
            assert torch.equal(h.view(torch.int32), want.view(torch.int32)), n
