"""The work counters of a trace count the same whatever walk the default
takes: the nodes of the two-child walk (triangles, spheres) and, for
tetrahedra in the reference's order, the nodes that walk pops."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import surface_b200 as sb  # noqa: E402
from surface_b200 import _lib  # noqa: E402
from surface_b200 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a)).cuda()


def traced(acc, rays, flags=0, max_iter=0):
    """(hits, counters, status) of one call with counters."""
    r = _dev(rays.view(np.float32).reshape(-1, 8))
    hits = torch.empty((r.shape[0], 4), device="cuda")
    stats = torch.zeros(4, dtype=torch.int64, device="cuda")
    o = _lib.TraceOpts()
    o.stats, o.flags, o.max_iter = stats.data_ptr(), flags, max_iter
    acc.ctx.use_torch_stream()
    _lib.check(acc.L.srt_trace_closest(acc.h, r.data_ptr(), r.shape[0], hits.data_ptr(),
                                       C.byref(o)))
    status = acc.L.srt_ctx_synchronize(acc.ctx.h)
    return hits, stats.tolist(), status


@pytest.mark.parametrize("kind", ["tri", "sph"])
@pytest.mark.parametrize("nrays", [33, 100_000, (1 << 19) - 1, 1 << 19])
def test_counters_do_not_depend_on_the_walk(kind, nrays):
    rng = np.random.default_rng(nrays)
    if kind == "tri":
        v, f = S.displaced_octasphere(6, seed=2)
        acc, c = sb.TriangleAccel(), np.zeros(3)
        acc.Build32(sb.Mesh(_dev(v), _dev(f.astype(np.int32))))
    else:
        p, r = S.particles(20000, seed=2, median_radius=0.01)
        acc, c = sb.ParticleAccel(), np.full(3, 0.5)
        acc.Build32(sb.Particles(_dev(p), _dev(r)))
    o = c + 2.5 * S._normalize(rng.normal(size=(nrays, 3)))
    rays = S.make_rays(o, c + 0.5 * rng.uniform(-1, 1, size=(nrays, 3)) - o)
    h, got, s = traced(acc, rays)
    w, want, t = traced(acc, rays, flags=_lib.SRT_TRACE_GRID)
    assert s == t == _lib.SRT_OK
    assert got == want and got[0] > nrays
    assert torch.equal(h.view(torch.int32), w.view(torch.int32))
    # and the call without counters, by whichever walk, finds the same hits
    plain = acc.Traverse(_dev(rays.view(np.float32).reshape(-1, 8)))
    assert torch.equal(plain.view(torch.int32), h.view(torch.int32))


def test_tetrahedra_count_the_nodes_popped():
    v, f, _ = S.tet_grid(1, seed=2)  # five tetrahedra: a root and two leaves, or one more branch
    acc = sb.TetraAccel()
    acc.Build32(sb.Tetrahedron(_dev(np.concatenate([v, v + 5])),
                               _dev(np.concatenate([f, f + v.shape[0]]).astype(np.int32))))
    nodes = acc.info().num_branches
    n = 500
    rng = np.random.default_rng(1)
    away = S.make_rays(np.full((n, 3), -3.0) - rng.uniform(0, 1, size=(n, 3)),
                       np.full((n, 3), -1.0))
    _, st, _ = traced(acc, away, flags=_lib.SRT_TRACE_SINGLE_PASS)
    assert st[:3] == [n, 0, 0]  # each pops the root alone
    o = np.tile(np.array([[0.5, 0.5, -2.0]]), (n, 1)) + rng.uniform(-0.2, 0.2, size=(n, 3))
    through = S.make_rays(o, np.tile(np.array([[0.01, 0.02, 1.0]]), (n, 1)))
    h, st, _ = traced(acc, through, flags=_lib.SRT_TRACE_SINGLE_PASS)
    assert (h[:, 3].view(torch.int32) != -1).all()
    # the root and both children of every branch entered
    assert (st[0] - n) % 2 == 0 and 2 * n <= st[0] - n <= 2 * n * nodes
    assert st[0] >= n + st[1]
