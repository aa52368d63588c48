"""Trees with more branches than wide nodes (one per six primitives above
1.57 million): built, they are walked by their two-child nodes, loaded from a
file, which makes a wide node for every branch, by the wide ones.  Same hits as
the walk in the reference's order, and the two-child walk takes no longer over
the built tree than over the loaded one (the boxes of both are in order, so
neither needs the reference's comparisons)."""
import ctypes as C
import os
import tempfile

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import surface_b200 as sb  # noqa: E402
from surface_b200 import _lib  # noqa: E402
from surface_b200 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu


def _centres():
    """65,536 groups of 26 points of a 1024^3 grid: 18 at a Morton code whose
    low 14 bits are 0 and one at each of its bits 6 to 13, so that a group is a
    chain of branches down to the deepest level."""
    low = np.concatenate([np.zeros(18, np.uint32), np.uint32(1) << np.arange(6, 14, dtype=np.uint32)])
    code = ((np.arange(65536, dtype=np.uint32) << 14)[:, None] | low[None]).reshape(-1)
    xyz = np.zeros((code.size, 3), np.uint32)
    for b in range(10):
        for k in range(3):
            xyz[:, k] |= ((code >> np.uint32(3 * b + 2 - k)) & 1) << np.uint32(b)
    return ((xyz + 0.5) / 1024.0).astype(np.float32)


def _accel(kind):
    c = _centres()
    size = (2e-4 * (1.0 + 0.01 * (np.arange(c.shape[0]) % 26))).astype(np.float32)
    if kind == "sph":
        data = sb.Particles(torch.as_tensor(c).cuda(), torch.as_tensor(size).cuda())
        acc, make = sb.ParticleAccel(), sb.ParticleAccel
    else:
        corner = np.array([[1, 0, -0.5], [-0.5, 0.8, -0.5], [-0.5, -0.8, 1]], np.float32)
        v = (c[:, None] + size[:, None, None] * corner).reshape(-1, 3)
        f = np.arange(v.shape[0], dtype=np.int32).reshape(-1, 3)
        data = sb.Mesh(torch.as_tensor(v).cuda(), torch.as_tensor(f).cuda())
        acc, make = sb.TriangleAccel(), sb.TriangleAccel
    acc.Build32(data)
    n, nb = c.shape[0], acc.info().num_branches
    assert (n - 1) // 6 > 1 << 18 and nb > (n - 1) // 6
    with tempfile.TemporaryDirectory() as td:
        path = os.path.join(td, "a.bin")
        acc.Dump(path)
        loaded = make()
        loaded.Load(path, data)
    return acc, loaded, c


def _rays(c, n, seed):
    rng = np.random.default_rng(seed)
    o = 0.5 + 2.0 * S._normalize(rng.normal(size=(n, 3)))
    to = c[rng.integers(0, c.shape[0], n)] + rng.normal(size=(n, 3)) * 1e-4
    return torch.as_tensor(S.make_rays(o, to - o).view(np.float32).reshape(-1, 8)).cuda()


def _launches(acc):
    return acc.L.srt_ctx_launch_count(acc.ctx.h)


@pytest.mark.parametrize("kind", ["tri", "sph"])
def test_more_branches_than_wide_nodes(kind):
    acc, loaded, c = _accel(kind)
    r = _rays(c, 5000, 1)
    want = acc.Traverse(r, single_pass=True)
    assert (want[:, 3].view(torch.int32) != -1).float().mean() > 0.3
    for a, kernels in ((acc, 3), (loaded, 2)):  # both first passes, or the wide one; the replay
        before = _launches(a)
        got = a.Traverse(r)
        assert _launches(a) - before == kernels
        fixed = torch.full_like(want, float("nan"))
        assert a.L.srt_trace_closest_noalloc(a.h, C.c_void_p(r.data_ptr()), r.shape[0],
                                             C.c_void_p(fixed.data_ptr())) == _lib.SRT_OK
        torch.cuda.synchronize()
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))
        assert torch.equal(fixed.view(torch.int32), want.view(torch.int32))
    # the two-child walk over either
    r = _rays(c, 1 << 20, 2)
    us = {}
    for name, a in (("built", acc), ("loaded", loaded)) * 4:
        e0, e1 = torch.cuda.Event(True), torch.cuda.Event(True)
        e0.record()
        a.Traverse(r, grid_launch=True)
        e1.record()
        torch.cuda.synchronize()
        us.setdefault(name, []).append(e0.elapsed_time(e1) * 1e3)
    print({k: [round(x) for x in v] for k, v in us.items()})
    assert min(us["built"][1:]) < 1.08 * min(us["loaded"][1:]), us
