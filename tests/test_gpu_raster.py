"""Rays in rows are walked in tiles of their rows: the same hit per ray as for
the same rays shuffled (which have no rows), for row lengths off the tile and
an unfinished last row, and for a batch whose scenes have rows of their own."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import surface_b200 as sb  # noqa: E402
from surface_b200 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a)).cuda()


def _accel(kind):
    if kind == "tri":
        v, f = S.displaced_octasphere(6, seed=2)
        acc = sb.TriangleAccel()
        acc.Build32(sb.Mesh(_dev(v), _dev(f.astype(np.int32))))
        return acc, (0, 0, 3), (0, 0, 0)
    if kind == "tet":
        v, f, _ = S.tet_grid(12, seed=2)
        acc = sb.TetraAccel()
        acc.Build32(sb.Tetrahedron(_dev(v), _dev(f.astype(np.int32))))
    elif kind == "sph":
        p, r = S.particles(40000, seed=2, median_radius=5e-3)
        acc = sb.ParticleAccel()
        acc.Build32(sb.Particles(_dev(p), _dev(r)))
    elif kind == "line":
        p, s, r = S.line_strands(300, 8, seed=2, radius=0.02)
        acc = sb.LineAccel()
        acc.Build(sb.Lines(_dev(p), _dev(s.astype(np.int32)), _dev(r)))
        return acc, (0, 0, 3.4), (0, 0, 0)
    else:
        v, ix = S.solid_grid(8, 11, seed=2)
        acc = sb.SolidAccel()
        acc.Build32(sb.Solid(8, _dev(v), _dev(ix.astype(np.int32))))
    return acc, (1.7, 1.3, 2.1), (0.5, 0.5, 0.5)


@pytest.mark.parametrize("kind", ["tri", "tet", "sph", "line", "solid"])
@pytest.mark.parametrize("w,h,extra", [(64, 4100, 0), (517, 509, 313), (1024, 1024, 0),
                                       (1087, 977, 1)])
def test_rows_and_shuffled_rays_agree(kind, w, h, extra):
    acc, eye, look = _accel(kind)
    rays = S.pinhole_rays(w, h + 1, eye, look)[:w * h + extra]
    r = _dev(rays.view(np.float32).reshape(-1, 8))
    p = torch.as_tensor(np.random.default_rng(w).permutation(r.shape[0])).cuda()
    a = acc.Traverse(r)
    b = acc.Traverse(r[p].contiguous())
    assert (a[:, 3].view(torch.int32) != -1).any()
    assert torch.equal(a[p].view(torch.int32), b.view(torch.int32))


def test_batch_rows():
    B = S.batched_scenes(nscenes=5, seed=3, lo=1e3, hi=2e4, sizes=(64, 96, 130, 257))
    args = (_dev(B["vertices"]), _dev(B["faces"].astype(np.int32)), B["face_offsets"])
    r = _dev(B["rays"].view(np.float32).reshape(-1, 8))
    ro = B["ray_offsets"].astype(np.int64)
    rng = np.random.default_rng(4)
    p = torch.as_tensor(np.concatenate([lo + rng.permutation(hi - lo)
                                        for lo, hi in zip(ro[:-1], ro[1:])])).cuda()
    from surface_b200.batch import TriangleBatch
    out = []
    for rays in (r, r[p].contiguous()):
        b = TriangleBatch()
        b.set_tuning()
        out.append(b.build_trace(*args, rays, ro))
    torch.cuda.synchronize()
    assert torch.equal(out[0][p].view(torch.int32), out[1].view(torch.int32))
