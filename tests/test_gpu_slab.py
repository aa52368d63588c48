"""The packed slab test and the sphere prefilter of the two-child walk against
the single pass, which keeps the reference's comparisons: identical hits for
rays with zero, negative-zero and infinite components and for trees whose
boxes are flat or coincide (or, for spheres, hold NaN), singly and in a
batch.  (With a NaN corner in a triangle the two passes and the single pass
need not agree: which boxes hide a hit depends on the order they are entered.)"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import surface_b200 as sb  # noqa: E402
from surface_b200 import scenes as S  # noqa: E402
from surface_b200.batch import TriangleBatch  # noqa: E402

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a)).cuda()


def _rays(c, n, seed):
    rng = np.random.default_rng(seed)
    o = c + rng.normal(size=(n, 3)) * 1.5
    d = c + 0.5 * rng.normal(size=(n, 3)) - o
    k = rng.integers(0, 8, size=n)
    d[k == 0, 0] = 0.0
    d[k == 1, 1:] = 0.0
    o[k == 1] = np.round(o[k == 1] * 4) / 4
    d[k == 2, 2] = -0.0
    d[k == 3] *= 1e-3
    return S.make_rays(o, d)


def _mesh(special):
    v, f = S.displaced_octasphere(4, seed=5)
    v = v.copy()
    if special == "flat":
        v[:, 1] = 0.25
    if special == "same":
        f = np.tile(f[:3], (700, 1))
    return v, f


@pytest.mark.parametrize("kind,special", [("tri", "plain"), ("tri", "flat"), ("tri", "same"),
                                          ("sph", "plain"), ("sph", "flat"), ("sph", "same"),
                                          ("sph", "nan")])
def test_two_child_walk_matches_single_pass(kind, special):
    if kind == "tri":
        v, f = _mesh(special)
        acc = sb.TriangleAccel()
        acc.Build32(sb.Mesh(_dev(v), _dev(f.astype(np.int32))))
        c = np.zeros(3)
    else:
        p, r = S.particles(3000, seed=5, median_radius=0.02)
        if special == "flat":
            p[:, 1] = 0.25
        if special == "same":
            p[:] = p[:1]
            r[:1500] = 0.0
        if special == "nan":
            p[11] = np.nan
        acc = sb.ParticleAccel()
        acc.Build32(sb.Particles(_dev(p), _dev(r)))
        c = np.full(3, 0.5)
    rt = _dev(_rays(c, 6000, 3).view(np.float32).reshape(-1, 8))
    a = acc.Traverse(rt, grid_launch=True)
    b = acc.Traverse(rt, single_pass=True)
    acc.ctx.use_torch_stream()
    acc.ctx.synchronize()
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))


def test_batch_matches_single_pass():
    verts, faces, rays, fo, ro, want = [], [], [], [0], [0], []
    for k, special in enumerate(("plain", "flat", "same")):
        v, f = _mesh(special)
        r = _rays(np.zeros(3), 500 + k, k).view(np.float32).reshape(-1, 8)
        acc = sb.TriangleAccel()
        acc.Build32(sb.Mesh(_dev(v), _dev(f.astype(np.int32))))
        want.append(acc.Traverse(_dev(r), single_pass=True))
        faces.append(f.astype(np.int32) + sum(x.shape[0] for x in verts))
        verts.append(v)
        rays.append(r)
        fo.append(fo[-1] + f.shape[0])
        ro.append(ro[-1] + r.shape[0])
    b = TriangleBatch()
    b.set_tuning()
    got = b.build_trace(_dev(np.concatenate(verts)), _dev(np.concatenate(faces)), fo,
                        _dev(np.concatenate(rays)), ro)
    torch.cuda.synchronize()
    assert torch.equal(got.view(torch.int32), torch.cat(want).view(torch.int32))
