"""A batch of the smallest and oddest scenes: leaf-size edges, duplicated
faces (deep trees), each against its own single build."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import surface_b200 as sb  # noqa: E402
from surface_b200 import scenes as S  # noqa: E402
from surface_b200.batch import TriangleBatch  # noqa: E402

pytestmark = pytest.mark.gpu


def test_small_scenes_match_single_builds():
    meshes = [S.octasphere_for_count(n, seed=n) for n in (2, 3, 17, 18, 19, 35, 300, 2049)]
    v, f = S.octasphere_for_count(64, seed=1)
    meshes.append((v, np.tile(f[:2], (350, 1))))
    v, f = S.octasphere_for_count(900, seed=2)
    meshes.append((v * np.float32(2.0) ** -np.arange(v.shape[0], dtype=np.float32)[:, None] ** 0.5,
                   f))
    verts, faces, rays, fo, ro, base = [], [], [], [0], [0], 0
    for k, (v, f) in enumerate(meshes):
        verts.append(v.astype(np.float32))
        faces.append(f.astype(np.int32) + base)
        base += v.shape[0]
        rays.append(S.pinhole_rays(20 + 3 * k, 17, (0.1, 0.2, 3.0), (0, 0, 0)))
        fo.append(fo[-1] + f.shape[0])
        ro.append(ro[-1] + rays[-1].size)
    v = torch.as_tensor(np.concatenate(verts)).cuda()
    f = torch.as_tensor(np.concatenate(faces)).cuda()
    r = torch.as_tensor(np.concatenate(rays).view(np.float32).reshape(-1, 8)).cuda()
    b = TriangleBatch()
    b.set_tuning()
    got = b.build_trace(v, f, fo, r, ro)
    torch.cuda.synchronize()
    for s in range(len(meshes)):
        acc = sb.TriangleAccel()
        acc.Build32(sb.Mesh(v, f[fo[s]:fo[s + 1]].contiguous()))
        want = acc.Traverse(r[ro[s]:ro[s + 1]].contiguous())
        assert torch.equal(got[ro[s]:ro[s + 1]].view(torch.int32), want.view(torch.int32)), s
