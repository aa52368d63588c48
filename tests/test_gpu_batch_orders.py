"""Unsorted rays of a batch: tiles in the scenes whose rays come in rows, array
order in the others -- the hits of each scene's own trace for batches of the
one, of the other and of both kinds, pinned and autotuned, through capture and
replay."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import surface_b200 as sb  # noqa: E402
from surface_b200 import scenes as S  # noqa: E402
from surface_b200.batch import TriangleBatch  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", ["all", "none", "every other", "one"])
@pytest.mark.parametrize("pinned", [True, False])
def test_scenes_with_and_without_rows(rows, pinned):
    B = S.batched_scenes(7, seed=3, lo=1e3, hi=2e4, sizes=(64, 97, 130))
    v = torch.as_tensor(B["vertices"]).cuda()
    f = torch.as_tensor(B["faces"].astype(np.int32)).cuda()
    fo, ro = B["face_offsets"].astype(np.int64), B["ray_offsets"].astype(np.int64)
    r = torch.as_tensor(B["rays"].view(np.float32).reshape(-1, 8)).cuda()
    g = torch.Generator().manual_seed(4)
    for s in range(7):
        if rows == "none" or (rows == "every other" and s % 2) or (rows == "one" and s != 3):
            p = torch.randperm(int(ro[s + 1] - ro[s]), generator=g).cuda()
            r[ro[s]:ro[s + 1]] = r[ro[s]:ro[s + 1]][p]
    b = TriangleBatch()
    if pinned:
        b.set_tuning()
    hits = torch.empty((r.shape[0], 4), device="cuda")
    for _ in range(3):
        hits.fill_(float("nan"))
        b.build_trace(v, f, fo, r, ro, hits=hits)
        torch.cuda.synchronize()
        for s in range(7):
            acc = sb.TriangleAccel()
            acc.Build32(sb.Mesh(v, f[fo[s]:fo[s + 1]].contiguous()))
            want = acc.Traverse(r[ro[s]:ro[s + 1]].contiguous())
            got = hits[ro[s]:ro[s + 1]]
            assert torch.equal(got.view(torch.int32), want.view(torch.int32)), s
