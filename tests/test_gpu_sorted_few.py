"""sort_rays on both sides of the count from which rays are first looked at for
rows, in rows and shuffled: the hits of the unsorted trace."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import surface_b200 as sb  # noqa: E402
from surface_b200 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 700, (1 << 15) - 1, 1 << 15])
@pytest.mark.parametrize("rows", [True, False])
def test_sorted_hits(n, rows):
    v, f, _ = S.tet_grid(12, seed=2)
    acc = sb.TetraAccel()
    acc.Build32(sb.Tetrahedron(torch.as_tensor(v).cuda(),
                               torch.as_tensor(f.astype(np.int32)).cuda()))
    rays = S.pinhole_rays(256, 129, (1.7, 1.3, 2.1), (0.5, 0.5, 0.5))[:n]
    r = torch.as_tensor(rays.view(np.float32).reshape(-1, 8)).cuda()
    if not rows:
        r = r[torch.randperm(n, generator=torch.Generator().manual_seed(n)).cuda()].contiguous()
    want = acc.Traverse(r)
    before = acc.L.srt_ctx_launch_count(acc.ctx.h)
    got = acc.Traverse(r, sort_rays=True)
    few = acc.L.srt_ctx_launch_count(acc.ctx.h) - before
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    if n == (1 << 15) - 1:  # two kernels fewer than with a look
        more = torch.cat([r, r[:1]])
        before = acc.L.srt_ctx_launch_count(acc.ctx.h)
        acc.Traverse(more, sort_rays=True)
        assert acc.L.srt_ctx_launch_count(acc.ctx.h) - before == few + 2
