"""Builds and loads with little device memory left: with room for the
two-child nodes but not for the wide ones behind them, the accel is walked by
the former and finds the same hits; with less, the call reports that memory is
short and the next one, with memory again, works."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import surface_b200 as sb  # noqa: E402
from surface_b200 import _lib  # noqa: E402
from surface_b200 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _kernels(acc, rays, hits):
    """Kernels of a trace: the wide walk and the replay, or the two-child
    walk besides."""
    before = acc.L.srt_ctx_launch_count(acc.ctx.h)
    acc.Traverse(rays, hits=hits)
    return acc.L.srt_ctx_launch_count(acc.ctx.h) - before


# a load holds a wide node for each branch; a build for each that a tree of up
# to 2^18 + 1 primitives could have
@pytest.mark.parametrize("how,n", [("load", 3_000_000), ("build", (1 << 18) + 1)])
def test_wide_nodes_that_do_not_fit(how, n, tmp_path):
    pos, rad = S.particles(n, seed=3, median_radius=0.3 / n ** (1 / 3))
    data = sb.Particles(torch.as_tensor(pos).cuda(), torch.as_tensor(rad).cuda())
    rays = torch.as_tensor(S.pinhole_rays(200, 150, (0.5, 0.5, 2.2), (0.5, 0.5, 0.5), fov_deg=30)
                           .view(np.float32).reshape(-1, 8)).cuda()
    hits = torch.empty((rays.shape[0], 4), device="cuda")
    path = str(tmp_path / "a.bin")

    def make():
        acc = sb.ParticleAccel()
        if how == "load":
            acc.Load(path, data)
        else:
            acc.Build32(data)
        return acc

    # (also grows the context's scratch for all that follows)
    whole = sb.ParticleAccel()
    whole.Build32(data)
    want = whole.Traverse(rays)
    assert (want[:, 3].view(torch.int32) != -1).float().mean() > 0.2
    nodes = whole.info().num_branches if how == "load" else n - 1
    whole.Dump(path)
    whole.close()
    first = make()
    assert _kernels(first, rays, hits) == 2
    first.close()
    wide_mb = nodes * 128 / MB
    rest_mb = ((4 + 4 + 16) * n + nodes * 64) / MB  # codes, order, records, two-child nodes
    seen = []
    for room in np.arange(rest_mb + wide_mb + 24, rest_mb - 24, -wide_mb / 4):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        hold = torch.empty(max(0, torch.cuda.mem_get_info()[0] - int(room * MB)),
                           dtype=torch.uint8, device="cuda")
        acc = None
        try:
            acc = make()
        except sb.SurfaceError as e:
            assert e.status == _lib.SRT_ERR_NO_MEMORY
            seen.append(2)
        else:
            hits.fill_(float("nan"))
            seen.append(_kernels(acc, rays, hits) - 2)
            acc.ctx.synchronize()
            assert torch.equal(hits.view(torch.int32), want.view(torch.int32))
            acc.Traverse(rays, hits=hits, grid_launch=True)
            assert torch.equal(hits.view(torch.int32), want.view(torch.int32))
            acc.close()
        del acc, hold
    torch.cuda.empty_cache()
    print(seen)
    # all of it, the two-child nodes alone, refused -- in this order as room shrinks
    assert seen == sorted(seen) and seen[0] == 0 and 1 in seen
    acc = make()
    assert _kernels(acc, rays, hits) == 2
    assert torch.equal(hits.view(torch.int32), want.view(torch.int32))
