"""Scene traces of enough rays to be taken in tiles of their rows, against the
same rays shuffled (which have no rows and keep array order): identical hits
and elements, bit for bit, with widths and counts that leave part tiles, for
primaries and for secondaries with their previous elements."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from surface_b200 import scenes as S  # noqa: E402

from test_gpu_scene import make_pair  # noqa: E402

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.float32).reshape(len(a), -1)).cuda()


@pytest.mark.parametrize("width,n", [(1024, 1 << 20), (1030, 1030 * 1023 + 77),
                                     (1024, (1 << 20) - 1)])
@pytest.mark.parametrize("more", [False, True])
def test_tiles_match_array_order(width, n, more):
    g, _, _, lo, hi = make_pair(
        S.scene_elements(seed=43, nline=1, nsolid=1) if more else S.scene_elements(seed=31))
    c = (lo.min(0) + hi.max(0)) / 2
    eye = c + (hi.max(0) - lo.min(0)) * np.array([0.9, 0.7, 1.3])
    rays = S.pinhole_rays(width, -(-n // width), eye, c, fov_deg=45)[:n].copy()
    perm = np.random.default_rng(3).permutation(n)
    at = torch.from_numpy(perm).cuda()
    rt = _dev(rays)
    prev = pn = None
    for _ in range(2):  # primaries, then the same rays past the primitives they hit
        hits, el = g.Trace(rt, prev, pn)
        ph, pe = g.Trace(rt[at].contiguous(), *(x if x is None else x[at].contiguous()
                                                for x in (prev, pn)))
        el, pe = el.view(torch.int32), pe.view(torch.int32)
        assert float((el != -1).float().mean()) > 0.05
        assert torch.equal(hits[at].view(torch.int32), ph.view(torch.int32))
        assert torch.equal(el[at], pe)
        rt = rt.clone()
        rt[:, 3] = hits[:, 3]
        prev, pn = el, torch.nn.functional.normalize(rt[:, 4:7]).neg().contiguous()
