"""The sort of large builds (8-bit passes over tiles of 8,192 keys): the order
of the build is the stable order of its codes, at tile edges, for one digit
value throughout and for scenes sorted together."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import surface_b200 as sb  # noqa: E402
from surface_b200 import _lib  # noqa: E402

pytestmark = pytest.mark.gpu


def _points(n, special):
    rng = np.random.default_rng(n)
    p = rng.random((n, 3), dtype=np.float32)
    if special == "same":
        p[:] = 0.5
    if special == "line":
        p[:, 1:] = 0.25
    if special == "ordered":
        p = p[np.lexsort(p.T)]
    return p


@pytest.mark.parametrize("n", [(1 << 18) + 1, 33 * 8192 - 1, 33 * 8192, 33 * 8192 + 1, 1000003])
@pytest.mark.parametrize("special", ["uniform", "same", "line", "ordered"])
def test_build_order_is_the_stable_order(n, special):
    p = _points(n, special)
    codes, _ = sb.stage_morton(_lib.SRT_SPHERES, p, constant_radius=1e-3)
    acc = sb.ParticleAccel()
    for _ in range(2):  # the look-back words of an earlier sort must not count
        acc.Build32(sb.Particles(p, constantRadius=1e-3))
        _, idx, sorted_codes = acc.export()
        want = np.argsort(codes, kind="stable")
        assert np.array_equal(idx, want)
        assert np.array_equal(sorted_codes, codes[want])


def test_scenes_sorted_together_match_single_builds():
    from surface_b200 import scenes as S
    from surface_b200.batch import TriangleBatch
    B = S.batched_scenes(nscenes=7, seed=9, lo=2e4, hi=1e5, sizes=(64,))
    v = torch.as_tensor(B["vertices"]).cuda()
    f = torch.as_tensor(B["faces"].astype(np.int32)).cuda()
    r = torch.as_tensor(B["rays"].view(np.float32).reshape(-1, 8)).cuda()
    assert f.shape[0] > 1 << 17
    b = TriangleBatch()
    b.set_tuning()
    hits = torch.empty(r.shape[0], 4, device="cuda")
    for _ in range(4):  # eager, eager, then replays of the captured graph
        hits.zero_()
        b.build_trace(v, f, B["face_offsets"], r, B["ray_offsets"], hits=hits)
    torch.cuda.synchronize()
    for s in range(7):
        fo, ro = B["face_offsets"].astype(int), B["ray_offsets"].astype(int)
        acc = sb.TriangleAccel()
        acc.Build32(sb.Mesh(v, f[fo[s]:fo[s + 1]].contiguous()))
        want = acc.Traverse(r[ro[s]:ro[s + 1]].contiguous())
        assert torch.equal(hits[ro[s]:ro[s + 1]].view(torch.int32), want.view(torch.int32))
