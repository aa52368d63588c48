"""Batches without rays, and with scenes that have none among scenes that
have some: accepted with every ray order, through capture and replay."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from surface_b200 import scenes as S  # noqa: E402
from surface_b200.batch import TriangleBatch  # noqa: E402

pytestmark = pytest.mark.gpu


def _batch():
    B = S.batched_scenes(4, seed=5, lo=1e3, hi=9e3, sizes=(64, 80), min_faces=2)
    return (torch.as_tensor(B["vertices"]).cuda(),
            torch.as_tensor(B["faces"].view(np.int32)).cuda(), B["face_offsets"],
            torch.as_tensor(B["rays"].view(np.float32).reshape(-1, 8)).cuda(),
            B["ray_offsets"].astype(np.int64))


@pytest.mark.parametrize("sort_bits", [None, 0, 12, 22])
def test_no_rays_at_all(sort_bits):
    v, f, fo, r, _ = _batch()
    b = TriangleBatch()
    if sort_bits is not None:
        b.set_tuning(sort_bits=sort_bits)
    hits = torch.full((1, 4), 7.0, device="cuda")
    for _ in range(3):
        b.build_trace(v, f, fo, r[:1].contiguous(), np.zeros(5, np.int64), hits=hits)
    torch.cuda.synchronize()
    assert (hits == 7.0).all()


@pytest.mark.parametrize("sort_bits", [None, 0, 12, 22])
def test_scenes_without_rays_between_others(sort_bits):
    v, f, fo, r, ro = _batch()
    want = TriangleBatch()
    want.set_tuning()
    all_hits = want.build_trace(v, f, fo, r, ro).clone()
    keep = [(ro[0], ro[1]), None, (ro[2], ro[3]), None]
    rays = torch.cat([r[a:b] for a, b in filter(None, keep)])
    off = np.concatenate([[0], np.cumsum([0 if k is None else k[1] - k[0] for k in keep])])
    b = TriangleBatch()
    if sort_bits is not None:
        b.set_tuning(sort_bits=sort_bits)
    hits = torch.empty((rays.shape[0], 4), device="cuda")
    for _ in range(3):
        hits.fill_(float("nan"))
        b.build_trace(v, f, fo, rays, off, hits=hits)
        torch.cuda.synchronize()
        expect = torch.cat([all_hits[x:y] for x, y in filter(None, keep)])
        assert torch.equal(hits.view(torch.int32), expect.view(torch.int32))
