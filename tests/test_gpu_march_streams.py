"""Marches own the memory that they use: two at once on two streams, and one
in a CUDA graph that is replayed after larger marches, give what each gives by
itself."""
import pytest

torch = pytest.importorskip("torch")

from surface_b200 import scenes as S  # noqa: E402
from surface_b200 import volume as V  # noqa: E402
from surface_b200.accel import Context  # noqa: E402

pytestmark = pytest.mark.gpu


def _volumes(n, side=96):
    """Densities with a dense ball each, somewhere else in each."""
    ax = torch.linspace(0, 1, side, device="cuda")
    z, y, x = torch.meshgrid(ax, ax, ax, indexing="ij")
    g = torch.Generator().manual_seed(7)
    out = []
    for _ in range(n):
        c = torch.rand(3, generator=g) * 0.6 + 0.2
        d = ((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2).sqrt()
        out.append((1.0 - 6.0 * d).clamp(min=0).contiguous())
    return out


def _bricks(ctx, run):
    """run()'s outputs; it marched with bricks (their kernel and the march)."""
    before = ctx.L.srt_ctx_launch_count(ctx.h)
    out = run()
    assert ctx.L.srt_ctx_launch_count(ctx.h) - before == 2
    return out


def _same(a, b):
    return all(torch.equal(x.view(torch.int32), y.view(torch.int32)) for x, y in zip(a, b))


def test_marches_at_once_on_two_streams():
    ctx = Context.default()
    tf = torch.as_tensor(S.transfer_function(256, seed=3), device="cuda")
    p = V.camera(420, 330, eye=(1.2, 0.9, 2.4), step=0.0123)
    vols = _volumes(8)
    want = [_bricks(ctx, lambda v=v: V.march(v, tf, p)) for v in vols]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = {}
    for turn in range(4):
        for k, v in enumerate(vols):
            with torch.cuda.stream(streams[(k + turn) % 2]):
                got[turn, k] = V.march(v, tf, p)
    torch.cuda.synchronize()
    for (_, k), out in got.items():
        assert _same(out, want[k])


@pytest.mark.parametrize("used", [False, True])
def test_march_in_a_graph(used):
    ctx = Context(0)
    tf = torch.as_tensor(S.transfer_function(256, seed=3), device="cuda")
    p = V.camera(420, 330, eye=(1.2, 0.9, 2.4), step=0.0123)
    first, second = _volumes(2)
    want = [V.march(v, tf, p) for v in (first, second)]
    vol = first.clone()
    torch.cuda.synchronize()
    if used:
        V.march(vol, tf, p, ctx=ctx)
        torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = _bricks(ctx, lambda: V.march(vol, tf, p, ctx=ctx))
    big = _volumes(1, 200)[0]
    q = V.camera(840, 660, eye=(1.2, 0.9, 2.4), step=0.0123)
    for v, w in ((first, want[0]), (second, want[1]), (first, want[0])):
        _bricks(ctx, lambda: V.march(big, tf, q, ctx=ctx))  # a larger one between replays
        vol.copy_(v)
        g.replay()
        _bricks(ctx, lambda: V.march(big, tf, q, ctx=ctx))
        torch.cuda.synchronize()
        assert _same(out, w)
    ctx.close()
    g.replay()  # the graph's memory is its own
    torch.cuda.synchronize()
    assert _same(out, want[0])
