"""The buffers that streams keep for their marches' brick marks: more streams
than have one, buffers that grow between marches, and several threads on one
stream each give what a march by itself gives."""
import threading

import pytest

torch = pytest.importorskip("torch")

from surface_b200 import scenes as S  # noqa: E402
from surface_b200 import volume as V  # noqa: E402
from surface_b200.accel import Context  # noqa: E402

pytestmark = pytest.mark.gpu


def _volume(seed, side):
    """A dense ball somewhere."""
    g = torch.Generator().manual_seed(seed)
    c = torch.rand(3, generator=g) * 0.6 + 0.2
    ax = torch.linspace(0, 1, side, device="cuda")
    z, y, x = torch.meshgrid(ax, ax, ax, indexing="ij")
    d = ((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2).sqrt()
    return (1.0 - 6.0 * d).clamp(min=0).contiguous()


def _camera():
    return V.camera(420, 330, eye=(1.2, 0.9, 2.4), step=0.0123)


def _same(a, b):
    return all(torch.equal(x.view(torch.int32), y.view(torch.int32)) for x, y in zip(a, b))


def test_many_streams_and_growing_buffers():
    ctx = Context(0)
    tf = torch.as_tensor(S.transfer_function(256, seed=3), device="cuda")
    p = _camera()
    # the third has more bricks than the first buffer of a stream has room for
    x = torch.linspace(0, 1, 600_000, device="cuda")
    vols = [_volume(0, 40), _volume(1, 96),
            (1.0 - 9.0 * (x - 0.4).abs()).clamp(min=0).reshape(1, 1, -1), _volume(3, 64)]
    want = [V.march(v, tf, p) for v in vols]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(12)]
    got = []
    for turn in range(3):
        for j, s in enumerate(streams):
            k = (j + turn) % len(vols)
            with torch.cuda.stream(s):
                before = ctx.L.srt_ctx_launch_count(ctx.h)
                got.append((k, V.march(vols[k], tf, p, ctx=ctx)))
                assert ctx.L.srt_ctx_launch_count(ctx.h) - before == 2
    ctx.close()  # waits for the marches under way
    torch.cuda.synchronize()
    for k, out in got:
        assert _same(out, want[k])


def test_threads_on_one_stream():
    ctx = Context(0)
    tf = torch.as_tensor(S.transfer_function(256, seed=3), device="cuda")
    p = _camera()
    vols = [_volume(k, 96) for k in range(4)]
    want = [V.march(v, tf, p) for v in vols]
    torch.cuda.synchronize()
    got = {}

    def work(k):
        for turn in range(20):
            got[k, turn] = V.march(vols[k], tf, p, ctx=ctx)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for (k, _), out in got.items():
        assert _same(out, want[k])
