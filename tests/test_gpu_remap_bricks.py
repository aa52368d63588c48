"""Remap tables whose values leave [0, 1]: on a clamped axis the fetch then
extrapolates from the edge texels (or rounds far from them), so a sample may
reach opaque table entries although no texel of its brick does.  Such samples
are marched: the image equals that of a table with no transparent entry (an
opacity of 1e-30 changes no sample's alpha), bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from surface_b200 import scenes as S  # noqa: E402
from surface_b200 import volume as V  # noqa: E402
from surface_b200.accel import Context  # noqa: E402

pytestmark = pytest.mark.gpu

N = 192  # texels along the remapped axis


def _table(values):
    t = np.linspace(0.0, 1.0, 60).astype(np.float32)
    if values.startswith("below"):
        t = np.linspace(-0.1, 1.0, 60).astype(np.float32)
    if values == "far above":
        t[-6:] = np.float32(3e6) * np.arange(1, 7, dtype=np.float32)
    if values == "nan":
        t[20:24] = np.nan
    if values == "infinite":
        t[30], t[31] = np.inf, -np.inf
    if values == "huge":
        t[5:9] = np.float32([1e30, -1e30, 3e9, 7.25])
    return np.repeat(t, 100) if values == "below, long" else t


@pytest.mark.parametrize("values", ["inside", "below", "below, long", "far above", "nan",
                                    "infinite", "huge"])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("clamp", [True, False])
def test_values_outside_the_unit_interval(values, axis, clamp):
    # transparent everywhere: at most 0.04 where the table's opacity starts at
    # 0.05, falling steeply at the low edge of the axis and not quite the same
    # number from texel to texel
    line = np.where(np.arange(N) < 8, 0.04 - 0.005 * np.arange(N), 0.03).astype(np.float32)
    rho = np.broadcast_to(line.reshape([-1 if k == 2 - axis else 1 for k in range(3)]),
                          [N if k == 2 - axis else 24 for k in range(3)])
    rho = torch.as_tensor(np.ascontiguousarray(rho), device="cuda")
    tf = torch.as_tensor(S.transfer_function(256, seed=3), device="cuda")
    marched = tf.clone()
    marched[marched[:, 3] == 0, 3] = 1e-30
    smp = V.Sampling(remap=tuple(_table(values) if k == axis else None for k in range(3)),
                     clamp=(clamp,) * 3)
    p = V.camera(420, 330, eye=(1.2, 0.9, 2.4), step=0.0123)
    ctx = Context.default()
    before = ctx.L.srt_ctx_launch_count(ctx.h)
    a, ta = V.march(rho, tf, p, sampling=smp)
    assert ctx.L.srt_ctx_launch_count(ctx.h) - before == 2  # the bricks, the march
    b, tb = V.march(rho, marched, p, sampling=smp)
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    assert torch.equal(ta.view(torch.int32), tb.view(torch.int32))
    # what the case is about: an image that is not the transparent one
    if clamp:
        assert (values == "inside") == bool((a == 0).all())
