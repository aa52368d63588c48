"""Marches long enough to take bricks, with images on both sides of the size
that picks the kernel: with an opacity of 1e-30 in place of 0 no brick is empty
and no sample's alpha changes (1 - exp of less than 2^-25 is 0, and a sum with
1e-30 rounds to its other term), so the images and transmittances are equal bit
for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from surface_b200 import scenes as S  # noqa: E402
from surface_b200 import volume as V  # noqa: E402
from surface_b200.accel import Context  # noqa: E402

pytestmark = pytest.mark.gpu


def _density(dims, special):
    rng = np.random.default_rng(sum(dims))
    z, y, x = np.meshgrid(*(np.linspace(0, 1, n) for n in dims), indexing="ij")
    rho = np.zeros(dims)
    for _ in range(4):
        c, s = rng.uniform(0.1, 0.9, 3), rng.uniform(0.03, 0.12)
        rho += np.exp(-((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2) / (2 * s * s))
    rho = (rho / rho.max()).astype(np.float32)
    if special == "negative":
        rho -= np.float32(0.4)
    if special == "above":
        rho *= np.float32(3.0)
    if special == "spikes":
        rho *= np.float32(0.03)
        rho.reshape(-1)[rng.integers(0, rho.size, 40)] = 0.9
    if special == "not finite":
        rho.reshape(-1)[rng.integers(0, rho.size, 5)] = np.nan
        rho.reshape(-1)[rng.integers(0, rho.size, 5)] = -np.inf
        rho.reshape(-1)[rng.integers(0, rho.size, 5)] = np.inf
        rho.reshape(-1)[rng.integers(0, rho.size, 5)] = np.finfo(np.float32).max
    return torch.as_tensor(rho, device="cuda")


SAMPLING = {"plain": None,
            "repeat": dict(clamp=(False, True, False)),
            "remap": dict(remap=(None, S.exp_coord_map(40), None)),
            "remap, repeat": dict(remap=(S.exp_coord_map(65), None, S.exp_coord_map(9)),
                                  clamp=(False, False, True))}


@pytest.mark.parametrize("image", [(420, 330, 0.0123, 150), (333, 270, 0.0082, 200)])
@pytest.mark.parametrize("dims", [(64, 64, 64), (33, 20, 290), (8, 9, 7), (1, 40, 17)])
@pytest.mark.parametrize("special", ["plain", "negative", "above", "spikes", "not finite"])
@pytest.mark.parametrize("sampling", list(SAMPLING))
def test_empty_bricks_change_nothing(image, dims, special, sampling):
    w, h, step, few = image
    assert (w * h >= 1 << 17) == (w == 420)
    smp = SAMPLING[sampling] and V.Sampling(**SAMPLING[sampling])
    rho = _density(dims, special)
    tf = torch.as_tensor(S.transfer_function(64, seed=3), device="cuda")
    tf[40:44, 3] = 0.0  # a transparent band inside the opaque part
    marched = tf.clone()
    marched[marched[:, 3] == 0, 3] = 1e-30
    ctx = Context.default()
    for eye, look, most in (((0, 0, 3), (0, 0, 0), 8192), ((1.9, -1.4, 2.2), (0, 0, 0), few),
                            ((0.2, 0.1, -0.3), (0.9, 0.4, 0.5), 8192)):
        p = V.camera(w, h, eye=eye, lookat=look, step=step, max_steps=most)
        before = ctx.L.srt_ctx_launch_count(ctx.h)
        a, ta = V.march(rho, tf, p, sampling=smp)
        b, tb = V.march(rho, marched, p, sampling=smp)
        assert ctx.L.srt_ctx_launch_count(ctx.h) - before == 4  # bricks and march, twice
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
        assert torch.equal(ta.view(torch.int32), tb.view(torch.int32))
