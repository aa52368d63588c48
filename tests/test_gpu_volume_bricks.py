"""The forward march skips the bricks that the transfer function leaves
transparent.  With an opacity of 1e-30 in place of 0 every brick is marched
and no sample's alpha changes (1 - exp of less than 2^-25 is 0, and a sum with
1e-30 rounds to its other term): the images and transmittances are equal bit
for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from surface_b200 import scenes as S  # noqa: E402
from surface_b200 import volume as V  # noqa: E402

pytestmark = pytest.mark.gpu


def _density(dims, special):
    d, h, w = dims
    rng = np.random.default_rng(d * h + w)
    z, y, x = np.meshgrid(*(np.linspace(0, 1, n) for n in dims), indexing="ij")
    rho = np.zeros(dims)
    for _ in range(5):
        c, s = rng.uniform(0.1, 0.9, 3), rng.uniform(0.05, 0.2)
        rho += np.exp(-((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2) / (2 * s * s))
    rho = (rho / rho.max()).astype(np.float32)
    if special == "negative":
        rho -= np.float32(0.4)
    if special == "above":
        rho *= np.float32(3.0)
    if special == "spikes":
        rho *= np.float32(0.03)
        rho.reshape(-1)[rng.integers(0, rho.size, 40)] = 0.9
    if special == "nan":
        rho.reshape(-1)[rng.integers(0, rho.size, 5)] = np.nan
        rho.reshape(-1)[rng.integers(0, rho.size, 5)] = -np.inf
    return torch.as_tensor(rho, device="cuda")


@pytest.mark.parametrize("dims", [(64, 64, 64), (33, 20, 290), (8, 9, 7), (1, 40, 17)])
@pytest.mark.parametrize("special", ["plain", "negative", "above", "spikes", "nan"])
@pytest.mark.parametrize("view", ["front", "oblique", "inside", "remap"])
def test_bricks_change_nothing(dims, special, view):
    eye = {"front": (0, 0, 3), "oblique": (1.9, -1.4, 2.2), "inside": (0.2, 0.1, -0.3),
           "remap": (0.7, 0.3, 2.9)}[view]
    look = (0, 0, 0) if view != "inside" else (0.9, 0.4, 0.5)
    p = V.camera(333, 270, eye=eye, lookat=look, step=0.0123, max_steps=150 if view == "oblique"
                 else 8192)
    smp = (V.Sampling(remap=(None, S.exp_coord_map(40), None), clamp=(False, True, False))
           if view == "remap" else None)
    rho = _density(dims, special)
    tf = torch.as_tensor(S.transfer_function(64, seed=3), device="cuda")
    tf[40:44, 3] = 0.0  # a transparent band inside the opaque part
    marched = tf.clone()
    marched[marched[:, 3] == 0, 3] = 1e-30
    a, ta = V.march(rho, tf, p, sampling=smp)
    b, tb = V.march(rho, marched, p, sampling=smp)
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    assert torch.equal(ta.view(torch.int32), tb.view(torch.int32))


def test_colour_that_is_not_finite_is_not_skipped():
    p = V.camera(320, 300, step=0.01)
    tf = torch.as_tensor(S.transfer_function(64, seed=3), device="cuda")
    tf[0, 1] = float("inf")
    img, _ = V.march(torch.zeros(16, 16, 16, device="cuda"), tf, p)
    assert torch.isnan(img[150, 160, 1])
