"""The sphere build above 2^18 spheres, which packs centre and radius before
the sort and gathers them afterwards: tree, order and hits against the oracle
on both sides of that size, with a radius each and with one for all, and
repeated in one context by sizes that go up and down (the packed records share
the refit's scratch)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import surface_b200 as sb  # noqa: E402
from oracle import oracle as O  # noqa: E402
from surface_b200 import scenes as S  # noqa: E402

from conftest import bits  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radii", [True, False])
def test_both_sides_of_the_size(radii):
    rays = S.pinhole_rays(96, 96, (0.5, 0.5, 2.2), (0.5, 0.5, 0.5), fov_deg=30)
    acc = sb.ParticleAccel()
    for n in (262_144, 262_145, 300_001, 262_143, 270_000):
        pos, rad = S.particles(n, seed=n)
        rad = rad * 8 if radii else None
        const = 0.0 if radii else 0.004
        acc.Build32(sb.Particles(pos, rad, const))
        o = O.OracleAccel(O.SPHERE, pos, None, rad, const)
        got = acc.Traverse(rays)
        want = o.trace(rays)
        assert (want["prim"] != O.MISS).mean() > 0.05
        assert np.array_equal(got["prim"], want["prim"])
        assert np.array_equal(bits(got["t"]), bits(want["t"]))
