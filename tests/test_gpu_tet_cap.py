"""The step cap of tetrahedron walks in the reference's order counts every
node popped: a ray whose walk pops T nodes is refused at a cap of T - 1 and
passes at T, also when the last nodes popped are children that it misses."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import surface_b200 as sb  # noqa: E402
from surface_b200 import _lib  # noqa: E402
from surface_b200 import scenes as S  # noqa: E402

from test_gpu_stats import traced  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("target", ["hit", "graze", "miss"])
def test_cap_is_the_number_of_nodes_popped(target):
    v, f, _ = S.tet_grid(8, seed=4)
    acc = sb.TetraAccel()
    acc.Build32(sb.Tetrahedron(torch.as_tensor(v).cuda(),
                               torch.as_tensor(f.astype(np.int32)).cuda()))
    n = 40
    rng = np.random.default_rng(5)
    o = 0.5 + 2.0 * S._normalize(rng.normal(size=(n, 3)))
    to = {"hit": 0.3 * rng.uniform(-1, 1, size=(n, 3)) + 0.5,
          # near the cube's edges: the box is entered, the mesh missed or just hit
          "graze": np.where(rng.uniform(size=(n, 3)) < 0.7, rng.integers(0, 2, size=(n, 3)),
                            rng.uniform(size=(n, 3))) * 1.002 - 0.001,
          "miss": 0.5 + 1.2 * S._normalize(rng.normal(size=(n, 3)))}[target]
    rays = S.make_rays(o, to - o)
    single = _lib.SRT_TRACE_SINGLE_PASS
    for k in range(n):
        one = rays[k:k + 1]
        h, st, s = traced(acc, one, flags=single)
        pops = st[0]
        assert s == _lib.SRT_OK and pops >= 1
        g, _, s = traced(acc, one, flags=single, max_iter=pops)
        assert s == _lib.SRT_OK and torch.equal(g.view(torch.int32), h.view(torch.int32))
        if pops > 1:
            assert traced(acc, one, flags=single, max_iter=pops - 1)[2] == _lib.SRT_ERR_LIMIT
