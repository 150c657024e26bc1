"""One solver through both IC(0) orderings: the cluster sweep's shape belongs to
an ordering, since its levels go to shared memory.  The strip is numbered as a
chain, so that the natural ordering has a level per node (10000 in both sweeps,
more than the shared memory holds) and the colour ordering a handful."""
import numpy as np
import pytest

from toastpp_gb300 import capi

pytestmark = pytest.mark.gpu


def strip(nx=50, ny=100):
    """nx x ny grid, rows numbered to and fro: each node is its successor's neighbour."""
    num = np.arange(nx * ny).reshape(ny, nx)
    num[1::2] = num[1::2, ::-1]
    coords = np.empty((nx * ny, 2))
    y, x = np.divmod(np.arange(nx * ny), nx)
    coords[num.ravel()] = np.stack([x, y], 1)
    a, b, c, d = num[:-1, :-1].ravel(), num[:-1, 1:].ravel(), num[1:, 1:].ravel(), num[1:, :-1].ravel()
    return coords, np.concatenate([np.stack([a, b, c], 1), np.stack([a, c, d], 1)]).astype(np.int32)


@pytest.mark.parametrize("orders", [(1, 0, 1), (0, 1)])
def test_shape_follows_the_ordering(orders, monkeypatch):
    monkeypatch.setenv("TOASTGPU_IC_PERSISTENT", "1")
    coords, elems = strip()
    gm = capi.Mesh(coords, elems)
    n = len(coords)
    cm, ck, ca = capi.optical_coefficients(np.full(n, 0.02), np.full(n, 1.0), np.full(n, 1.4))
    B = np.random.default_rng(1).random((4, n))
    s = capi.FwdSolver(gm, "GMRES", 1e-10, "ICH", False, precision="mixed")
    x = {}
    for o in orders:
        s.set_refinement(1e-4, 12, o)
        s.reset(cm, ck, ca, 0.0)
        y, res = s.calc_fields(B)
        assert all(r[1] == 0 for r in res), res
        assert np.array_equal(x.setdefault(o, y), y)
    # two solves to a componentwise backward error of 1e-10
    assert np.linalg.norm(x[0] - x[1]) < 1e-9 * np.linalg.norm(x[1])
