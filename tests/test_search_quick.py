"""The bond search's decision from the separation alone against the oracle's
search: lattices, jittered lattices whose distances to a cell straddle the
horizon and the margins around it, nodes closer than half a spacing, horizons
from half a spacing up, families beyond 256, and coordinates far from the
origin (where nothing is decided early)."""
import numpy as np
import pytest

import oracle_lib as O
import pdmtel_b200 as P

pytestmark = pytest.mark.gpu


def _nodes(kind, dims, dx, r):
    g = np.stack(np.meshgrid(*[np.arange(n) for n in dims[::-1]], indexing="ij"), -1)[..., ::-1].reshape(-1, 3)
    x = (g - np.array(dims) / 2.0) * dx
    if kind == "jitter":
        x = x + r.uniform(-0.3, 0.3, x.shape) * dx
    elif kind == "slight":  # within the margin of the lattice distances
        x = x + r.uniform(-0.02, 0.02, x.shape) * dx
    elif kind == "close":
        x = np.concatenate([x, x[::3] + r.uniform(-0.4, 0.4, x[::3].shape) * dx])
    elif kind == "far":
        x = x + 1e11 * dx
    return np.ascontiguousarray(x.reshape(-1))


@pytest.mark.parametrize("horizon", [0.5, 1.0, 2.96, 3.015, 4.2])
@pytest.mark.parametrize("kind", ["lattice", "slight", "jitter", "close", "far"])
def test_search_equals_oracle(kind, horizon):
    dx = 1e-3
    x = _nodes(kind, (9, 8, 7) if horizon < 4 else (11, 11, 11), dx, np.random.default_rng(4))
    n = x.size // 3
    slit = [(-2.2 * dx, 1.7 * dx, 0.31 * dx, 0.31 * dx, -1.0, 1.0)]
    ctx = P.DeviceContext.create(x, np.zeros(n, np.int32), [dict(spring=1.0, density=1.0, ecrit=1e20)],
                                 grid_spacing=dx, horizon=horizon * dx, integration=P.INTG_CCI, slits=slit)
    halves, broken, shortest = ctx.bond_search()
    rp, col, br = ctx.get_family(halves)
    want_rp, want_col, want_min = O.bond_search(x, dx, horizon * dx)
    assert np.array_equal(rp, want_rp) and np.array_equal(col, want_col)
    assert shortest == want_min
    assert np.array_equal(br, O.slit_mark(x, want_rp, want_col, slit))
    assert broken == br.sum()
    ctx.close()
