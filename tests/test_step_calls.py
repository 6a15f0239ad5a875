"""pd_rk4_step on a stream that takes no capture."""
import numpy as np
import pytest

import pdmtel_b200 as P

pytestmark = pytest.mark.gpu

H = 1e-3
LEGACY = 1  # the handle of the legacy default stream


def context(dims=(6, 5, 4), stream=None):
    z, y, x = np.meshgrid(*[np.arange(n) * H for n in dims[::-1]], indexing="ij")
    xyz = np.stack([x, y, z], -1).reshape(-1, 3)
    ctx = P.DeviceContext.create(xyz, np.zeros(len(xyz), np.int32), [dict(spring=2e19, density=2440.0, ecrit=1e20)],
                                 grid_spacing=H, horizon=3.015 * H, integration=P.INTG_CCI, stream=stream)
    ctx.bond_search()
    ctx.set_state(1e-6 * np.random.default_rng(1).standard_normal(3 * ctx.n), np.zeros(3 * ctx.n))
    return ctx


def test_legacy_default_stream():
    out = []
    for stream in (None, LEGACY):
        ctx = context(stream=stream)
        energies = [ctx.rk4_step(1e-9, 1e-9 * (k + 1)) for k in range(5)]
        out.append((energies, ctx.get_state()))
        ctx.close()
    (ea, a), (eb, b) = out
    assert ea == eb and np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
