"""The bond weight c V / r^3 of the family-list static operator and its
right-hand side is the quotient of the rounded r^2 r, each operation rounded
once: pairs of nodes along one axis, whose rows are a few products that numpy
forms alike, bit for bit; separations inside and outside the range of the
branch-free root and quotient."""
import math

import numpy as np
import pytest

import pdmtel_b200 as P

pytestmark = pytest.mark.gpu

H, C = 1e-3, 2.3e19


@pytest.mark.parametrize("pairs", [1001, 8003])  # a warp per node, eight lanes
@pytest.mark.parametrize("scale", [1.0, 1e-70, 1e60])
def test_weight_is_rounded_once(pairs, scale):
    r = np.random.default_rng(9)
    a = H * scale * r.uniform(0.3, 3.0, pairs)
    n = 2 * pairs
    xyz = np.zeros((n, 3))
    xyz[:, 1] = np.repeat(np.arange(pairs) * 10 * H, 2)
    xyz[1::2, 0] = a
    bc = np.full(n, -1, np.int32)
    bc[1::2] = 0
    ctx = P.DeviceContext.create(
        xyz, np.zeros(n, np.int32), [dict(spring=C, density=2440.0, ecrit=1e20)],
        [dict(type=P.BC_DISPL, dir=(1, 0, 0), value=(1.0, 0.0, 0.0))], bc, grid_spacing=H, horizon=3.015 * H,
        integration=P.INTG_CCI)
    ctx.set_family(np.arange(n + 1), np.arange(n) ^ 1)
    ctx.set_option(P.OPT_STATIC_STENCIL, 0)
    r2 = a * a
    w = (C * math.pow(H, 3.0)) / (r2 * np.sqrt(r2))
    x = np.zeros((n, 3))
    x[0::2, 0] = 1.0
    y = ctx.static_matvec(1.0, x).reshape(n, 3)
    assert np.array_equal(y[0::2, 0], w * a * a)  # the far end is prescribed: masked to zero
    b = ctx.static_rhs(1.0).reshape(n, 3)
    assert np.array_equal(b[0::2, 0], w * a * a) and np.all(b[1::2, 0] == 1.0)
    ctx.close()
