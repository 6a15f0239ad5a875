"""The FP32-form force of the one-point scheme and of one and 27 Gauss points,
with 32, 8 and 4 lanes per node, against the FP64 force; and its fused stages
against the stages apart, bit for bit."""
import numpy as np
import pytest

import pdmtel_b200 as P

pytestmark = pytest.mark.gpu

H = 1e-3
RULES = {1: ([0.0], [2.0]), 3: ([-np.sqrt(0.6), 0.0, np.sqrt(0.6)], [5 / 9, 8 / 9, 5 / 9])}


def context(dims, points, factors):
    r = np.random.default_rng(2)
    z, y, x = np.meshgrid(*[np.arange(n) - (n - 1) / 2 for n in dims[::-1]], indexing="ij")
    xyz = np.stack([x, y, z], -1).reshape(-1, 3) * H
    n = len(xyz)
    mats = [dict(spring=2e19 * (1 + k), density=2440.0, ecrit=1e20, grav=(0.0, 1e5, -2e5)) for k in range(2)]
    bc = np.full(n, -1, dtype=np.int32)
    bc[:9] = 0
    gauss = (dict(integration=P.INTG_FGI, intg_point=points, abscissae=RULES[points][0], weights=RULES[points][1])
             if points else dict(integration=P.INTG_CCI, cci_modified=int(factors)))
    ctx = P.DeviceContext.create(xyz, np.arange(n) % 2, mats, [dict(type=P.BC_DISPL, dir=(1, 0, 1), value=(1e-6, 0, 2e-6))],
                                 bc, grid_spacing=H, horizon=3.015 * H,
                                 slits=[(-0.2 * dims[0] * H, 0.2 * dims[0] * H, 0.3 * H, 0.3 * H, -1.0, 1.0)],
                                 spring_factor=np.exp(0.2 * r.standard_normal(n)) if factors else None, **gauss)
    ctx.bond_search()
    if factors:
        ctx.set_bdry_eff(1.0 + 0.1 * r.random(n))
    if points > 1:  # one point takes the node's displacement
        ctx.mls_setup(3.0 * H)
    ctx.set_energy(False)
    return ctx, xyz


@pytest.mark.parametrize("dims,points", [((5, 4, 3), 0), ((33, 23, 17), 0), ((149, 111, 8), 0), ((5, 4, 3), 1),
                                         ((33, 23, 17), 1), ((149, 111, 8), 1), ((9, 7, 5), 3), ((33, 23, 17), 3)])
@pytest.mark.parametrize("factors", [False, True])
def test_any_points(dims, points, factors):
    ctx, x = context(dims, points, factors)
    r = np.random.default_rng(8)
    U = 1e-3 * (x @ r.standard_normal((3, 3)) + 0.3 * H * r.standard_normal(x.shape))
    V = r.standard_normal(x.shape)
    k = []
    for precision in (P.PREC_FP64, P.PREC_FP32C):
        ctx.set_precision(precision)
        ctx.reset_state()
        ctx.set_state(U, np.zeros_like(V))
        if points:
            ctx.gather(0.0)
        ctx.init_dynamic()
        k.append(ctx.force_stage(1e-9, 1e-9, U.ravel()))
    # some 20 roundings of 2^-24 per term; 250 terms of either sign, whose
    # magnitudes add up to some 16 times their sum
    assert np.max(np.abs(k[1] - k[0])) <= 20 * 16 * 2.0 ** -24 * np.max(np.abs(k[0]))
    out = []
    for apart in (True, False):
        ctx.reset_state()
        ctx.set_state(U, V)
        if points:
            ctx.gather(0.0)
        if apart:
            ctx.profile_step(1e-9, 1e-9)
        else:
            ctx.rk4_steps(1e-9, 0.0, 1)
        ctx.sync()
        out.append(ctx.get_state() + (ctx.get_vbuf(),))
    for a, b in zip(*out):
        assert np.all(np.isfinite(a)) and np.array_equal(a, b)
    ctx.close()
