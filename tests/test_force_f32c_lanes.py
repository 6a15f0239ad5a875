"""The FP32-form force with 32, 8 and 4 lanes per node against the persistent
kernel (two nodes per thread), bit for bit: lattices and jittered nodes, one
and two materials, a critical stretch, slits and ragged families, strains in
and beyond the series range."""
import numpy as np
import pytest

import pdmtel_b200 as P

pytestmark = pytest.mark.gpu

H = 1e-3
A = 1 / np.sqrt(3.0)


def context(dims, jitter=0.0, materials=1, fail=False, factors=False):
    r = np.random.default_rng(2)
    z, y, x = np.meshgrid(*[np.arange(n) - (n - 1) / 2 for n in dims[::-1]], indexing="ij")
    xyz = np.stack([x, y, z], -1).reshape(-1, 3) * H
    xyz = xyz + r.uniform(-jitter, jitter, xyz.shape) * H
    n = len(xyz)
    mats = [dict(spring=2e19 * (1 + k), density=2440.0, ecrit=4e-3 if fail else 1e20) for k in range(materials)]
    ctx = P.DeviceContext.create(xyz, np.arange(n) % materials, mats, grid_spacing=H, horizon=3.015 * H, intg_point=2,
                                 abscissae=[-A, A], weights=[1.0, 1.0],
                                 slits=[(-0.2 * dims[0] * H, 0.2 * dims[0] * H, 0.3 * H, 0.3 * H, -1.0, 1.0)],
                                 spring_factor=np.exp(0.2 * r.standard_normal(n)) if factors else None)
    ctx.bond_search()
    if factors:
        ctx.set_bdry_eff(1.0 + 0.1 * r.random(n))
    ctx.mls_setup(3.0 * H)
    ctx.set_energy(False)
    ctx.set_precision(P.PREC_FP32C)
    return ctx, xyz


@pytest.mark.parametrize("strain", [1e-4, 5e-2])
@pytest.mark.parametrize("dims,kw", [
    ((9, 7, 5), {}), ((9, 7, 5), dict(jitter=0.2)), ((11, 6, 7), dict(materials=2, fail=True)),
    ((11, 6, 7), dict(factors=True)), ((33, 23, 17), {}), ((33, 23, 17), dict(jitter=0.1, factors=True)),
    ((33, 23, 17), dict(fail=True)), ((149, 111, 8), {}), ((149, 111, 8), dict(fail=True))])
def test_lanes_equal_pairs(dims, kw, strain):
    ctx, x = context(dims, **kw)
    r = np.random.default_rng(8)
    U = strain * (x @ r.standard_normal((3, 3)) + 0.3 * H * r.standard_normal(x.shape))
    V = r.standard_normal(x.shape)
    out = []
    for step in (ctx.rk4_steps, ctx.rk4_steps_persistent):
        ctx.reset_state()
        ctx.set_state(U, V)
        ctx.gather(0.0)
        step(1e-9, 0.0, 2)
        ctx.sync()
        out.append(ctx.get_state())
    assert np.all(np.isfinite(out[0][0]))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    if kw in ({}, dict(factors=True)):  # the same from chunk-major blocks
        ctx.set_option(P.OPT_FORCE_STENCIL, 3)
        ctx.reset_state()
        ctx.set_state(U, V)
        ctx.gather(0.0)
        ctx.rk4_steps(1e-9, 0.0, 2)
        ctx.sync()
        U3, V3 = ctx.get_state()
        assert np.array_equal(out[0][0], U3) and np.array_equal(out[0][1], V3)
    ctx.close()
