"""Steps whose force kernels take the stage's epilogue along (as launches and
as a graph) against the same stages with their epilogues apart, bit for bit:
both point schemes, both precisions, each kind of condition."""
import numpy as np
import pytest

import pdmtel_b200 as P

pytestmark = pytest.mark.gpu

H = 1e-3
A = 1 / np.sqrt(3.0)


def context(dims, points, precision, energy):
    z, y, x = np.meshgrid(*[np.arange(n) - (n - 1) / 2 for n in dims[::-1]], indexing="ij")
    xyz = np.stack([x, y, z], -1).reshape(-1, 3) * H
    n = len(xyz)
    bc = np.full(n, -1, dtype=np.int32)
    bc[: 5 * 7] = np.arange(5 * 7) % 5 - 1
    bcs = [dict(type=P.BC_DISPL, dir=(1, 0, 1), value=(1e-6, 2e-6, -1e-6), load_type=1.0, end_time=2.5e-9),
           dict(type=P.BC_VELOC, dir=(1, 1, 0), value=(0.2, -0.1, 0.3), end_time=1.5e-9),
           dict(type=P.BC_TRACTION, dir=(0, 1, 1), value=(1e5, 2e5, 3e5), load_type=1.0, end_time=1.0),
           dict(type=P.BC_DISPLGRAD, dir=(1, 0, 1), value=tuple(1e-4 * (k - 4) for k in range(9)), load_type=1.0,
                end_time=1.0)]
    gauss = (dict(integration=P.INTG_FGI, intg_point=points, abscissae=[-A, A], weights=[1.0, 1.0]) if points
             else dict(integration=P.INTG_CCI))
    ctx = P.DeviceContext.create(xyz, np.zeros(n, dtype=int), [dict(spring=2e19, density=2440.0, ecrit=1e20)],
                                 grid_spacing=H, horizon=3.015 * H, bcs=bcs, bc_id=bc, damping=1e6, **gauss)
    ctx.bond_search()
    if points:
        ctx.mls_setup(3.0 * H)
    ctx.set_energy(energy)
    ctx.set_precision(precision)
    return ctx, xyz


@pytest.mark.parametrize("energy", [False, True])
@pytest.mark.parametrize("points,precision", [(0, P.PREC_FP64), (2, P.PREC_FP64), (2, P.PREC_FP32C)])
@pytest.mark.parametrize("dims", [(7, 5, 3), (29, 23, 21)])
def test_fused_stages_equal_stages_apart(dims, points, precision, energy):
    ctx, x = context(dims, points, precision, energy)
    r = np.random.default_rng(4)
    U = 1e-4 * (x @ r.standard_normal((3, 3)) + 0.3 * H * r.standard_normal(x.shape))
    V = r.standard_normal(x.shape)
    dt = 1e-9
    out = []
    for way in ("apart", "steps", "together"):
        ctx.reset_state()
        ctx.set_state(U, V)
        if points:
            ctx.gather(0.0)
        if way == "together":
            ctx.rk4_steps(dt, 0.0, 3)
        t = 0.0
        for _ in range(3 if way != "together" else 0):
            t += dt
            kinetic = ctx.profile_step(dt, t) if way == "apart" else ctx.rk4_step(dt, t)[0]
        ctx.sync()
        out.append(ctx.get_state() + (ctx.get_vbuf(), ctx.get_energy_density()))
        if way == "steps" and energy:
            want = 0.5 * 2440.0 * H ** 3 * np.sum(out[-1][1] ** 2)
            np.testing.assert_allclose(kinetic, want, rtol=1e-11)
    assert np.all(np.isfinite(out[0][0])) and np.any(out[0][1] != V.ravel())
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b)
    ctx.close()
