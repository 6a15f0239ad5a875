"""The MLS gather with a lane per Gauss point against the sum written out, bit
for bit: contributor lists of a few entries, of whole chunks of eight and with
remainders, node counts that leave groups of a warp without a node, nodes with
boundary conditions; and the FP32 form against its one-thread-per-point
variant."""
import numpy as np
import pytest

import pdmtel_b200 as P

pytestmark = pytest.mark.gpu

H, A = 1e-3, 1 / np.sqrt(3.0)


def context(dims, rw):
    z, y, x = np.meshgrid(*[np.arange(n) - (n - 1) / 2 for n in dims[::-1]], indexing="ij")
    xyz = np.stack([x, y, z], -1).reshape(-1, 3) * H
    bc = np.full(len(xyz), -1, np.int32)
    bc[:3], bc[-2:] = 0, 1
    ctx = P.DeviceContext.create(
        xyz, np.zeros(len(xyz), np.int32), [dict(spring=2e19, density=2440.0, ecrit=1e20)],
        [dict(type=P.BC_DISPL, dir=(1, 0, 1), value=(1e-7, 2e-7, 3e-7)),
         dict(type=P.BC_DISPLGRAD, dir=(0, 1, 1), value=tuple(1e-4 * (k + 1) for k in range(9)))], bc,
        grid_spacing=H, horizon=3.015 * H, intg_point=2, abscissae=[-A, A], weights=[1.0, 1.0])
    ctx.bond_search()
    ctx.mls_setup(rw * H)
    return ctx, xyz, bc


@pytest.mark.parametrize("dims,rw", [((4, 4, 4), 1.8), ((5, 4, 4), 2.0), ((7, 5, 6), 2.3), ((6, 6, 5), 3.0),
                                     ((9, 8, 7), 2.9)])
def test_gather_equals_the_sum(dims, rw):
    ctx, x, bc = context(dims, rw)
    n = ctx.n
    cp, ci, co = ctx.get_mls()
    assert len({int(v) % 8 for v in np.diff(cp)}) > 1
    us = np.random.default_rng(6).standard_normal((n, 3)) * 1e-6
    ctx.gather(0.0, us)
    got = ctx.get_gauss_displ().reshape(n, 8, 3)
    for i in np.nonzero(bc < 0)[0]:
        b, e = cp[i], cp[i + 1]
        c = co[8 * b:8 * e].reshape(8, -1)
        want = np.zeros((8, 3))
        for k in range(e - b):
            want += us[ci[b + k]] * c[:, k:k + 1]
        assert np.array_equal(got[i], want), i
    assert np.all(got[:3, :, 0] == 1e-7) and np.all(got[:3, :, 2] == 3e-7) and np.all(got[:3, :, 1] == 0.0)
    assert np.all(got[-2:, :, 0] == 0.0) and np.all(got[-2:, :, 1:] != 0.0)
    ctx.set_precision(P.PREC_FP32C)
    out = []
    for per_point in (0, 1):
        ctx.set_option(P.OPT_GATHER_PER_POINT, per_point)
        ctx.reset_state()
        ctx.set_state(us, us * 1e5)
        ctx.gather(0.0)
        ctx.rk4_steps(1e-9, 0.0, 2)
        ctx.sync()
        out.append(ctx.get_state())
    # supports of few nodes give moment matrices next to singular, whose steps
    # overflow in both variants alike
    for a, b in zip(*out):
        assert np.array_equal(a, b, equal_nan=True)
    if rw >= 2.9:
        assert np.all(np.isfinite(out[0][0]))
    ctx.close()
