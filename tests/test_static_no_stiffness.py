"""Cracked boxes in which nodes have lost their stiffness, in all directions (a
corner node and an inner node that slits cut off) or in one (the layer beyond
a slit across the section): the rows without stiffness are exact zeros, the
solves converge, and both are those of the family lists."""
import numpy as np
import pytest

import pdmtel_b200 as P

pytestmark = pytest.mark.gpu

H = 1e-3


def cut(node, sides):
    """Patches half a spacing from a lattice node that cross all its bonds: a
    bond leaves through the side of its longest component."""
    out = []
    for axis in range(3):
        for side in sides:
            box = [[v - 0.51 * H, v + 0.51 * H] for v in node]
            box[axis] = [node[axis] + 0.5 * side * H] * 2
            out.append(tuple(np.ravel(box)))
    return out


def context(dims, where, factors):
    z, y, x = np.meshgrid(*[np.arange(n) * H for n in dims[::-1]], indexing="ij")
    xyz = np.stack([x, y, z], -1).reshape(-1, 3)
    at = np.rint(xyz / H).astype(int)
    far = np.array(dims) - 1
    if where == "layer":
        slits, lost = [((far[0] - 0.5) * H,) * 2 + (-1.0, 1.0, -1.0, 1.0)], at[:, 0] == far[0]
    else:
        node = far if where == "corner" else np.array(dims) // 2
        slits, lost = cut(node * H, (-1,) if where == "corner" else (-1, 1)), np.all(at == node, 1)
    bc = np.where(at[:, 2] == 0, 0, np.where((at[:, 2] == far[2]) & (at[:, 0] < far[0] - 1), 1, -1))
    ctx = P.DeviceContext.create(
        xyz, np.zeros(len(xyz), np.int32), [dict(spring=2e19, density=2440.0, ecrit=1e20)],
        [dict(type=P.BC_DISPL, dir=(1, 1, 1), value=(0.0, 0.0, 0.0)),
         dict(type=P.BC_TRACTION, dir=(1, 1, 0), value=(1e6, 5e5, 0.0))], bc.astype(np.int32), grid_spacing=H,
        horizon=3.015 * H, integration=P.INTG_CCI, slits=slits)
    halves, _, _ = ctx.bond_search()
    rp, _, br = ctx.get_family(halves)
    if where != "layer":
        assert all(br[rp[i]:rp[i + 1]].all() for i in np.nonzero(lost)[0])
    if factors:
        ctx.set_spring_factor(np.exp(0.2 * np.random.default_rng(1).standard_normal(ctx.n)))
    zero = np.zeros((ctx.n, 3), bool)
    zero[lost & (bc != 0)] = (True, False, False) if where == "layer" else (True, True, True)
    return ctx, zero.ravel()


@pytest.mark.parametrize("factors", [False, True])
@pytest.mark.parametrize("where", ["corner", "inner", "layer"])
@pytest.mark.parametrize("dims", [(8, 8, 8), (13, 7, 11)])
def test_rows_without_stiffness(dims, where, factors):
    ctx, zero = context(dims, where, factors)
    x = np.random.default_rng(5).standard_normal(3 * ctx.n) * 1e-7
    ctx.set_option(P.OPT_STATIC_STENCIL, 0)
    assert not ctx.static_prepare()
    want = ctx.static_matvec(1.0, x)
    assert zero.any() and not want[zero].any()
    u0, it0, _ = ctx.static_solve(1.0, P.PREC_FP64, 1e-10)
    ctx.set_option(P.OPT_STATIC_STENCIL, 1)
    assert ctx.static_prepare()
    for split in (4, 2, 8, 0):
        ctx.set_option(P.OPT_STATIC_SPLIT, split)
        y = ctx.static_matvec(1.0, x)
        assert not y[zero].any(), split
        assert np.linalg.norm(y - want) <= 1e-13 * np.linalg.norm(want), split
    ctx.set_option(P.OPT_STATIC_SPLIT, 4)
    for prec in (P.PREC_FP64, P.PREC_FP32C):
        u, it, rel = ctx.static_solve(1.0, prec, 1e-10, maxit=1000)
        assert rel <= 1e-10 and it <= 1.2 * it0 + 10
        assert not u[zero].any()
        assert np.linalg.norm(u - u0) <= 1e-8 * np.linalg.norm(u0)
    ctx.close()
