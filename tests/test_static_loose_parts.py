"""Boxes that several cuts leave with parts held by few bonds, or by none: hard
systems of up to a few thousand iterations.  Both precisions converge on the
lattice stencil as FP64 does on the family lists, to the same displacements."""
import numpy as np
import pytest

import pdmtel_b200 as P

pytestmark = pytest.mark.gpu

H = 1e-3


def context(seed):
    r = np.random.default_rng(seed)
    dims = r.integers(4, 15, 3)
    z, y, x = np.meshgrid(*[np.arange(n) * H for n in dims[::-1]], indexing="ij")
    X = np.stack([x, y, z], -1).reshape(-1, 3) - r.choice([0, 1]) * np.array(dims) * H / 2
    at, n = np.rint((X - X.min(0)) / H).astype(int), len(X)
    slits = []
    for _ in range(int(r.integers(1, 6))):
        axis = int(r.integers(0, 2)) if r.random() < 0.8 else 2
        lo, hi = X.min(0), X.max(0)
        s = [[-1.0, 1.0] if r.random() < 0.5 else [lo[k] + (hi[k] - lo[k]) * v for v in sorted(r.uniform(-0.2, 1.2, 2))]
             for k in range(3)]
        layer = int(r.choice([0, dims[axis] - 2, r.integers(0, dims[axis] - 1)]))
        s[axis] = [lo[axis] + H * (layer + 0.5)] * 2
        slits.append(tuple(np.ravel(s)))
    inner = np.all((at[:, :2] > 1) & (at[:, :2] < dims[:2] - 2), 1)
    bc = np.where(at[:, 2] == 0, 0, np.where((at[:, 2] == dims[2] - 1) & inner, 1, -1)).astype(np.int32)
    factor = np.exp(0.2 * r.standard_normal(n)) if r.random() < 0.4 else None
    ctx = P.DeviceContext.create(
        X, np.zeros(n, np.int32), [dict(spring=2e19, density=2440.0, ecrit=1e20)],
        [dict(type=P.BC_DISPL, dir=(1, 1, 1), value=(0.0, 0.0, 0.0)),
         dict(type=P.BC_TRACTION, dir=(1, 1, 1), value=(1e6, 5e5, -3e5))], bc, H,
        float(r.choice([2.015, 3.015, 3.015, 4.1])) * H, integration=P.INTG_CCI, slits=slits, spring_factor=factor)
    ctx.bond_search()
    return ctx


@pytest.mark.parametrize("seed", [45, 121, 185, 218, 233, 365, 368, 487, 544, 585])
def test_solves_converge(seed):
    ctx = context(seed)
    ctx.set_option(P.OPT_STATIC_STENCIL, 0)
    want, _, _ = ctx.static_solve(1.0, P.PREC_FP64, 1e-10, maxit=3000)
    ctx.set_option(P.OPT_STATIC_STENCIL, 1)
    assert ctx.static_prepare()
    for prec in (P.PREC_FP64, P.PREC_FP32C):
        u, _, rel = ctx.static_solve(1.0, prec, 1e-10, maxit=3000)
        assert rel <= 1e-10
        assert np.linalg.norm(u - want) <= 1e-7 * np.linalg.norm(want)
    ctx.close()
