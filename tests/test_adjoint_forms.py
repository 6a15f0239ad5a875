"""The reverse sweep that evaluates every force point once (a warp per node
below 12,288 nodes, eight lanes above) against the one that evaluates it from
both ends, which a family without some mirror entries takes: two nodes far from
the specimen carry a bond listed at one end only, which changes nothing on the
specimen.  Boundary factors, two materials with a critical stretch, lengths
outside the range of the branch-free roots, a bond listed twice."""
import numpy as np
import pytest

import pdmtel_b200 as P

pytestmark = pytest.mark.gpu

A = 1 / np.sqrt(3.0)


def specimen(dims, h, materials, factors):
    """The specimen's context arguments, family and MLS data, and its nodes
    followed by the two far ones."""
    r = np.random.default_rng(2)
    z, y, x = np.meshgrid(*[np.arange(n) - (n - 1) / 2 for n in dims[::-1]], indexing="ij")
    xyz = np.stack([x, y, z], -1).reshape(-1, 3) * h
    n = len(xyz)
    tiny = h < 1e-50
    kw = dict(grid_spacing=h, horizon=3.015 * h, intg_point=2, abscissae=[-A, A], weights=[1.0, 1.0],
              materials=[dict(spring=(1e200 if tiny else 2e19) * (1 + k), density=1e60 if tiny else 2440.0,
                              ecrit=2e-4 if materials > 1 else 1e20) for k in range(materials)])
    one = P.DeviceContext.create(xyz, np.arange(n) % materials, **kw)
    halves, _, _ = one.bond_search()
    rp, col, _ = one.get_family(halves)
    one.mls_setup(3.0 * h)
    cp, ci, co = one.get_mls()
    one.close()
    far = xyz.max(0) + 40 * h
    xyz = np.concatenate([xyz, [far, far + [h, 0, 0]]])
    cp = np.concatenate([cp, cp[-1] + [1, 2]])
    ci = np.concatenate([ci, [n, n + 1]]).astype(np.int32)
    co = np.concatenate([co, np.ones(16)])
    return dict(kw, xyz=xyz, mat=np.arange(n + 2) % materials, factor=np.exp(0.2 * r.standard_normal(n + 2)),
                bdry=1.0 + 0.1 * r.random(n + 2) if factors else None, rp=rp, col=col, mls=(cp, ci, co))


def gradient(s, mirrored, precision, h, dt):
    kw = {k: s[k] for k in ("grid_spacing", "horizon", "intg_point", "abscissae", "weights")}
    n = len(s["xyz"]) - 2
    ctx = P.DeviceContext.create(s["xyz"], s["mat"], s["materials"], spring_factor=s["factor"], **kw)
    more = [n + 1, n] if mirrored else [n + 1]
    ctx.set_family(np.concatenate([s["rp"], s["rp"][-1] + [1, len(more)]]), np.concatenate([s["col"], more]))
    if s["bdry"] is not None:
        ctx.set_bdry_eff(s["bdry"])
    ctx.set_mls(*s["mls"])
    ctx.set_precision(precision)
    r = np.random.default_rng(5)
    x = s["xyz"]
    U = 1e-4 * (x @ r.standard_normal((3, 3)) + 0.1 * h * r.standard_normal(x.shape))
    ctx.set_state(U, 1e-4 * h / dt * r.standard_normal(x.shape))
    ctx.gather(0.0)
    ctx.adjoint_forward(dt, 0.0, 2, 1)
    out = ctx.get_state()
    g = ctx.adjoint_backward(r.standard_normal(x.shape), r.standard_normal(x.shape) * dt)
    ctx.close()
    assert np.all(np.isfinite(g)) and np.any(g[:n])
    return out[0][:3 * n], out[1][:3 * n], g[:n]


def twice(rp, col, i, k):
    """Entry k of node i's row, and its mirror, listed once more."""
    j = col[rp[i] + k]
    for a, b in ((i, j), (j, i)):
        at = rp[a] + np.searchsorted(col[rp[a]:rp[a + 1]], b)
        col = np.insert(col, at, b)
        rp = rp + (np.arange(len(rp)) > a)
    return rp, col


@pytest.mark.parametrize("kw", [{}, dict(factors=True), dict(materials=2), dict(precision=P.PREC_FP64A),
                                dict(precision=P.PREC_FP32C), dict(tiny=True), dict(twice=True)],
                         ids=lambda kw: "-".join(kw) or "plain")
@pytest.mark.parametrize("dims", [(9, 7, 5), (29, 23, 19)])  # 317 and 12,675 nodes
def test_one_evaluation_equals_two(dims, kw):
    h = 1e-70 if kw.get("tiny") else 1e-3
    s = specimen(dims, h, kw.get("materials", 1), kw.get("factors", False))
    if kw.get("twice"):
        s["rp"], s["col"] = twice(s["rp"], s["col"], 100, 3)
    dt = 1.0 if kw.get("tiny") else 5e-8
    prec = kw.get("precision", P.PREC_FP64)
    want, got = (gradient(s, mirrored, prec, h, dt) for mirrored in (False, True))
    assert np.array_equal(want[0], got[0]) and np.array_equal(want[1], got[1])
    assert np.linalg.norm(got[2] - want[2]) <= 1e-12 * np.linalg.norm(want[2])
