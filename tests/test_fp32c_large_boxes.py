"""The gather's coefficient ring and the stencil force, which problems of 65,536
nodes and more run, against the lists and the lane kernel, bit for bit: a box
with odd rows, a slit and a ragged last slice, every block shape, boundary and
spring factors, strains beyond the series range, a critical stretch, several
boxes in one context, a changed work order and new MLS data."""
import numpy as np
import pytest

import pdmtel_b200 as P
from test_force_f32c_lanes import A, H, context

pytestmark = pytest.mark.gpu

DIMS = (149, 111, 4)  # 66,156 nodes


def steps(ctx, x, strain, n=2):
    r = np.random.default_rng(8)
    U = strain * (x @ r.standard_normal((3, 3)) + 0.3 * H * r.standard_normal(x.shape))
    ctx.reset_state()
    ctx.set_state(U, r.standard_normal(x.shape))
    ctx.gather(0.0)
    ctx.rk4_steps(1e-9, 0.0, n)
    ctx.sync()
    out = ctx.get_state()
    assert np.all(np.isfinite(out[0])) and np.any(out[0] != U.ravel())
    return out


def same(a, b):
    return np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


def test_ring_gather_equals_lists():
    ctx, x = context(DIMS)
    assert ctx.n >= 65536 and ctx.n % 16
    want = steps(ctx, x, 1e-4)
    ctx.set_option(P.OPT_GATHER_SELL, 1)
    ctx.set_option(P.OPT_GATHER_STENCIL, 1)
    assert same(steps(ctx, x, 1e-4), want)
    ctx.set_option(P.OPT_TILE, 2 | 1 << 8 | 1 << 16)
    assert same(steps(ctx, x, 1e-4), want)
    cp, ci, co = ctx.get_mls()
    co *= 1.0 + 1e-3 * np.random.default_rng(2).random(co.size)
    ctx.set_mls(cp, ci, co)
    assert ctx.get_option(P.OPT_GATHER_STENCIL) == 1
    ring = steps(ctx, x, 1e-4)
    assert not same(ring, want)
    ctx.set_option(P.OPT_GATHER_SELL, 0)
    assert same(steps(ctx, x, 1e-4), ring)
    ctx.close()


@pytest.mark.parametrize("strain", [1e-4, 5e-2])
@pytest.mark.parametrize("bdry,sfac", [(False, False), (True, False), (False, True), (True, True)])
def test_stencil_force_equals_lanes(bdry, sfac, strain):
    ctx, x = context(DIMS)
    r = np.random.default_rng(6)
    if bdry:
        ctx.set_bdry_eff(1.0 + 0.1 * r.random(ctx.n))
    if sfac:
        ctx.set_spring_factor(np.exp(0.2 * r.standard_normal(ctx.n)))
    want = steps(ctx, x, strain)
    for shape in (1, 2, 3, 4):
        ctx.set_option(P.OPT_FORCE_STENCIL, shape)
        assert same(steps(ctx, x, strain), want), shape
    ctx.close()


@pytest.mark.parametrize("factors", [False, True])
def test_stencil_force_with_critical_stretch(factors):
    """The lane kernel's general variant forms the bond vectors from split
    coordinates, the stencil from lattice offsets: equal to FP32 rounding, and
    the block shapes to each other bit for bit."""
    ctx, x = context(DIMS, fail=True, factors=factors)
    want = steps(ctx, x, 2e-3)
    first = None
    for shape in (1, 2, 3, 4):
        ctx.set_option(P.OPT_FORCE_STENCIL, shape)
        got = steps(ctx, x, 2e-3)
        first = first or got
        assert same(got, first), shape
        assert np.linalg.norm(got[0] - want[0]) <= 1e-6 * np.linalg.norm(want[0])
    ctx.close()


def test_stencil_force_and_ring_on_several_boxes():
    offsets, xyz, local, at = [0], [], [], 0
    for dims in ((97, 60, 5), (41, 33, 21), (63, 64, 3), (9, 7, 3), (16, 32, 8)):  # tiles, runs of pairs
        z, y, x = np.meshgrid(*[np.arange(n) for n in dims[::-1]], indexing="ij")
        box = np.stack([x, y, z], -1).reshape(-1, 3) * H
        local.append(box - box.mean(0))
        xyz.append(box + np.array([at * H, 0, 0]))
        offsets.append(offsets[-1] + len(box))
        at += dims[0] + 6
    xyz, local = np.concatenate(xyz), np.concatenate(local)
    n = len(xyz)
    assert n >= 65536
    r = np.random.default_rng(4)
    ctx = P.DeviceContext.create(xyz, np.zeros(n, np.int32), [dict(spring=2e19, density=2440.0, ecrit=1e20)],
                                 grid_spacing=H, horizon=3.015 * H, intg_point=2, abscissae=[-A, A],
                                 weights=[1.0, 1.0], spring_factor=np.exp(0.2 * r.standard_normal(n)))
    ctx.bond_search()
    ctx.mls_setup(3.0 * H, local)
    ctx.set_energy(False)
    ctx.set_precision(P.PREC_FP32C)
    ctx.set_boxes(offsets)
    want = steps(ctx, local, 1e-4)
    ctx.set_option(P.OPT_GATHER_SELL, 1)
    ctx.set_option(P.OPT_GATHER_STENCIL, 1)
    for shape in (1, 2, 3, 4):
        ctx.set_option(P.OPT_FORCE_STENCIL, shape)
        assert same(steps(ctx, local, 1e-4), want), shape
    ctx.close()


def test_sell_copy_holds_the_coefficients_and_nothing_else():
    import torch

    def made(ctx):
        before = torch.cuda.mem_get_info()[0]
        ctx.set_option(P.OPT_GATHER_SELL, 1)
        return before - torch.cuda.mem_get_info()[0]

    ctx, _ = context(DIMS)
    width = np.diff(ctx.get_mls()[0])
    at = np.stack(np.unravel_index(np.arange(ctx.n), DIMS[::-1]), -1)[:, ::-1]  # x, y, z
    shift = np.array([3, 2, 2])
    tile, inner = at >> shift, at & ((1 << shift) - 1)
    order = np.lexsort((inner[:, 0], inner[:, 1], inner[:, 2], tile[:, 0], tile[:, 1], tile[:, 2]))
    slices = np.concatenate([width[order], np.zeros(-ctx.n % 16, width.dtype)]).reshape(-1, 16).max(1)
    assert made(ctx) <= slices.sum() * 16 * 8 * 4 + (8 << 20)
    ctx.close()
    ctx, _ = context((40, 30, 20))  # no gather reads it below 65,536 nodes
    assert made(ctx) <= 2 << 20 and ctx.get_option(P.OPT_GATHER_SELL) == 1
    ctx.close()
