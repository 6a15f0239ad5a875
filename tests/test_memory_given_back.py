"""Buffers that a context keeps for its next static solve or reverse sweep are
given back when another call finds no room, and made again when they are
needed: with the rest of the device's memory taken, calls succeed that fit
beside the problem but not beside those buffers.  A static preparation that
fails keeps none of its scratch memory."""
import numpy as np
import pytest

import pdmtel_b200 as P

pytestmark = pytest.mark.gpu

H, A = 1e-3, 1 / np.sqrt(3.0)
MB = 1 << 20


class Taken:
    """All of the device's free memory but about `leave` bytes."""

    def __init__(self, leave):
        import torch

        self.torch, self.held = torch, []
        torch.cuda.empty_cache()
        for step in (256 * MB, 32 * MB, 2 * MB):
            while True:
                free = torch.cuda.mem_get_info()[0]
                if free < leave + step:
                    break
                take = max(step, (free - leave) // step * step)
                self.held.append(torch.empty(take, dtype=torch.uint8, device="cuda"))

    def __enter__(self):
        assert self.torch.cuda.mem_get_info()[0] < 40 * MB
        return self

    def __exit__(self, *a):
        self.held.clear()
        self.torch.cuda.empty_cache()


def context(dims, **kw):
    z, y, x = np.meshgrid(*[np.arange(n) * H for n in dims[::-1]], indexing="ij")
    xyz = np.stack([x, y, z], -1).reshape(-1, 3)
    bc = np.where(xyz[:, 2] == 0, 0, np.where(xyz[:, 2] > (dims[2] - 1.5) * H, 1, -1)).astype(np.int32)
    ctx = P.DeviceContext.create(
        xyz, np.zeros(len(xyz), np.int32), [dict(spring=2e19, density=2440.0, ecrit=1e20)],
        [dict(type=P.BC_DISPL, dir=(1, 1, 1), value=(0.0, 0.0, 0.0)),
         dict(type=P.BC_TRACTION, dir=(1, 0, 0), value=(1e6, 0.0, 0.0))], bc, grid_spacing=H, horizon=3.015 * H,
        intg_point=2, abscissae=[-A, A], weights=[1.0, 1.0], **kw)
    halves, _, _ = ctx.bond_search()
    return ctx, halves


def test_after_a_reverse_sweep():
    ctx, halves = context((29, 29, 24), spring_factor=np.ones(29 * 29 * 24))
    ctx.mls_setup(3.0 * H)
    r = np.random.default_rng(1)
    lam = r.standard_normal(3 * ctx.n)

    def sweep():
        ctx.reset_state()
        ctx.set_state(1e-7 * np.cos(np.arange(3.0 * ctx.n)), None)
        ctx.gather(0.0)
        ctx.adjoint_forward(1e-8, 0.0, 1, 1)
        return ctx.adjoint_backward(lam)

    first = sweep()
    family = ctx.get_family(halves)
    # a search makes about 36 MB of lists beside the present ones; the sweep
    # keeps 160 MB of mirror entries and shares
    with Taken(16 * MB):
        assert ctx.bond_search()[0] == halves
        again = ctx.get_family(halves)
    assert all(np.array_equal(a, b) for a, b in zip(family, again))
    assert np.array_equal(sweep(), first)
    ctx.close()


@pytest.mark.parametrize("stencil", [1, 0])
def test_after_a_static_solve(stencil):
    ctx, _ = context((64, 64, 64))
    ctx.set_option(P.OPT_STATIC_STENCIL, stencil)
    first = ctx.static_solve(1.0, P.PREC_FP64, 1e-2)
    ug = 1e-6 * np.random.default_rng(2).standard_normal(24 * ctx.n)
    # 50 MB of staging; the solve keeps 38 MB of vectors and more
    with Taken(16 * MB):
        ctx.set_gauss_displ(ug)
    assert np.array_equal(ctx.get_gauss_displ(), ug)
    again = ctx.static_solve(1.0, P.PREC_FP64, 1e-2)
    assert np.array_equal(first[0], again[0]) and first[1:] == again[1:]
    b = ctx.static_rhs(1.0)
    assert np.any(b) and np.array_equal(b, ctx.static_rhs(1.0))
    ctx.close()


def test_an_error_is_reported_once():
    ctx, halves = context((64, 64, 64))
    other, few = context((9, 8, 7))
    with Taken(16 * MB), pytest.raises(P.PdError):
        ctx.set_gauss_displ(np.zeros(24 * ctx.n))
    assert other.bond_search()[0] == few
    other.mls_setup(3.0 * H)
    other.rk4_step(1e-9, 1e-9)
    ctx.close()
    other.close()


def test_a_failed_preparation_leaves_no_scratch():
    import torch

    used = []
    for failures in (0, 4):
        before = torch.cuda.mem_get_info()[0]
        ctx, _ = context((64, 64, 64))
        for _ in range(failures):
            # the 8 MB offset table fits, the operator's 19 MB do not
            with Taken(16 * MB), pytest.raises(P.PdError):
                ctx.static_prepare()
            ctx.set_option(P.OPT_STATIC_STENCIL, 1)
        assert ctx.static_prepare()
        used.append(before - torch.cuda.mem_get_info()[0])
        ctx.close()
    assert used[1] - used[0] < 8 * MB
