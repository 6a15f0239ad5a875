"""The static operator on cracked boxes: the lattice stencil less its broken
bonds against the family lists (a warp per node below 12,288 nodes, eight
lanes above), with and without spring factors, in every operator form."""
import numpy as np
import pytest

import pdmtel_b200 as P
from pdmtel_b200 import decks as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("factors", [False, True])
@pytest.mark.parametrize("dims", [(17, 10, 5), (33, 24, 17)])
def test_cracked_stencil_equals_family_lists(tmp_path, dims, factors):
    d = D.config_plate(dims=dims, spacing=1e-3, slit_half_length=0.2e-3 * dims[0])
    d.bcs = D.config_bar(dims=dims, spacing=1e-3).bcs
    d.bc_spaces = D.config_bar(dims=dims, spacing=1e-3).bc_spaces
    d.write(str(tmp_path))
    dm = P.pdDataManager(str(tmp_path))
    P.pdSolve.InitialProblem(dm)
    ctx = dm.context()
    assert dm.info().num_broken > 0
    r = np.random.default_rng(3)
    if factors:
        ctx.set_spring_factor(np.exp(0.2 * r.standard_normal(ctx.n)))
    x = r.standard_normal(3 * ctx.n) * 1e-7
    ctx.set_option(P.OPT_STATIC_STENCIL, 0)
    assert not ctx.static_prepare()
    want = ctx.static_matvec(1.0, x)
    u0, it0, _ = ctx.static_solve(1.0, P.PREC_FP64, 1e-10)
    ctx.set_option(P.OPT_STATIC_STENCIL, 1)
    assert ctx.static_prepare()
    for split in (4, 2, 8, 0):
        ctx.set_option(P.OPT_STATIC_SPLIT, split)
        assert np.linalg.norm(ctx.static_matvec(1.0, x) - want) <= 1e-13 * np.linalg.norm(want), split
    ctx.set_option(P.OPT_STATIC_SPLIT, 4)
    for prec in (P.PREC_FP64, P.PREC_FP32C):
        u, it, rel = ctx.static_solve(1.0, prec, 1e-10)
        assert rel <= 1e-10 and it <= 1.2 * it0 + 10
        assert np.linalg.norm(u - u0) <= 1e-8 * np.linalg.norm(u0)
    dm.close()
