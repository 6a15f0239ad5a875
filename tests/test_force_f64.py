"""The FP64 force with a warp and with eight lanes per node against the
oracle, bit for bit, on displacements inside and outside the range of its
branch-free square roots and quotients: at rest, small, near the smallest and
beyond the smallest normal numbers, overflowing, and with a NaN."""
import numpy as np
import pytest

import pdmtel_b200 as P
from conftest import CASES, deck_dir, load_golden
from golden_model import model_from_golden, params

pytestmark = pytest.mark.gpu


def states(n, dx):
    r = np.random.default_rng(11).standard_normal(n)
    nan = 1e-4 * dx * r
    nan[n // 2] = np.nan
    mixed = np.where(np.arange(n) % 5 == 0, 1e-4 * dx * r, 0.0)
    return {"rest": np.zeros(n), "small": 1e-4 * dx * r, "front": mixed, "tiny": 1e-230 * r, "denormal": 1e-315 * r,
            "far": 1e3 * dx * r, "overflow": 1e170 * r, "nan": nan}


@pytest.mark.parametrize("lanes", [32, 8])
@pytest.mark.parametrize("name", CASES)
def test_force_equals_oracle_in_and_out_of_range(name, lanes):
    g = load_golden(name)
    p = params(g)
    dm = P.pdDataManager(deck_dir(name))
    P.pdSolve.InitialProblem(dm)
    ctx = dm.context()
    ctx.set_option(P.OPT_F64_LANES_BELOW, 1 << 30 if lanes == 32 else 0)
    n, npt = ctx.n, ctx.npt
    assert n < 12288
    us = states(3 * n, p["dx"])
    ug = states(3 * n * npt, p["dx"])
    for state in us:
        m = model_from_golden(g, ug=ug[state])
        ctx.reset_state()
        ctx.init_dynamic()
        ctx.set_gauss_displ(ug[state])
        with np.errstate(all="ignore"):
            want = m.force_stage(1e-9, 1e-9, us[state])
        got = ctx.force_stage(1e-9, 1e-9, us[state])
        assert np.array_equal(got, want, equal_nan=True), state
        assert np.array_equal(ctx.get_vbuf(), m.vbuf, equal_nan=True), state
        np.testing.assert_allclose(ctx.get_energy_density(), m.eed, rtol=1e-12)
    dm.close()
