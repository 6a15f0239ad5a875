"""pd_rk4_step call by call: on a stream that takes no capture, and with step
sizes that change every few calls, which a graph per change would slow down."""
import time

import numpy as np
import pytest

import pdmtel_b200 as P

pytestmark = pytest.mark.gpu

H = 1e-3
LEGACY = 1  # the handle of the legacy default stream


def context(dims=(6, 5, 4), stream=None):
    z, y, x = np.meshgrid(*[np.arange(n) * H for n in dims[::-1]], indexing="ij")
    xyz = np.stack([x, y, z], -1).reshape(-1, 3)
    ctx = P.DeviceContext.create(xyz, np.zeros(len(xyz), np.int32), [dict(spring=2e19, density=2440.0, ecrit=1e20)],
                                 grid_spacing=H, horizon=3.015 * H, integration=P.INTG_CCI, stream=stream)
    ctx.bond_search()
    ctx.set_state(1e-6 * np.random.default_rng(1).standard_normal(3 * ctx.n), np.zeros(3 * ctx.n))
    return ctx


def test_legacy_default_stream():
    out = []
    for stream in (None, LEGACY):
        ctx = context(stream=stream)
        energies = [ctx.rk4_step(1e-9, 1e-9 * (k + 1)) for k in range(5)]
        out.append((energies, ctx.get_state()))
        ctx.close()
    (ea, a), (eb, b) = out
    assert ea == eb and np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("run", [2, 3])
def test_changing_step_sizes_cost_no_more_than_launches(run):
    """Steps whose size changes with every call never make a graph; sizes that
    change every few calls may not cost more than those (a third is for noise of
    the host; a capture per change doubles two-call runs and adds more than half
    to three-call ones).  The best of five runs each, without their slowest
    tenth."""
    def mean(sizes):
        ctx = context()
        took, t = [], 0.0
        for k in range(400):
            dt = sizes[k % len(sizes)]
            t += dt
            start = time.perf_counter()
            ctx.rk4_step(dt, t)
            took.append(time.perf_counter() - start)
        ctx.close()
        return np.mean(np.sort(took[40:])[:-36])

    launches, changing = [], []
    for _ in range(5):
        launches.append(mean([1e-9, 2e-9]))
        changing.append(mean([1e-9] * run + [2e-9] * run))
    assert min(changing) <= 1.33 * min(launches)


def test_changing_step_sizes_change_no_result():
    sizes = [1e-9] * 3 + [2e-9] * 2 + [1e-9, 3e-9] * 2 + [3e-9] * 20 + [1e-9] * 9
    out = []
    for way in ("calls", "apart"):
        ctx = context()
        t = 0.0
        for dt in sizes:
            t += dt
            ctx.rk4_step(dt, t) if way == "calls" else ctx.rk4_steps(dt, t - dt, 1)
        ctx.sync()
        out.append(ctx.get_state())
        ctx.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
