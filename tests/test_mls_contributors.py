"""The device's MLS contributor lists against the rule written out: the node,
then its family in ascending order within the support, or within one and a
half supports where fewer than ten qualify (corners and edges here, whose
second list is stored over the first)."""
import numpy as np
import pytest

import pdmtel_b200 as P

pytestmark = pytest.mark.gpu

H, A = 1e-3, 1 / np.sqrt(3.0)


@pytest.mark.parametrize("rw", [1.8, 2.1, 3.0])
@pytest.mark.parametrize("dims,jitter", [((4, 4, 4), 0.0), ((9, 8, 7), 0.0), ((9, 8, 7), 0.1), ((40, 3, 3), 0.0)])
def test_contributors_follow_the_rule(dims, jitter, rw):
    z, y, x = np.meshgrid(*[np.arange(n) - (n - 1) / 2 for n in dims[::-1]], indexing="ij")
    xyz = np.stack([x, y, z], -1).reshape(-1, 3) * H
    xyz = xyz + np.random.default_rng(3).uniform(-jitter, jitter, xyz.shape) * H
    ctx = P.DeviceContext.create(xyz, np.zeros(len(xyz), np.int32), [dict(spring=2e19, density=2440.0, ecrit=1e20)],
                                 grid_spacing=H, horizon=3.015 * H, intg_point=2, abscissae=[-A, A],
                                 weights=[1.0, 1.0])
    halves, _, _ = ctx.bond_search()
    rp, col, _ = ctx.get_family(halves)
    ctx.mls_setup(rw * H)
    cp, ci, _ = ctx.get_mls()
    wide = 0
    for i in range(ctx.n):
        fam = col[rp[i]:rp[i + 1]]
        d = xyz[fam] - xyz[i]
        r = np.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2])
        near = fam[r <= rw * H]
        if len(near) + 1 < 10:
            near, wide = fam[r <= rw * H * 1.5], wide + 1
        assert np.array_equal(ci[cp[i]:cp[i + 1]], np.concatenate([[i], near])), i
    assert wide > 0 or rw > 2
    ctx.close()
