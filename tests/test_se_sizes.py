"""The statistical equilibrium at the edges of its solvers, against the oracle
(GPU).

Systems of up to 32 unknowns are one warp's (16, 24 or 32 columns in its
registers), up to 96 a team of four warps' (12, 20 or 24 columns a warp);
larger ones are factorised.  One warp and a team perform the same operations
per element, so the forced choice gives equal bits at every size, and so does
the batched kernel.  Tolerance: that of test_gpu_parity.py's solve, 1e-10 of
the node's largest population."""
import dataclasses

import numpy as np
import pytest

from portal_gb300 import synth
from test_gpu_parity import _against_oracle_se, _small

pytestmark = pytest.mark.gpu


def _problem(levels, kmax, points=300):
    cloud, _, rc = _small(points, nlev=3, t_law="loglinear")
    # more than 20 levels of a heavier rotor: the lines stay below 1.2 THz
    mol = synth.linear_rotor(levels) if levels <= 20 else synth.linear_rotor(levels, b_rot_hz=15e9)
    frac = synth.lte_fractions(mol, np.maximum(cloud.t_kin, 1.0))
    cloud = dataclasses.replace(cloud, lev_p=np.ascontiguousarray(frac * (cloud.ab_all * cloud.h2_dens)[:, None]))
    rc.kmax = kmax
    nu = np.asarray(mol.nu)
    J0 = 1.4744995e-50 * nu ** 3 / np.expm1(4.79924e-11 * nu / np.maximum(cloud.t_kin, 1.0)[:, None])
    J2 = 1e-3 * J0 * np.cos(np.arange(cloud.node_num))[:, None]
    return cloud, mol, rc, J0, J2


# unknowns: 3, 15, 17, 24, 25, 31, 33, 48, 49, 78, 82, 96, 99
@pytest.mark.parametrize("levels,kmax", [(2, 2), (8, 2), (9, 2), (9, 4), (13, 2), (16, 2), (17, 2), (17, 4), (25, 2),
                                         (21, 6), (22, 6), (33, 4), (34, 4)])
def test_se_sizes(built_lib, monkeypatch, levels, kmax):
    import portal_gb300 as pg
    cloud, mol, rc, J0, J2 = _problem(levels, kmax)
    with pg.Context(0) as ctx:
        ctx.set_molecule(mol)
        ctx.set_cloud(cloud)
        p, s = ctx.solve_se(kmax, J0, J2)
        for team in ("1", "4"):
            monkeypatch.setenv("PORTAL_SE_TEAM", team)
            q, t = ctx.solve_se(kmax, J0, J2)
            assert np.array_equal(p, q) and np.array_equal(s, t)
    assert not (s & pg.NODE_SINGULAR).any()
    assert not p[cloud.bulk_node_num:].any()
    _against_oracle_se(p, cloud, mol, rc, J0, J2, nodes=8)


@pytest.mark.parametrize("levels,kmax", [((5, 17), 4), ((6, 14, 24), 6)])
def test_se_batch_sizes(built_lib, levels, kmax):
    """Batches whose largest system takes a team of four, each with a small
    system among them."""
    import portal_gb300 as pg
    ctxs, want = [], []
    for k, lev in enumerate(levels):
        cloud, mol, rc, _, _ = _problem(lev, kmax, points=250 + 40 * k)
        c = pg.Context(0)
        c.set_molecule(mol)
        c.set_cloud(cloud)
        c.radiation_field(rc)
        want.append(c.solve_se(kmax))
        ctxs.append(c)
    with pg.Batch(0) as b:
        for c in ctxs:
            b.add(c)
        b.prepare(rc, autotune=False)
        b.run()
        for c, (pp, _) in zip(ctxs, want):
            np.testing.assert_array_equal(c.results()[2], pp)
    for c in ctxs:
        c.close()
