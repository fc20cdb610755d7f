"""The extra_info rates around the sizes of a team (GPU): three kinds of n sums
over its threads, one warp's or a team of four's, from the inverse and from the
factorisation.  Tolerance: that of the rates in test_gpu_parity.py."""
import numpy as np
import pytest

from test_se_sizes import _problem

pytestmark = pytest.mark.gpu


# unknowns: 3, 31, 33, 42, 43 (126 and 129 sums for 128 threads), 96, 99 (factorised)
@pytest.mark.parametrize("levels,kmax", [(2, 2), (16, 2), (17, 2), (12, 6), (22, 2), (33, 4), (34, 4)])
def test_rates_at_their_edges(built_lib, monkeypatch, levels, kmax):
    import oracle
    import portal_gb300 as pg

    cloud, mol, rc, J0, J2 = _problem(levels, kmax, points=200)
    with pg.Context(0) as ctx:
        ctx.set_molecule(mol)
        ctx.set_cloud(cloud)
        plain = ctx.solve_se(kmax, J0, J2)[0]
        pops, _, rates = ctx.solve_se(kmax, J0, J2, rates=True)
        np.testing.assert_array_equal(pops, plain)
        for team in ("1", "4"):
            monkeypatch.setenv("PORTAL_SE_TEAM", team)
            np.testing.assert_array_equal(ctx.solve_se(kmax, J0, J2, rates=True)[2], rates)
    bulk, n = cloud.bulk_node_num, 16
    assert not rates[bulk:].any()
    want = oracle.OracleProblem(cloud, mol).solve_se(kmax, J0, J2, 1, n, rates=True)[3][:n]
    scale = np.abs(want).max(axis=2, keepdims=True) + 1e-300
    assert np.abs(want).max() > 0
    assert (np.abs(rates[:n] - want) / scale).max() < 1e-10
