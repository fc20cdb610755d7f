"""The split field (J_eff, L*) in every form of the radiation-field kernel, and
items of rays in which some nodes' walks fail (GPU).

Tolerances are those of test_accel.py's split.  J_eff is held against J0, whose
terms it has but for the node's own emission."""
import numpy as np
import pytest

from portal_gb300 import synth
from test_gpu_parity import _check_J

pytestmark = pytest.mark.gpu


def _case(points, levels, angles, nvel, dust):
    mol = synth.linear_rotor(levels) if levels <= 20 else synth.linear_rotor(levels, b_rot_hz=15e9)
    cloud = synth.power_law_sphere(points, levels, mol, t_law="loglinear", b_random=0.3)
    if dust:
        cloud.dust_p = cloud.h2_dens * synth.F4(2.32e-27) / 100.0
    return cloud, mol, synth.RunConfig(nth=angles, nph=angles, nvel=nvel, kmax=2, n_depth=500,
                                       gvec=synth.gauge_vector(3))


# items of rays: one slot, an even number, three; full and odd groups, two of
# them, four; 20 directions (sixteens) and 12 (eights); dust in one, two and
# three slots; 4 directions (whole nodes): one slot, two, three, dust
@pytest.mark.parametrize("points,levels,angles,nvel,dust", [
    (3000, 4, 8, 8, False), (1200, 11, 8, 16, False), (2600, 13, 8, 20, False), (1000, 14, 6, 40, False),
    (600, 40, 6, 16, False), (4000, 4, 5, 8, False), (4000, 3, 4, 32, False), (3000, 4, 8, 12, True),
    (1500, 7, 8, 20, True), (1000, 8, 6, 40, True),
    (900, 5, 2, 15, False), (900, 12, 2, 32, False), (900, 6, 2, 40, False), (900, 7, 2, 20, True)])
def test_split_field(built_lib, points, levels, angles, nvel, dust):
    import oracle
    import portal_gb300 as pg

    cloud, mol, rc = _case(points, levels, angles, nvel, dust)
    with pg.Context(0) as ctx:
        ctx.set_molecule(mol)
        ctx.set_cloud(cloud)
        J0, J2, JE, LS, st = ctx.radiation_field_split(rc)
        pJ0, pJ2 = ctx.radiation_field(rc)[:2]
    assert not st.any()
    np.testing.assert_array_equal(J0, pJ0)
    np.testing.assert_array_equal(J2, pJ2)
    # the first nodes, some in the middle, the last (the shortest items)
    bulk = cloud.bulk_node_num
    nodes = np.concatenate([np.arange(40), np.arange(bulk // 2, bulk // 2 + 24), np.arange(bulk - 40, bulk)])
    o = oracle.OracleProblem(cloud, mol).radiation_field_nodes(rc, nodes, split=True)
    oJ0, oJ2, oJE, oLS = (a[nodes] for a in o[:4])
    _check_J(J0[nodes], J2[nodes], oJ0, oJ2)
    rel = np.abs(JE[nodes] - oJE) / np.abs(oJ0)
    assert rel.max() < 2e-4 and np.median(rel) < 2e-7
    assert np.abs(LS[nodes] - oLS).max() < 2e-6


@pytest.mark.parametrize("angles,nvel,dust", [(8, 8, False), (5, 8, False), (4, 16, False), (8, 12, True)])
def test_failed_walks_among_good_ones(built_lib, angles, nvel, dust):
    """n_depth too small for some of the nodes: an item of rays holds failed
    nodes beside good ones.  The good ones' results are those of the run with
    room, bit for bit; the failed ones' are 0, and their segments those of the
    whole batches of rays before, as the batched kernel's whole nodes count."""
    import portal_gb300 as pg

    cloud, mol, rc = _case(1500, 5, angles, nvel, dust)
    N, L = cloud.node_num, mol.r_num
    g = np.ascontiguousarray(rc.gvec)
    with pg.Context(0) as ctx, pg.Batch(0) as batch:
        ctx.set_molecule(mol)
        ctx.set_cloud(cloud)

        def field(n_depth):
            a = [np.full((N, L), np.nan) for _ in range(4)]
            st = np.full(N, -1, dtype=np.int32)
            code = pg.lib().portal_radiation_field_split(
                ctx._h, rc.nth, rc.nph, rc.nvel, pg._p(g), rc.dx, n_depth, *[pg._p(x) for x in a],
                pg._p(st, pg.P_I), None)
            return code, a, st, ctx.field_moments(), ctx.node_segments()

        code, want, st, moments, seg = field(500)
        assert code == 0 and not st.any()
        # few enough cells that a tenth of the nodes or more fail, and as many are good
        for n_depth in range(8, 64, 4):
            code, got, st, gm, gs = field(n_depth)
            bad = st == pg.NODE_DEPTH
            if 0.1 < bad[:cloud.bulk_node_num].mean() < 0.9:
                break
        assert code == -4 and 0.1 < bad[:cloud.bulk_node_num].mean() < 0.9
        assert ((st == 0) | bad).all()
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a[~bad], b[~bad])
            assert not a[bad].any()
        np.testing.assert_array_equal(gm[~bad], moments[~bad])
        assert not gm[bad].any()
        np.testing.assert_array_equal(gs[~bad], seg[~bad])
        rc.n_depth = n_depth
        batch.add(ctx)
        batch.prepare(rc, autotune=False)
        batch.run()
        np.testing.assert_array_equal(ctx.results(pops=False)[0], got[0])
        np.testing.assert_array_equal(ctx.node_segments(), gs)
