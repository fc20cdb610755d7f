"""The radiation-field kernel at the edges of its line groups, packs and
channel slots, against the oracle and against the batched kernel (GPU).

Line groups hold up to 10 lines (5 with dust), two lines to a pack; channels
run in passes of two 32-channel slots, with one channel more taken
lanes-over-lines (33, 65, 129, 257 channels).  Clouds this small run as ray
ranges summed afterwards; the batched kernel always takes whole nodes, so
equal bits between the two pin that sum's order as well.  Tolerances are
those of test_gpu_parity.py: the formulas are the same at every shape."""
import numpy as np
import pytest

from portal_gb300 import synth
from test_gpu_parity import _check_J

pytestmark = pytest.mark.gpu


# (levels, nvel, dust): one line; an odd group and one slot; a full group and
# a single odd slot with a remainder; two groups; two odd groups and three
# slots; two groups of ten and a remainder on two passes; four groups (40
# levels: more than 32 lines, no remainder channel); dust: one group, two
@pytest.mark.parametrize("levels,nvel,dust", [(2, 8, False), (4, 15, False), (11, 16, False), (12, 32, False),
                                              (14, 40, False), (20, 64, False), (40, 16, False), (6, 16, True),
                                              (8, 40, True)])
def test_line_groups_and_slots(built_lib, levels, nvel, dust):
    import oracle
    import portal_gb300 as pg

    # 40 levels of a heavier rotor: the lines stay below 1.2 THz, as in the 20-level cases
    mol = synth.linear_rotor(levels) if levels <= 20 else synth.linear_rotor(levels, b_rot_hz=15e9)
    cloud = synth.power_law_sphere(300, levels, mol, t_law="loglinear", b_random=0.3)
    if dust:
        cloud.dust_p = cloud.h2_dens * synth.F4(2.32e-27) / 100.0
    rc = synth.RunConfig(nth=6, nph=6, nvel=nvel, kmax=2, n_depth=500, gvec=synth.gauge_vector(3))
    with pg.Context(0) as ctx, pg.Batch(0) as batch:
        ctx.set_molecule(mol)
        ctx.set_cloud(cloud)
        J0, J2, st, nseg = ctx.radiation_field(rc)
        seg, moments = ctx.node_segments(), ctx.field_moments()
        assert not st.any() and seg.sum() == nseg
        batch.add(ctx)
        batch.prepare(rc, autotune=False)
        bseg, _ = batch.run()
        bJ0, bJ2, _ = ctx.results(pops=False)
        assert bseg == nseg
        np.testing.assert_array_equal(bJ0, J0)
        np.testing.assert_array_equal(bJ2, J2)
        np.testing.assert_array_equal(ctx.field_moments(), moments)
    oJ0, oJ2, _, _, _ = oracle.OracleProblem(cloud, mol).radiation_field(rc, 1, 100)
    _check_J(J0[:100], J2[:100], oJ0[:100], oJ2[:100])


# (points, angles, nvel, dust): ranges of 32, 16 and 8 rays of 44 directions;
# 20 directions (no thirty-twos: an item has two nodes at most) and 12 (eights
# alone); dust; two slots and more lines than a group
@pytest.mark.parametrize("points,angles,nvel,dust,levels", [(3000, 8, 8, False, 4), (4000, 5, 8, False, 4),
                                                            (4000, 4, 8, False, 3), (3000, 8, 12, True, 4),
                                                            (2600, 8, 20, False, 13)])
def test_items_of_rays(built_lib, points, angles, nvel, dust, levels):
    """Ranges of rays that cross from a node to the next, summed afterwards:
    equal bits to the batched kernel's whole nodes, and the split field's plain
    part too."""
    import portal_gb300 as pg

    mol = synth.linear_rotor(levels)
    cloud = synth.power_law_sphere(points, levels, mol, t_law="loglinear", b_random=0.3)
    if dust:
        cloud.dust_p = cloud.h2_dens * synth.F4(2.32e-27) / 100.0
    rc = synth.RunConfig(nth=angles, nph=angles, nvel=nvel, kmax=2, n_depth=500, gvec=synth.gauge_vector(3))
    with pg.Context(0) as ctx, pg.Batch(0) as batch:
        ctx.set_molecule(mol)
        ctx.set_cloud(cloud)
        sJ0, sJ2 = ctx.radiation_field_split(rc)[:2]
        J0, J2, st, nseg = ctx.radiation_field(rc)
        seg, moments = ctx.node_segments(), ctx.field_moments()
        assert not st.any() and seg.sum() == nseg
        np.testing.assert_array_equal(sJ0, J0)
        np.testing.assert_array_equal(sJ2, J2)
        batch.add(ctx)
        batch.prepare(rc, autotune=False)
        bseg, _ = batch.run()
        bJ0, bJ2, _ = ctx.results(pops=False)
        assert bseg == nseg
        np.testing.assert_array_equal(bJ0, J0)
        np.testing.assert_array_equal(bJ2, J2)
        np.testing.assert_array_equal(ctx.field_moments(), moments)
        np.testing.assert_array_equal(ctx.node_segments(), seg)
