"""A pass of the iterated node loop whose walks fail leaves the results of the
last good one (GPU)."""
import numpy as np
import pytest

from portal_gb300 import synth

pytestmark = pytest.mark.gpu


def _image(ctx):
    return ctx.image([1], [2], 0.3, 0.2, 4, 300.0, 0.0, 4, 0.4, quantities=4)[0]


# items of rays; few directions, so whole nodes; star mode, the batched kernel
@pytest.mark.parametrize("angles,star", [(8, None), (2, None), (8, (5000.0, 1e11, (0.0, 0.0, 0.0)))])
def test_failed_pass_keeps_the_populations(built_lib, angles, star):
    """n_depth 24 is too few cells for some of the nodes' walks.  The populations
    and levels that an image takes are those from before, bit for bit."""
    import portal_gb300 as pg

    mol = synth.linear_rotor(5)
    cloud = synth.power_law_sphere(1024, 8, mol, t_uniform=20.0)
    rc = synth.RunConfig(nth=angles, nph=angles, nvel=8, kmax=2, gvec=synth.gauge_vector(8), n_depth=500)
    short = synth.RunConfig(**{**rc.__dict__, "n_depth": 24})
    with pg.Context(0) as ctx:
        ctx.set_molecule(mol)
        ctx.set_cloud(cloud)
        ctx.set_star(star)
        ctx.radiation_field(rc)
        ctx.solve_se(rc.kmax)
        want = _image(ctx)
        assert np.isfinite(want[0]).any()
        for local in (False, True):
            with pytest.raises(pg.PortalError) as e:
                ctx.lambda_iterate(short, max_iter=3, local_operator=local)
            assert e.value.code == -4 and "n_depth" in str(e.value)
            np.testing.assert_array_equal(_image(ctx), want)
