"""The image march's FP32 prediction against the oracle's step-by-step march
(GPU): the recorded lists decide the optical depth, so tau pixel by pixel."""
import numpy as np
import pytest

from portal_gb300 import synth

pytestmark = pytest.mark.gpu


# (points, extra neighbours per list, per-node maps): a sparse cloud (few,
# long cells), one as dense as the default workload, lists past the 64
# neighbours of the candidate mask, rays through nodes
@pytest.mark.parametrize("points,extra,nodes", [(64, 0, False), (4096, 0, False), (600, 70, False), (600, 70, True),
                                                (2048, 0, True)])
def test_march_against_oracle(built_lib, points, extra, nodes):
    import oracle
    import portal_gb300 as pg

    mol = synth.linear_rotor(4)
    cloud = synth.power_law_sphere(points, 3, mol, b_random=0.3)
    if extra:
        rng = np.random.default_rng(1)
        off, idx = [0], []
        for i in range(points):
            own = set(cloud.nb_idx[cloud.nb_off[i]:cloud.nb_off[i + 1]].tolist())
            more = [int(x) for x in rng.choice(points, extra, replace=False) if x != i]
            idx += sorted(own | set(more))
            off.append(len(idx))
        cloud.nb_off, cloud.nb_idx = np.array(off, dtype=np.int64), np.array(idx, dtype=np.int32)
        assert np.diff(cloud.nb_off).min() > 64
    g = np.sqrt(2.0 * mol.j_lev + 1.0)
    pp = np.zeros((points, 2 * mol.nlev))
    pp[:, 0::2] = cloud.lev_p / cloud.lev_p.sum(axis=1, keepdims=True) / g
    pp[:, 1::2] = 1e-2 * pp[:, 0::2]
    P = oracle.OracleProblem(cloud, mol)
    nvel, pix = 4, 9
    npx, nch = 2 * pix + 1, 2 * nvel + 1
    with pg.Context(0) as ctx:
        ctx.set_molecule(mol)
        ctx.set_cloud(cloud)
        if nodes:
            cube, _, st = ctx.image_nodes([1], [2], 0.7, 0.3, nvel, 100.0, 0.0, pol_pops=pp)
            ref, _, ost, nf = P.image_nodes([1], [2], pp, 0.7, 0.3, nvel, 100.0, 0.0)
            tau, otau = cube[3, 0], ref[3].reshape(points, nch).T
        else:
            cube, st = ctx.image([1], [2], 0.7, 0.3, nvel, 100.0, 0.0, pix, 0.7, pol_pops=pp)
            ref, ost, nf = P.image([1], [2], pp, 0.7, 0.3, nvel, 100.0, 0.0, pix, 0.7)
            tau, otau = cube[3, 0], ref[3].reshape(npx, npx, nch).transpose(2, 1, 0)
    assert nf == 0 and not st.any()
    assert np.array_equal(np.isnan(tau), np.isnan(otau))
    ok = ~np.isnan(otau)
    # equal lists leave the FP32 rounding of each term (a few 6e-8) and of the compensated sum
    assert np.abs(tau[ok] - otau[ok]).max() <= 1e-6 * np.abs(otau[ok]).max()
