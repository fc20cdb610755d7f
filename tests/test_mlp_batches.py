"""Training batches around the 16 rows of a CTA of the whole-network kernels
(GPU): gradients against the oracle with its BF16 rounding points, tolerances
of test_mlp.py."""
import numpy as np
import pytest

import oracle.mlp as om
from test_mlp import _params


@pytest.mark.gpu
@pytest.mark.parametrize("B", [15, 16, 17, 48, 64])
def test_gradients_around_a_block_of_rows(built_lib, B):
    import portal_gb300 as pg

    shape = (9, 72, 2, 24)
    shapes = om.layer_shapes(*shape)
    p = _params(shapes, 5)
    rng = np.random.default_rng(B)
    X = rng.normal(size=(B, shape[0])).astype(np.float32)
    T = rng.normal(size=(B, shape[3])).astype(np.float32)
    with pg.MLP(*shape, seed=1) as m:
        m.set_params(p)
        loss, g = m.gradients(X, T)
    lref, gref = om.loss_and_grad(p, shapes, X, T, bf16=True)
    assert abs(loss - lref) <= 1e-5 * lref
    o = 0
    for fo, fi in shapes:
        for n in (fo * fi, fo):
            a, r = g[o:o + n].astype(np.float64), gref[o:o + n]
            assert np.abs(a - r).max() <= 2e-3 * np.abs(r).max(), (o, n)
            o += n
