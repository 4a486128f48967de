"""Inference of the learned guess where a CTA walks over several tiles (the next tile's inputs are worked out
behind the present one's layers): the same rows in one call and in calls of one tile per CTA, bit for bit (a
row's arithmetic does not depend on its tile), around multiples of the tile and of a round of 152 tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 127, 129, 152 * 128, 152 * 128 + 1, 2 * 152 * 128 + 77, 65000])
def test_rows_do_not_depend_on_their_tile(rows):
    from helios_gb300 import api, learned
    P = learned.default_model()
    X = np.random.default_rng(rows).normal(size=(rows, 8)).astype(np.float32)
    Y = api.mlp_predict(P, X)
    assert np.isfinite(Y).all()
    step = 152 * 128 - 64                        # rows move to other places in their tiles
    Z = np.concatenate([api.mlp_predict(P, X[k:k + step]) for k in range(0, rows, step)])
    assert np.array_equal(Y, Z)
