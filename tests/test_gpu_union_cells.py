"""The union of same-cell-linked cells on dense cells whose links are found late."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("m", [2, 65])
def test_cells_joined_meanwhile_are_not_tested_to_the_end(ctx, full, m):
    """Four cells of 4,000 points in a row on a line (cells are 0.9995 eps wide and start at
    the smallest coordinate).  The first and second and the third and fourth touch through
    their first points.  The second and third touch too, but not through their first 64
    points, so no probe of first points finds that link, while the first and third hold no
    pair in range: 16M pairs when tested to the end."""
    rng = np.random.default_rng(3)
    n = 4000
    jitter = rng.uniform(0, 1e-3, (4, n))
    at = np.empty((4, n))
    at[0] = 0.5
    at[1] = np.where(np.arange(n) < 64, 1.05, 1.9)  # the first points near cell 0
    at[2] = np.where(np.arange(n) < 64, 2.95, 2.1)  # the first points near cell 3
    at[3] = 3.4
    x = (at + jitter).T.reshape(-1, 1)  # the cells' points in turn, each cell's in order
    x = np.concatenate([np.zeros((1, 1)), x]).astype(np.float32)
    assert {len(set(np.floor(v / 0.9995).astype(int))) for v in at + jitter} == {1}
    nn_o, ci_o, meta = oracle.grid(x, 1.0, m)
    nn, ci, r = ctx.run(x, 1.0, m, full_count=full)
    np.testing.assert_array_equal(ci, ci_o)
    np.testing.assert_array_equal(nn if full else np.minimum(nn, m), nn_o if full else np.minimum(nn_o, m))
    assert (r.clusters, r.noise, r.core_count) == (meta["clusters"], meta["noise"], meta["cores"])
    s = ctx.stats()
    assert s["same_cell_linked"] == 1 and s["n_cells"] == 4
    # the link of the second and third is found after 64 of 4,000 points; a test that goes on
    # meanwhile looks at the roots once per 64 points
    assert s["union_pairs"] < n * n // 8
