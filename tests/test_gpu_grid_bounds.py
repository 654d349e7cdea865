"""Where the grid phase changes its bounds: jobs up to 65,536 points launch over an upper
bound of their cells, larger ones over the cells' count; prefix tiles of 2,048 points,
1,024 cells and 65,536 bitmap bits; jobs with no point, or one, in the grid.  Against the
oracle, exact integers."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def check(ctx, x, eps, m):
    nn_o, ci_o, meta = oracle.grid(x, eps, m)
    for full in (True, False):
        nn, ci, r = ctx.run(x, eps, m, full_count=full)
        np.testing.assert_array_equal(nn if full else np.minimum(nn, m), nn_o if full else np.minimum(nn_o, m))
        np.testing.assert_array_equal(ci, ci_o)
        assert (r.clusters, r.noise, r.core_count) == (meta["clusters"], meta["noise"], meta["cores"])
        s = ctx.stats()
        assert 0 <= s["n_cells"] <= s["n_valid"] and s["n_cells"] <= s["n_tiles"] <= s["n_valid"]


@pytest.mark.parametrize("n", [65535, 65536, 65537])
@pytest.mark.parametrize("d,eps,m", [(2, 0.3, 4), (3, 1.0, 5), (5, 3.5, 6)])
def test_around_the_cell_bound(ctx, n, d, eps, m):
    rng = np.random.default_rng(n + d)
    c = rng.uniform(0, 100, (30, d))
    x = c[rng.integers(0, 30, n)] + rng.normal(0, 1.5, (n, d))
    x[rng.random(n) < 0.1] *= 1.3
    check(ctx, x.astype(np.float32), eps, m)


@pytest.mark.parametrize("d", [1, 2, 3, 5, 9])
@pytest.mark.parametrize("valid", [0, 1, 2])
@pytest.mark.parametrize("m", [0, 1, 2])
def test_few_points_in_the_grid(ctx, d, valid, m):
    x = np.full((70, d), np.nan, dtype=np.float32)
    x[10:10 + valid] = 1.0
    x[40, 0] = np.finfo(np.float32).max
    check(ctx, x, 0.5, m)
