"""A context's first run allocates for the cells that the job has: a dense job of up to
65,536 points does not get a row table for as many cells as points (12 MB here, where the
job's buffers need 6), whose allocation would cost more than the rest of the run.  Later
runs may: the context is then one that comes back."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def test_first_run_of_a_dense_job(pkg):
    rng = np.random.default_rng(6)
    n = 60_000
    x = (rng.integers(0, 3, (n, 3)) * 6 + rng.normal(0, 0.25, (n, 3))).astype(np.float32)
    nn_o, ci_o, meta = oracle.grid(x, 1.0, 5)
    with pkg.Context(0) as c:
        for first in (True, False):
            nn, ci, r = c.run(x, 1.0, 5, full_count=True)
            np.testing.assert_array_equal(nn, nn_o)
            np.testing.assert_array_equal(ci, ci_o)
            assert (r.clusters, r.noise, r.core_count) == (meta["clusters"], meta["noise"], meta["cores"])
            assert c.device_bytes() < 12 << 20 or not first


def test_first_run_of_a_small_job_sizes_its_row_table_by_its_cells(pkg):
    """40,000 points in few cells, 2-D: five stencil rows of 8 bytes a cell.  The second run
    bounds the cells by the points, 1.6 MB of rows; the first one has counted them."""
    x = np.random.default_rng(2).uniform(0, 10, (40_000, 2)).astype(np.float32)
    with pkg.Context(0) as c:
        nn, ci, _ = c.run(x, 1.0, 5)
        first = c.device_bytes()
        assert c.stats()["n_cells"] < 400
        nn2, ci2, _ = c.run(x, 1.0, 5)
        assert first + 1_500_000 < c.device_bytes()
    np.testing.assert_array_equal(ci, ci2)
    np.testing.assert_array_equal(np.minimum(nn, 5), np.minimum(nn2, 5))
