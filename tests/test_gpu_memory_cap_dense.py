"""A context under a memory cap runs what the cap has room for: a job of up to 65,536
points in few cells needs row tables and items for those cells only, not for as many
cells as it has points.  Against the oracle, exact integers."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


# (d, points, eps, minPts, tensor filter, cap): the buffers of these jobs at their own
# sizes hold 8 and 17 MB; row tables for one cell per point would add 13 MB to either
@pytest.mark.parametrize("d,n,eps,m,tensor,cap", [(3, 65_536, 1.0, 10, False, 10 << 20),
                                                  (12, 60_000, 3.0, 24, True, 20 << 20)])
def test_cap_admits_a_dense_job(pkg, d, n, eps, m, tensor, cap):
    rng = np.random.default_rng(d)
    x = (rng.integers(0, 3, (n, d)) * (np.arange(d) < 2) * 6 + rng.normal(0, 0.25, (n, d))).astype(np.float32)
    nn_o, ci_o, meta = oracle.grid(x, eps, m)
    with pkg.Context(0) as c:
        c.set_memory_limit(cap)
        nn, ci, r = c.run(x, eps, m, tensor_filter=tensor)
        assert c.device_bytes() <= cap
    np.testing.assert_array_equal(np.minimum(nn, m), np.minimum(nn_o, m))
    np.testing.assert_array_equal(ci, ci_o)
    assert (r.clusters, r.noise, r.core_count) == (meta["clusters"], meta["noise"], meta["cores"])
