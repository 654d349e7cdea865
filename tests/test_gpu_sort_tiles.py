"""The radix sort at the edges of its tiles (4,096 elements for 32-bit cell keys, 2,048
for 64-bit ones), through whole jobs: a misplaced element moves a point to another cell
and changes its count.  Exact integers, no tolerance."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 255, 2047, 2048, 2049, 4095, 4096, 4097, 8193, 20481])
@pytest.mark.parametrize("wide", [False, True])
def test_sort_tiles(ctx, n, wide):
    rng = np.random.default_rng(n)
    # wide: more than 2^32 cells, so 64-bit keys and eight passes at most
    x = rng.uniform(0, 3000 if wide else 40, (n, 3)).astype(np.float32)
    if n > 40:
        x[:40] = x[-40:] + np.float32(0.1)  # some pairs in range
        x[5, 1] = np.nan                    # a point outside the grid sorts to the end
    nn_o, ci_o, meta = oracle.grid(x, 1.0, 2)
    nn, ci, r = ctx.run(x, 1.0, 2, full_count=True)
    if wide and n > 2000:
        assert ctx.stats()["key_bytes"] == 8
    np.testing.assert_array_equal(nn, nn_o)
    np.testing.assert_array_equal(ci, ci_o)
    assert (r.clusters, r.noise, r.core_count) == (meta["clusters"], meta["noise"], meta["cores"])
