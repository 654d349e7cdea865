"""Items that the CUDA-core count hands on to the tensor-core count: data on which hardly a
point is done early, against the plain count, bit for bit (whole numbers: no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def gauss(n, d, seed, sigma=3.0):
    return np.random.default_rng(seed).normal(0, sigma, (n, d)).astype(np.float32)


def same(got, want, m):
    nn, ci, r = got
    nn_o, ci_o, r_o = want
    np.testing.assert_array_equal(np.minimum(nn, m), np.minimum(nn_o, m))
    np.testing.assert_array_equal(ci, ci_o)
    assert tuple(r) == tuple(r_o)


@pytest.mark.parametrize("d", [12, 13, 16])
@pytest.mark.parametrize("n", [65_537, 80_003])
def test_items_handed_on(ctx, d, n):
    x = gauss(n, d, d)
    eps = 1.2 * d ** 0.5  # 0.28 of the mean distance: stencils of a large share of the points, few neighbours
    for m in (3, 24, 65, 66, 1000):  # lists from short to their cap, and none
        for kw in ({}, {"gram_filter": True}):
            want = ctx.run(x, eps, m, exact_count=True)
            assert ctx.stats()["tensor_filter"] == 0
            same(ctx.run(x, eps, m, **kw), want, m)
            s = ctx.stats()
            if m >= 24:
                assert s["tensor_filter"] == 1 and s["tensor_items"] > s["n_tiles"] // 2


def test_items_stay_where_points_are_done_early(ctx):
    """Forty clusters, all points core: no item is handed on; and none on small jobs."""
    rng = np.random.default_rng(4)
    x = (rng.uniform(0, 100, (40, 13))[rng.integers(0, 40, 90_000)] + rng.normal(0, 0.5, (90_000, 13))).astype(np.float32)
    want = ctx.run(x, 3.0, 8, exact_count=True)
    same(ctx.run(x, 3.0, 8), want, 8)
    assert ctx.stats()["tensor_items"] == 0
    y = gauss(65_536, 13, 5)
    same(ctx.run(y, 6.8, 24), ctx.run(y, 6.8, 24, exact_count=True), 24)


def test_items_handed_on_in_a_batch(ctx):
    """Jobs of different eps and minPts in one pipeline of more than 65,536 points."""
    jobs = [(gauss(n, 13, n), e * 13 ** 0.5, m) for n, e, m in
            ((40_001, 1.2, 24), (33, 1.0, 3), (40_000, 1.1, 64), (20_011, 1.3, 2), (1, 1.0, 1))]
    got = ctx.run_batched(jobs)
    assert ctx.stats()["tensor_items"] > 0
    for g, (x, e, m) in zip(got, jobs):
        same(g, ctx.run(x, e, m, exact_count=True), m)
