"""The neighbour count where its work items change shape: cells of 1 to 70 points (items
are 32 points of a cell), candidate lists that end inside a step, neighbour lists from
one entry to past their cap, points of one item finishing at different steps.  Every
count kernel against the oracle, bit for bit (integers: no tolerance)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def clumps(d, sizes, seed):
    """Clumps of the given sizes on a coarse lattice: inside a clump distances range from
    0 to about 2 eps (eps = 1), and neighbouring clumps just touch."""
    rng = np.random.default_rng(seed)
    out = []
    for q, m in enumerate(sizes):
        c = np.zeros(d)
        c[0], c[min(1, d - 1)] = 1.5 * (q % 5), c[min(1, d - 1)] + 1.5 * (q // 5)
        out.append(c + rng.uniform(-0.9, 0.9, (m, d)) / np.sqrt(d))
    x = np.concatenate(out)
    return np.ascontiguousarray(x[rng.permutation(len(x))].astype(np.float32))


SIZES = (1, 2, 5, 31, 32, 33, 63, 64, 65, 70, 7, 15, 16, 17, 96, 1, 40, 200, 3, 129)


@pytest.mark.parametrize("d", [1, 2, 3, 4, 5, 7, 8, 9, 13, 16])
@pytest.mark.parametrize("form", ["exact", "gram", "tensor"])
def test_count_items_against_oracle(ctx, d, form):
    if form != "exact" and d < 8:
        pytest.skip("the filters are built for d >= 8")
    x = clumps(d, SIZES, 100 + d)
    kw = {"exact_count": form == "exact", "gram_filter": form == "gram", "tensor_filter": form == "tensor"}
    for m in (1, 2, 17, 33, 66):
        nn_o, ci_o, meta = oracle.grid(x, 1.0, m)
        for full in (True, False):
            nn, ci, r = ctx.run(x, 1.0, m, full_count=full, **kw)
            if full:
                np.testing.assert_array_equal(nn, nn_o)
            else:
                np.testing.assert_array_equal(np.minimum(nn, m), np.minimum(nn_o, m))
            np.testing.assert_array_equal(ci, ci_o)
            assert (r.clusters, r.noise, r.core_count) == (meta["clusters"], meta["noise"], meta["cores"])


@pytest.mark.parametrize("d", [4, 5, 6, 7, 8, 11, 16])
@pytest.mark.parametrize("eps", [1.0, 2.0])
def test_pairs_exactly_at_eps(ctx, d, eps):
    """Integer points: most pairs near eps are exactly at eps, where the FMA sum leaves the
    decision to the reference's sum; half of them moved by a few ulp to either side."""
    rng = np.random.default_rng(d)
    x = rng.integers(0, 3, (3000, d)).astype(np.float32)
    x[::2] += (rng.integers(-2, 3, x[::2].shape) * np.float32(2.0 ** -23)).astype(np.float32)
    for m in (2, 9, 40):
        nn_o, ci_o, meta = oracle.grid(x, eps, m)
        for full in (True, False):
            nn, ci, r = ctx.run(x, eps, m, full_count=full)
            np.testing.assert_array_equal(nn if full else np.minimum(nn, m), nn_o if full else np.minimum(nn_o, m))
            np.testing.assert_array_equal(ci, ci_o)
            assert (r.clusters, r.noise, r.core_count) == (meta["clusters"], meta["noise"], meta["cores"])


@pytest.mark.parametrize("d", [4, 5, 7, 8, 9, 13, 16])
def test_default_count_items_against_oracle(ctx, d):
    """The same shapes by the FMA sum, the default at d >= 4."""
    x = clumps(d, SIZES, 100 + d)
    ctx.set_tuning(tc_min_dim=17)  # CUDA cores
    try:
        for m in (1, 2, 17, 33, 66):
            nn_o, ci_o, meta = oracle.grid(x, 1.0, m)
            for full in (True, False):
                nn, ci, r = ctx.run(x, 1.0, m, full_count=full)
                np.testing.assert_array_equal(nn if full else np.minimum(nn, m), nn_o if full else np.minimum(nn_o, m))
                np.testing.assert_array_equal(ci, ci_o)
                assert (r.clusters, r.noise, r.core_count) == (meta["clusters"], meta["noise"], meta["cores"])
    finally:
        ctx.reset_tuning()


@pytest.mark.parametrize("d", [1, 2, 3, 4, 8, 16])
@pytest.mark.parametrize("extra", [0, 499, 501, 1000, 3999, 4001])
def test_cells_of_little_more_than_a_point(pkg, d, extra):
    """1,000 places on a jittered line or lattice, some with more points: the exact counts of
    grids with fewer than 3/2 points per cell (d <= 2: 5), and just above, have a form of
    their own.  Every third place is within eps of the next."""
    rng = np.random.default_rng(d + extra)
    at = np.zeros((1000, d))
    q = np.arange(1000)
    for k, side in zip(range(min(d, 3)), {1: (1000,), 2: (40, 25), 3: (10, 10, 10)}[min(d, 3)]):
        at[:, k] = 2.6 * (q % side)
        q = q // side
    at[::3, 0] += 1.75  # towards the next place
    x = np.concatenate([at, at[np.arange(extra) % 1000]])
    x = (x + rng.uniform(-0.02, 0.02, x.shape)).astype(np.float32)
    x = np.ascontiguousarray(x[rng.permutation(len(x))])
    for m in (1, 2, 3, 70):
        nn_o, ci_o, meta = oracle.grid(x, 1.0, m)
        for kw in ({}, {"exact_count": True}, {"gram_filter": True}) if d >= 8 else ({}, {"exact_count": True}):
            for full in (True, False):
                with pkg.Context(0) as c:  # a first run knows its cells' number, and so does a batch
                    c.set_tuning(tc_min_dim=17)
                    got = [c.run(x, 1.0, m, full_count=full, **kw)]
                    got += c.run_batched([(x, 1.0, m), (x, 1.0, m)], full_count=full, **kw)
                for nn, ci, r in got:
                    np.testing.assert_array_equal(nn if full else np.minimum(nn, m),
                                                  nn_o if full else np.minimum(nn_o, m))
                    np.testing.assert_array_equal(ci, ci_o)
                    assert (r.clusters, r.noise, r.core_count) == (meta["clusters"], meta["noise"], meta["cores"])
