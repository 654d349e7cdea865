"""The unions over core points (grids whose cells are not linked) where their work list
changes shape: no candidates, a few segments, several segments per item, more segments
than the list holds; with neighbour lists and without.  Cluster ids are exact integers:
no tolerance."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [4, 7, 8, 16])
@pytest.mark.parametrize("m", [1, 3, 12, 70])
def test_chains_of_clumps_against_oracle(ctx, d, m):
    """Clumps of 300 to 3,000 points whose neighbours touch through a few points only, so
    lists alone leave several components per cell."""
    rng = np.random.default_rng(10 * d + m)
    parts = []
    for q, size in enumerate((3000, 300, 1500, 40, 2500, 1, 700)):
        c = np.zeros(d)
        c[q % 4] = 1.4 * (q + 1)
        parts.append(c + rng.normal(0, 0.28, (size, d)))
    bridge = np.zeros((60, d))
    bridge[:, 0] = np.linspace(0, 8, 60)
    x = np.concatenate(parts + [bridge]).astype(np.float32)
    x = x[rng.permutation(len(x))]
    eps = 0.25 * np.sqrt(d)
    _, ci_o, meta = oracle.grid(x, eps, m)
    for full in (True, False):
        _, ci, r = ctx.run(x, eps, m, full_count=full)
        np.testing.assert_array_equal(ci, ci_o)
        assert (r.clusters, r.noise, r.core_count) == (meta["clusters"], meta["noise"], meta["cores"])


def test_more_segments_than_the_list_holds(ctx):
    """Two balls of 120,000 and 80,000 points, each wholly within eps, and minPts past the
    neighbour-list cap: about 320,000 segments for a list of 200,000."""
    rng = np.random.default_rng(5)
    x = rng.uniform(-0.2, 0.2, (200_000, 4))
    ball = np.arange(200_000) % 5 < 2
    x[ball, 1] += 50.0
    x = x.astype(np.float32)
    _, ci, r = ctx.run(x, 1.0, 70)
    assert tuple(r) == (2, 0, 200_000, 200_000)
    # the smallest point of the balls: 0 (the second ball) and 2 (the first)
    np.testing.assert_array_equal(ci, np.where(ball, 0, 2))


@pytest.mark.parametrize("d,m", [(4, 2), (9, 32), (16, 28)])
def test_exact_counts_on_points_all_near_leave_little_to_the_scan(ctx, d, m):
    """20,000 points within eps of each other, 625 items: joined before the scan of
    candidates, which would otherwise test every item against hundreds of others."""
    x = np.random.default_rng(d).uniform(0, 1, (20_000, d)).astype(np.float32)
    nn, ci, r = ctx.run(x, 1.01 * np.sqrt(d), m, full_count=True)
    assert tuple(r) == (1, 0, 20_000, 20_000)
    np.testing.assert_array_equal(nn, 20_000)
    np.testing.assert_array_equal(ci, 0)
    assert ctx.stats()["union_pairs"] < 20_000
    (nn, ci, r), (nn2, ci2, r2) = ctx.run_batched([(x, 1.01 * np.sqrt(d), m), (x[:777], 1.01 * np.sqrt(d), m)],
                                                  full_count=True)
    assert tuple(r) == (1, 0, 20_000, 20_000) and tuple(r2) == (1, 0, 777, 777)
    np.testing.assert_array_equal(ci, 0)
    assert ctx.stats()["union_pairs"] < 20_777
