"""The tensor-core count with the early exit where its chunks change length: chunks are
equal shares of a cell of at most 32 to 256 points, by the points of the run and minPts, and
a chunk's points wait for a column.  Runs of 100,000 to 8M points in cells of every
ragged size against the plain count, exact integers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ragged(n, d, seed):
    """Clumps (a cell or a few) of 1 to 700 points, next to each other in pairs."""
    rng = np.random.default_rng(seed)
    sizes = rng.integers(1, 701, 2 * n // 350 + 2)
    sizes = sizes[:int(np.searchsorted(np.cumsum(sizes), n)) + 1]
    c = np.zeros((len(sizes), d))
    q = np.arange(len(sizes))
    c[:, 0], c[:, 1], c[:, 2], c[:, 3] = q % 2 * 1.6, q // 2 % 32 * 6, q // 64 % 32 * 6, q // 2048 * 6
    x = np.repeat(c, sizes, axis=0)[:n] + rng.uniform(-0.9, 0.9, (n, d)) / np.sqrt(d)
    return np.ascontiguousarray(x[rng.permutation(n)].astype(np.float32))


# chunks of 32 points (or more, by the rule that lays them out)
@pytest.mark.parametrize("d,n", [(8, 100_000), (8, 800_011), (12, 400_003), (16, 200_001), (16, 800_011)])
@pytest.mark.parametrize("m", [5, 32, 60, 300, 600])
def test_queue_against_the_plain_count(ctx, d, n, m):
    x = ragged(n, d, n + d)
    nn_e, ci_e, r_e = ctx.run(x, 1.0, m, exact_count=True)
    nn, ci, r = ctx.run(x, 1.0, m, tensor_filter=True)
    assert ctx.stats()["tensor_filter"] == 1
    np.testing.assert_array_equal(np.minimum(nn, m), np.minimum(nn_e, m))
    np.testing.assert_array_equal(ci, ci_e)
    assert r == r_e


# chunks of 64 points; 96 (64 from minPts 512 on); 256
@pytest.mark.parametrize("d,n", [(9, 1_900_003), (16, 2_900_011), (8, 8_000_003)])
@pytest.mark.parametrize("m", [5, 60, 600])
def test_long_chunks_against_the_plain_count(ctx, d, n, m):
    test_queue_against_the_plain_count(ctx, d, n, m)
