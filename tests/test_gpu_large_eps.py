"""eps whose square is next to the largest FP32 number.  There the FMA sum of a pair can
round to infinity while the reference's sum is eps^2, so such runs take the reference's
sum for every pair.  Against the oracle, exact integers."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def check(ctx, x, eps, m):
    nn_o, ci_o, _, meta = oracle.reference(x, eps, m)
    for full in (True, False):
        nn, ci, r = ctx.run(x, eps, m, full_count=full)
        np.testing.assert_array_equal(nn if full else np.minimum(nn, m), nn_o if full else np.minimum(nn_o, m))
        np.testing.assert_array_equal(ci, ci_o)
        assert (r.clusters, r.noise, r.core_count) == (meta["clusters"], meta["noise"], meta["cores"])
    return nn_o


def largest_eps(step):
    """The step-th largest FP32 number whose FP32 square is finite."""
    e = np.nextafter(np.float32(2.0) ** 64, np.float32(0))
    for _ in range(step):
        e = np.nextafter(e, np.float32(0))
    with np.errstate(over="ignore"):
        assert np.isfinite(e * e)
    return float(e)


def test_pair_whose_sum_is_the_largest_square(ctx):
    h = [float.fromhex(s) for s in ("0x1.bbd4c8p+62", "0x1.238804p+63", "0x1.a7da92p+62", "0x1.201632p+63")]
    x = np.array([[0.0] * 4, h], dtype=np.float32)
    assert list(check(ctx, x, largest_eps(0), 2)) == [2, 2]


@pytest.mark.parametrize("d", [4, 8, 16])
@pytest.mark.parametrize("step", range(5))
def test_pairs_within_a_few_ulp_of_the_largest_eps(ctx, d, step):
    rng = np.random.default_rng(10 * d + step)
    eps = largest_eps(step)
    u = rng.normal(size=(1500, d))
    r = eps * (1 + rng.integers(-4, 5, (1500, 1)) * 2.0 ** -24)
    x = np.concatenate([np.zeros((1, d)), u / np.linalg.norm(u, axis=1, keepdims=True) * r]).astype(np.float32)
    check(ctx, x, eps, 3)
