"""The statistics of a run say what ran."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,per_pair", [({}, lambda d: 2 * d + 1 if d >= 4 else 3 * d),
                                           ({"exact_count": True}, lambda d: 3 * d),
                                           ({"gram_filter": True}, lambda d: d + 3)])
@pytest.mark.parametrize("d", [2, 3, 4, 8, 11])
@pytest.mark.parametrize("full", [True, False])
def test_fp32_operations_are_those_of_the_count_that_ran(ctx, form, per_pair, d, full):
    if "gram_filter" in form and d < 8:
        pytest.skip("the Gram filter is built for d >= 8")
    rng = np.random.default_rng(d)
    x = (rng.integers(0, 4, (4000, 1)) * 5 + rng.normal(0, 0.5, (4000, d))).astype(np.float32)
    ctx.set_tuning(tc_min_dim=17)  # CUDA cores
    try:
        ctx.run(x, 0.4 * d ** 0.5, 2 * d, full_count=full, **form)
        s = ctx.stats()
        assert s["tensor_filter"] == 0 and s["count_pairs"] > 0
        assert s["count_fp32_ops"] == s["count_pairs"] * per_pair(d)
        ctx.run_batched([(x, 0.4 * d ** 0.5, 2 * d), (x[:2000], 0.4 * d ** 0.5, 2 * d)], full_count=full, **form)
        s = ctx.stats()
        assert s["count_fp32_ops"] == s["count_pairs"] * per_pair(d)
    finally:
        ctx.reset_tuning()


@pytest.mark.parametrize("full", [True, False])
def test_fp32_operations_of_pairs_on_the_tensor_cores(ctx, full):
    rng = np.random.default_rng(1)
    x = (rng.integers(0, 4, (4000, 1)) * 5 + rng.normal(0, 0.5, (4000, 8))).astype(np.float32)
    ctx.run(x, 1.2, 16, full_count=full, tensor_filter=True)  # every item on the tensor cores
    s = ctx.stats()
    assert s["tensor_items"] == s["n_tiles"] and s["count_pairs"] > 0
    assert s["count_fp32_ops"] == 3 * s["count_pairs"] and s["count_pair_dims"] == 8 * s["count_pairs"]
    ctx.run_batched([(x, 1.2, 16), (x[:1500], 1.2, 16)], full_count=full, tensor_filter=True)
    s = ctx.stats()
    assert s["tensor_items"] == s["n_tiles"] and s["count_fp32_ops"] == 3 * s["count_pairs"] > 0


def test_border_time_covers_the_border_step(ctx):
    """With neighbour lists the border ids are written by the output pass.  20M points: it
    reads a count, a flag and an index of 4 + 1 + 4 bytes and writes 8 bytes a point, 340
    MB, past the L2; at 8 TB/s that is 42 us, and an event pair without a launch in
    between reads about 3."""
    import torch
    n = 20_000_000
    x = torch.rand((n, 2), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)) * 3000
    nn = torch.empty(n, dtype=torch.int32, device="cuda")
    ci = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx.run_device(x.data_ptr(), n, 2, 0.8, 5, nn.data_ptr(), ci.data_ptr())
    s = ctx.stats()
    assert s["ms_border_kernel"] >= 17 * n / 8e12 * 1e3
    assert s["ms_border_kernel"] <= s["ms_border"]
