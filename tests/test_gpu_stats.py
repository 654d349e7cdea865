"""The statistics of a run say what ran."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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
