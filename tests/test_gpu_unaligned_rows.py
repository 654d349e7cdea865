"""Device coordinates that are aligned to 4 bytes only: rows take scalar loads instead of
vector loads, with the same results as an aligned copy (exact integers)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [2, 3, 4, 8, 16])
@pytest.mark.parametrize("shift", [1, 2, 3])
def test_unaligned_device_rows(ctx, d, shift):
    import torch
    rng = np.random.default_rng(d)
    n = 3001
    x = (rng.integers(0, 5, (n, 1)) * 4 + rng.normal(0, 0.5, (n, d))).astype(np.float32)
    x[7, d - 1] = np.inf
    flat = torch.zeros(n * d + shift, dtype=torch.float32, device="cuda")
    flat[shift:] = torch.from_numpy(x.reshape(-1)).cuda()
    aligned = torch.from_numpy(x).cuda()
    outs = []
    for p in (aligned.data_ptr(), flat.data_ptr() + 4 * shift):
        nn = torch.empty(n, dtype=torch.int32, device="cuda")
        ci = torch.empty(n, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        r = ctx.run_device(p, n, d, 0.45 * d ** 0.5, 5, nn.data_ptr(), ci.data_ptr(), full_count=True)
        outs.append((nn.cpu().numpy(), ci.cpu().numpy(), r))
    np.testing.assert_array_equal(outs[0][0], outs[1][0])
    np.testing.assert_array_equal(outs[0][1], outs[1][1])
    assert outs[0][2] == outs[1][2]
