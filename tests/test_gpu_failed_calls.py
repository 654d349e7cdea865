"""A run that fails in its label phase: the counts are in the caller's buffer all the same,
and nothing of the call outlives it (the grid and the counts stay for
ndb_b200_assign_labels, which writes its own buffer only)."""
import ctypes

import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu
SENTINEL = -123456


def device_job(name="c2_n6000", repeat=1):
    import torch
    g = load_golden(name)
    x = np.tile(g["coords"], (repeat, 1))
    x[:, 0] += np.repeat(np.arange(repeat, dtype=np.float32) * 4096, len(g["coords"]))
    x = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    nn = torch.full((len(x),), SENTINEL, dtype=torch.int32, device="cuda")
    ci = torch.full((len(x),), SENTINEL, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return x, float(g["eps"]), int(g["min_pts"]), nn, ci


def expected(pkg, x, eps, m):
    with pkg.Context(0) as c:
        return c.run(x.cpu().numpy(), eps, m, full_count=True)


def finish(pkg, c, ci):
    res = pkg.lib.NdbResult()
    st = pkg.lib.load().ndb_b200_assign_labels(c.handle, ctypes.c_void_p(ci.data_ptr()), ctypes.byref(res))
    assert st == 0
    return res.clusters, res.noise, res.core_count, res.n


def check_after_the_failure(pkg, c, x, nn, ci, want):
    import torch
    np.testing.assert_array_equal(nn.cpu().numpy(), want[0])  # the failed call's counts
    nn.fill_(SENTINEL)  # the buffer is the caller's again
    torch.cuda.synchronize()
    assert finish(pkg, c, ci) == tuple(want[2])
    assert (nn.cpu().numpy() == SENTINEL).all()
    np.testing.assert_array_equal(ci.cpu().numpy(), want[1])


def test_host_pointer_for_the_labels(pkg):
    x, eps, m, nn, ci = device_job()
    want = expected(pkg, x, eps, m)
    host = np.empty(len(x), dtype=np.int32)
    with pkg.Context(0) as c:
        with pytest.raises(pkg.lib.NdbError, match="INVALID_ARGUMENT"):
            c.run_device(x.data_ptr(), *x.shape, eps, m, nn.data_ptr(), host.ctypes.data, full_count=True)
        check_after_the_failure(pkg, c, x, nn, ci, want)


def test_label_phase_past_the_memory_cap(pkg):
    x, eps, m, nn, ci = device_job(repeat=12)  # 72,000 points
    want = expected(pkg, x, eps, m)
    with pkg.Context(0) as c:  # the footprint of phase 1
        flags = pkg.lib.FLAG_DEVICE_PTRS | pkg.lib.FLAG_FULL_COUNT
        st = pkg.lib.load().ndb_b200_classify(c.handle, ctypes.c_void_p(x.data_ptr()), *x.shape, ctypes.c_float(eps),
                                              m, flags, ctypes.c_void_p(nn.data_ptr()))
        assert st == 0
        phase1 = c.device_bytes()
    nn.fill_(SENTINEL)
    with pkg.Context(0) as c:
        c.set_memory_limit(phase1)
        with pytest.raises(pkg.lib.NdbError, match="OUT_OF_MEMORY"):
            c.run_device(x.data_ptr(), *x.shape, eps, m, nn.data_ptr(), ci.data_ptr(), full_count=True)
        c.set_memory_limit(0)
        check_after_the_failure(pkg, c, x, nn, ci, want)


def test_batch_right_after_a_refused_run(pkg):
    """The refused run's kernels are done when it returns, so the batch that follows at once
    finds the transfer buffer they share idle."""
    names = ("c1_n4000", "blobs_d8", "c2_n6000")
    golden = [load_golden(k) for k in names]
    problems = [(g["coords"], float(g["eps"]), int(g["min_pts"])) for g in golden]
    x, eps, m, _, _ = device_job(repeat=10)  # 60,000 points
    host = np.empty(len(x), dtype=np.int32)
    with pkg.Context(0) as c:
        c.run_batched(problems, full_count=True)  # the buffer at its size for the batch
        for _ in range(10):
            with pytest.raises(pkg.lib.NdbError, match="INVALID_ARGUMENT"):
                c.run_device(x.data_ptr(), *x.shape, eps, m, None, host.ctypes.data, full_count=True)
            for g, (nn, ci, r) in zip(golden, c.run_batched(problems, full_count=True)):
                np.testing.assert_array_equal(nn, g["nn"])
                np.testing.assert_array_equal(ci, g["cluster_index"])
                assert list(r) == list(g["meta"])
