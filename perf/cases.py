"""What a user of this framework has it do, as cases that can be timed and compared.

Every case is one DBSCAN job, or one batch of jobs, through the package's public entry
points: `Context.run_device` on device tensors, `Context.run` and `data_process` on host
arrays, `ndb_b200_run_noalloc` for callers that may not allocate, and
`Context.run_batched_jobs` / `Context.run_batched` for many jobs at once.  The sizes and
distributions are those of the benchmark workloads (`synthetic.py`), drawn on the GPU:

  mix2   2-D, 20 Gaussians in [0, 100]^2, 5 % noise (eps 0.8, minPts 5 at 100k points)
  mix3   3-D, 500 anisotropic Gaussians in [0, 1000]^3, 2 % noise (eps 1.5, minPts 10)
  mix8   8-D, 200 Gaussians in [0, 50]^8, 5 % noise (eps 1.2, minPts 8)
  skew   2-D, Zipf-sized Gaussians and filaments in [0, 10000]^2 (eps 0.5, minPts 4)
  job    any d, 5 to 50 Gaussians in [0, 100]^d, 5 % noise; eps is the 90th percentile, over
         1 % of the points, of the distance to the 4th neighbour, minPts = 2d (one job of
         the 4,096-job batch)

With the early exit (`full` false) a core's neighbour count only says "at least minPts",
so those cases return the counts clamped at minPts: all that the call defines.  All
outputs are whole numbers decided by separately rounded FP32 sums, so there is no 64-bit
value for them, and this file defines no `exact`.
"""
import ctypes
import importlib
import math
import random

import numpy as np
import torch

pkg = importlib.import_module("nextdbscan-exa_b200")

# the smallest and largest job, and the dimensionalities, of the 4,096-job batch
JOB_MIN, JOB_MAX, JOB_DIMS = 1_000, 200_000, (2, 3, 8, 16)


def listed():
    return [
        # the smallest job of the batch workload, alone: latency and launches are the cost
        dict(name="small-2d-1k", entry="device", data="job", n=1_000, d=2, eps=0.0, min_pts=4, full=False),
        # a service that reserved its memory at start-up and may not allocate: ragged, 3-D
        dict(name="noalloc-3d-20k", entry="noalloc", data="job", n=20_011, d=3, eps=0.0, min_pts=6, full=False),
        # the plain 2-D workload on device tensors
        dict(name="plain-2d-100k", entry="device", data="mix2", n=100_000, d=2, eps=0.8, min_pts=5, full=False),
        # the reference's own program: host arrays, both phases, exact counts for every point
        dict(name="dropin-2d-100k", entry="dropin", data="mix2", n=100_000, d=2, eps=0.8, min_pts=5, full=True),
        # a dimensionality between the low ones (cells linked) and the high ones, ragged size, exact counts
        dict(name="full-5d-300k", entry="device", data="job", n=300_007, d=5, eps=0.0, min_pts=10, full=True),
        # host arrays end to end: copies in, the job, copies out
        dict(name="host-3d-1m", entry="host", data="mix3", n=1_000_003, d=3, eps=3.0, min_pts=10, full=True),
        # the plain 3-D workload at full size
        dict(name="plain-3d-10m", entry="device", data="mix3", n=10_000_000, d=3, eps=1.5, min_pts=10, full=False),
        # the 8-D workload: core flags and clusters only, and exact counts for every point
        dict(name="plain-8d-2m", entry="device", data="mix8", n=2_000_000, d=8, eps=1.2, min_pts=8, full=False),
        dict(name="full-8d-2m", entry="device", data="mix8", n=2_000_000, d=8, eps=1.2, min_pts=8, full=True),
        # the largest 16-D job of the batch workload, alone, ragged
        dict(name="plain-16d-200k", entry="device", data="job", n=199_999, d=16, eps=0.0, min_pts=32, full=False),
        # the skewed 2-D workload at full size: clusters of very different density
        dict(name="skew-2d-100m", entry="device", data="skew", n=100_000_000, d=2, eps=0.5, min_pts=4, full=False),
        # the benchmark's batch: thousands of independent jobs in one call, device tensors
        dict(name="batch-4096", entry="batch", jobs=4096),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choices(("device", "host", "dropin", "noalloc", "batch", "batch_host"), (45, 12, 8, 10, 17, 8))[0]
    if entry in ("batch", "batch_host"):
        return dict(entry=entry, jobs=_log_uniform(rng, 8, 1024 if entry == "batch" else 128))
    d = rng.choice((1, 2, 2, 3, 3, 4, 5, 6, 7, 8, 8, 10, 12, 13, 16, 16))
    top = 10_000_000 if d <= 3 else 2_000_000 if d <= 8 else 400_000
    if entry == "noalloc":
        top = 32_768
    elif entry in ("host", "dropin"):
        top = min(top, 2_000_000)
    full = entry in ("host", "dropin") or rng.random() < 0.3
    return dict(entry=entry, data="job", n=_log_uniform(rng, 1_000, top), d=d, eps=0.0, min_pts=2 * d, full=full)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device="cuda")


def _mixture(g, n, centers, sigma, noise, box):
    """n points of the Gaussians (centers k x d, sigma k x d), a share `noise` of them uniform in [0, box]^d."""
    k, d = centers.shape
    which = torch.randint(k, (n,), generator=g, device="cuda")
    x = torch.randn(n, d, generator=g, device="cuda").mul_(sigma[which]).add_(centers[which])
    stray = (_rand(g, n) < noise).nonzero()[:, 0]
    x[stray] = _rand(g, stray.numel(), d) * box
    return x


def _skewed(g, rng, n):
    k, box = 10_000, 10_000.0
    cdf = (torch.arange(1, k + 1, device="cuda", dtype=torch.float64) ** -1.2).cumsum(0)
    cdf = (cdf / cdf[-1]).float()
    centers, sigma = _rand(g, k, 2) * box, _rand(g, k, 1) * 2.9 + 0.1
    which = torch.searchsorted(cdf, _rand(g, n)).clamp_(max=k - 1)
    x = torch.randn(n, 2, generator=g, device="cuda").mul_(sigma[which]).add_(centers[which])
    del which
    kind = _rand(g, n)
    stray = (kind < 0.01).nonzero()[:, 0]
    x[stray] = _rand(g, stray.numel(), 2) * box
    for f in range(10):  # filaments: polylines of 2 to 7 legs, 5 % of the points
        at = ((kind >= 0.01 + 0.005 * f) & (kind < 0.015 + 0.005 * f)).nonzero()[:, 0]
        verts = _rand(g, rng.randint(3, 8), 2) * box
        legs = (verts[1:] - verts[:-1]).norm(dim=1)
        ends = legs.cumsum(0)
        t = _rand(g, at.numel()) * ends[-1]
        leg = torch.searchsorted(ends, t).clamp_(max=legs.numel() - 1)
        frac = ((t - ends[leg] + legs[leg]) / legs[leg])[:, None]
        x[at] = verts[leg] + (verts[leg + 1] - verts[leg]) * frac + torch.randn(
            at.numel(), 2, generator=g, device="cuda") * 0.2
    return x


def _points(case, g, rng):
    n, d, data = case["n"], case["d"], case["data"]
    if data == "skew":
        return _skewed(g, rng, n)
    if data == "mix2":
        return _mixture(g, n, _rand(g, 20, 2) * 100, (_rand(g, 20, 1) * 1.5 + 0.5).expand(20, 2), 0.05, 100.0)
    if data == "mix3":
        return _mixture(g, n, _rand(g, 500, 3) * 1000, 0.5 * 10 ** _rand(g, 500, 3), 0.02, 1000.0)
    if data == "mix8":
        return _mixture(g, n, _rand(g, 200, 8) * 50, (_rand(g, 200, 1) * 0.7 + 0.3).expand(200, 8), 0.05, 50.0)
    k = rng.randint(5, 50)
    return _mixture(g, n, _rand(g, k, d) * 100, (_rand(g, k, 1) * 1.5 + 0.5).expand(k, d), 0.05, 100.0)


def _fourth_neighbours(x):
    """The distances of the first 1 % of the points (10 to 256) to their 4th neighbours."""
    n = x.shape[0]
    m = x[:max(10, min(n // 100, 256, (1 << 28) // n))]
    d2 = (m * m).sum(1)[:, None] + (x * x).sum(1) - 2 * (m @ x.T)  # near enough for a choice of eps
    return d2.topk(5, largest=False).values[:, -1].clamp_(min=0).sqrt_()


def _eps_4nn(x):
    return float(torch.quantile(_fourth_neighbours(x), 0.9))


def _job_shapes(case):
    """(n, d) of the jobs of a batch, by d: the same for every seed."""
    rng = random.Random(case["jobs"])
    shapes = [(_log_uniform(rng, JOB_MIN, JOB_MAX), rng.choice(JOB_DIMS)) for _ in range(case["jobs"])]
    return sorted(shapes, key=lambda s: s[1])


def _batch_points(shapes, g, rng):
    """The points of every job (a flat tensor, job after job) and every job's eps."""
    flat, eps = [], []
    for d in sorted({d for _, d in shapes}):
        sizes = [n for n, dd in shapes if dd == d]
        ks = torch.tensor([rng.randint(5, 50) for _ in sizes], device="cuda")
        first = ks.cumsum(0) - ks
        centers, sigma = _rand(g, int(ks.sum()), d) * 100, _rand(g, int(ks.sum()), 1) * 1.5 + 0.5
        job = torch.repeat_interleave(torch.arange(len(sizes), device="cuda"), torch.tensor(sizes, device="cuda"))
        which = first[job] + (_rand(g, job.numel()) * ks[job]).long().clamp_(max=49).minimum(ks[job] - 1)
        x = torch.randn(job.numel(), d, generator=g, device="cuda").mul_(sigma[which]).add_(centers[which])
        del which, job
        stray = (_rand(g, x.shape[0]) < 0.05).nonzero()[:, 0]
        x[stray] = _rand(g, stray.numel(), d) * 100
        at = 0
        for n in sizes:
            eps.append(_fourth_neighbours(x[at:at + n]))
            at += n
        flat.append(x.reshape(-1))
    ends = np.cumsum([e.numel() for e in eps])[:-1]
    return torch.cat(flat), [float(np.quantile(e, 0.9)) for e in np.split(torch.cat(eps).cpu().numpy(), ends)]


# ---------------------------------------------------------------------------
# one call
# ---------------------------------------------------------------------------
def prepare(case, seed):
    g, rng = _generator(seed), random.Random(int(seed))
    s = dict(case)
    if case["entry"] != "noalloc":
        s["ctx"] = pkg.Context(0)  # the handle a program keeps
    if case["entry"] in ("batch", "batch_host"):
        shapes = _job_shapes(case)
        x, eps = _batch_points(shapes, g, rng)
        return _prepare_batch(s, shapes, x, eps) if case["entry"] == "batch" else _prepare_batch_host(s, shapes, x, eps)
    x = _points(case, g, rng)
    s["eps"] = case["eps"] or _eps_4nn(x)
    if case["entry"] in ("host", "dropin"):
        s["x"] = x.cpu().numpy()
        return s
    s["x"] = x
    s["nn"] = torch.empty(case["n"], dtype=torch.int32, device="cuda")
    s["ci"] = torch.empty(case["n"], dtype=torch.int32, device="cuda")
    s["stream"] = torch.cuda.Stream()  # the program's stream: the library's work and the program's own follow each other
    if case["entry"] == "noalloc":
        f = pkg.lib.load().ndb_b200_run_noalloc
        f.argtypes = [ctypes.c_void_p, ctypes.c_int64, ctypes.c_int32, ctypes.c_float, ctypes.c_int32, ctypes.c_uint32,
                      ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
        f.restype = ctypes.c_int
        s["noalloc"] = f
    else:
        s["ctx"].set_stream(s["stream"].cuda_stream)
    return s


def _prepare_batch(s, shapes, x, eps):
    total = sum(n for n, _ in shapes)
    s["x"] = x
    s["nn"] = torch.empty(total, dtype=torch.int32, device="cuda")
    s["ci"] = torch.empty(total, dtype=torch.int32, device="cuda")
    s["stream"] = torch.cuda.Stream()
    s["ctx"].set_stream(s["stream"].cuda_stream)
    jobs = (pkg.lib.NdbJob * len(shapes))()
    at_x = at = 0
    s["same_d"] = {}
    for j, ((n, d), e) in enumerate(zip(shapes, eps)):
        jobs[j].coords = x.data_ptr() + 4 * at_x
        jobs[j].n, jobs[j].d, jobs[j].eps, jobs[j].min_pts = n, d, e, 2 * d
        jobs[j].nn_out = s["nn"].data_ptr() + 4 * at
        jobs[j].cluster_index_out = s["ci"].data_ptr() + 4 * at
        at_x += n * d
        at += n
        s["same_d"].setdefault(d, [at - n, at])[1] = at
    s["job_table"] = jobs
    words = np.frombuffer(jobs, dtype=np.int32).reshape(len(shapes), -1)
    first = pkg.lib.NdbJob.result.offset // 4
    s["meta"] = words[:, first:first + 5]  # every job's result and status, as the call leaves them
    return s


def _prepare_batch_host(s, shapes, x, eps):
    x = x.cpu().numpy()
    s["problems"], at = [], 0
    for (n, d), e in zip(shapes, eps):
        s["problems"].append((x[at:at + n * d].reshape(n, d), e, 2 * d))
        at += n * d
    return s


def run(s):
    entry = s["entry"]
    if entry == "device":
        r = s["ctx"].run_device(s["x"].data_ptr(), s["n"], s["d"], s["eps"], s["min_pts"], s["nn"].data_ptr(),
                                s["ci"].data_ptr(), full_count=s["full"])
        return {"nn": _defined_counts(s), "ci": s["ci"], "meta": tuple(r)}
    if entry == "noalloc":
        r = pkg.lib.NdbResult()
        flags = pkg.lib.FLAG_DEVICE_PTRS | (pkg.lib.FLAG_FULL_COUNT if s["full"] else 0)
        st = s["noalloc"](s["x"].data_ptr(), s["n"], s["d"], s["eps"], s["min_pts"], flags, s["nn"].data_ptr(),
                          s["ci"].data_ptr(), ctypes.byref(r), s["stream"].cuda_stream)
        pkg.lib.check(st, "ndb_b200_run_noalloc")
        return {"nn": _defined_counts(s), "ci": s["ci"], "meta": (r.clusters, r.noise, r.core_count, r.n)}
    if entry == "host":
        nn, ci, r = s["ctx"].run(s["x"], s["eps"], s["min_pts"], full_count=s["full"])
        return {"nn": nn, "ci": ci, "meta": tuple(r)}
    if entry == "dropin":
        dp = pkg.data_process(s["x"], s["min_pts"], s["eps"], s["d"], s["n"], False, full_count=s["full"],
                              context=s["ctx"])
        dp.select_and_process()
        dp.select_cores_and_process()
        return {"nn": dp.v_coord_nn, "ci": dp.v_coord_cluster_index, "meta": dp.get_result_meta()}
    if entry == "batch":
        st = s["ctx"].run_batched_jobs(s["job_table"], len(s["job_table"]), pkg.lib.FLAG_DEVICE_PTRS)
        pkg.lib.check(st, "ndb_b200_run_batched")
        with torch.cuda.stream(s["stream"]):
            for d, (a, b) in s["same_d"].items():
                s["nn"][a:b].clamp_(max=2 * d)
        return {"nn": s["nn"], "ci": s["ci"], "meta": s["meta"]}
    got = s["ctx"].run_batched(s["problems"], full_count=True)
    return {"nn": np.concatenate([nn for nn, _, _ in got]), "ci": np.concatenate([ci for _, ci, _ in got]),
            "meta": np.array([r for _, _, r in got], dtype=np.int32)}


def _defined_counts(s):
    if not s["full"]:
        with torch.cuda.stream(s["stream"]):
            s["nn"].clamp_(max=s["min_pts"])
    return s["nn"]


def work(case):
    """Coordinates read, counts and cluster ids written, and minPts pair predicates (3 operations per dimension) per
    point: below that many no count is decided."""
    shapes = _job_shapes(case) if "jobs" in case else [(case["n"], case["d"])]
    min_pts = (lambda d: 2 * d) if "jobs" in case else (lambda d: case["min_pts"])
    return {"bytes": float(sum(n * (4 * d + 8) for n, d in shapes)),
            "flops": float(sum(n * min_pts(d) * 3 * d for n, d in shapes))}
