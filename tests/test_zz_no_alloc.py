"""The batch entry point that allocates nothing (bc_lde_batch_noalloc).

It exists for callers that cannot call cudaMalloc -- a prover whose own pool
already holds nearly all of device memory, or a submission path that must not
trigger cudaMalloc's device-wide synchronisation -- and keeps its schedule in
a fixed array inside the library.  Its output must equal the existing
bc_lde_fused entry point, bit for bit, on two calls in a row (the second call
reuses the array the first one left behind).  This file is collected last so
that a run stopping at the first failure has already run every other test.
"""
import ctypes

import numpy as np
import pytest

from conftest import raw_u64, to_dev, to_host

pytestmark = pytest.mark.gpu

SPECS_A = [(3, 2, 1), (12, 3, 2), (13, 1, 1), (16, 5, 3), (18, 2, 1), (20, 1, 2)]
SPECS_B = [(10, 4, 3), (14, 7, 1), (17, 3, 2), (21, 2, 1)]


def _jobs(rng, specs):
    import torch

    import bc_ntt

    out = []
    for log_n, cols, log_b in specs:
        n = 1 << log_n
        ev = to_dev(raw_u64(rng, cols * n))
        dst = torch.full(((1 << log_b) * cols * n,), 0x11, dtype=torch.int64, device="cuda")
        out.append((ev, dst, log_n, cols, log_b))
    arr = (bc_ntt.LdeJob * len(out))()
    for i, (ev, dst, log_n, cols, log_b) in enumerate(out):
        n = 1 << log_n
        arr[i] = bc_ntt.LdeJob(ev.data_ptr(), dst.data_ptr(), n, n, cols * n, log_n, cols, log_b, 0)
    return out, arr


def _run_noalloc(arr, n):
    import torch

    import bc_ntt

    status = ctypes.c_uint32(0xFFFF)
    rc = bc_ntt.lib().bc_lde_batch_noalloc(ctypes.cast(arr, ctypes.c_void_p), n,
                                           torch.cuda.current_stream().cuda_stream, ctypes.byref(status))
    assert rc == 0, f"bc_lde_batch_noalloc returned {rc}"
    assert status.value == 0


def _check_against_fused(jobs):
    import torch

    import bc_ntt

    for ev, dst, log_n, cols, log_b in jobs:
        ref = torch.empty_like(dst)
        bc_ntt.lde(ev, ref, log_n, cols, log_b, fused=True)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(to_host(dst), to_host(ref), err_msg=f"log_n={log_n} cols={cols}")


def test_noalloc_batch_matches_fused_twice(gpu_ctx):
    rng = np.random.default_rng(2025)
    jobs_a, arr_a = _jobs(rng, SPECS_A)
    _run_noalloc(arr_a, len(SPECS_A))
    _check_against_fused(jobs_a)
    # second call in a row, different jobs: the array still holds the first schedule
    jobs_b, arr_b = _jobs(rng, SPECS_B)
    _run_noalloc(arr_b, len(SPECS_B))
    _check_against_fused(jobs_b)


def test_noalloc_batch_rejects_oversized_schedule(gpu_ctx):
    import torch

    import bc_ntt

    # one job whose schedule needs far more than the fixed array: 2^24 x 4096 columns (pointers are never touched)
    big = (bc_ntt.LdeJob * 1)()
    big[0] = bc_ntt.LdeJob(16, 16, 1 << 24, 1 << 24, 4096 << 24, 24, 4096, 1, 0)
    rc = bc_ntt.lib().bc_lde_batch_noalloc(ctypes.cast(big, ctypes.c_void_p), 1,
                                           torch.cuda.current_stream().cuda_stream, None)
    assert rc == 1  # cudaErrorInvalidValue


def test_noalloc_batch_rejects_stream_capture(gpu_ctx):
    """Its schedule is copied from host memory the call frees on return, so a call on a capturing stream is
    refused (cudaErrorStreamCaptureUnsupported) and enqueues nothing; the stream stays usable afterwards."""
    import torch

    import bc_ntt

    rng = np.random.default_rng(7)
    jobs, arr = _jobs(rng, [(12, 2, 1)])
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    rcs = []
    with torch.cuda.graph(graph, stream=side):
        rcs.append(bc_ntt.lib().bc_lde_batch_noalloc(ctypes.cast(arr, ctypes.c_void_p), 1, side.cuda_stream, None))
    assert rcs == [900]  # cudaErrorStreamCaptureUnsupported
    del graph
    _run_noalloc(arr, 1)
    _check_against_fused(jobs)


@pytest.mark.parametrize("log_n,cols,jobs_per_batch", [(8, 1, 36000), (13, 1, 7400)])
def test_noalloc_batch_holds_many_small_jobs(gpu_ctx, log_n, cols, jobs_per_batch):
    """The fixed array holds 36,000 one-kernel or 7,400 three-kernel jobs: 16 bytes and a kernel's own parameters for
    each kernel, 8 bytes a work item."""
    import torch

    import bc_ntt

    n, log_b = 1 << log_n, 1
    (job,), _ = _jobs(np.random.default_rng(3), [(log_n, cols, log_b)])
    outs = torch.full((jobs_per_batch, (cols * n) << log_b), 0x11, dtype=torch.int64, device="cuda")
    arr = (bc_ntt.LdeJob * jobs_per_batch)()
    for i in range(jobs_per_batch):
        arr[i] = bc_ntt.LdeJob(job[0].data_ptr(), outs.data_ptr() + 8 * i * outs.shape[1], n, n, cols * n, log_n, cols, log_b, 0)
    status = ctypes.c_uint32(0xFFFF)
    rc = bc_ntt.lib().bc_lde_batch_noalloc(ctypes.cast(arr, ctypes.c_void_p), jobs_per_batch,
                                           torch.cuda.current_stream().cuda_stream, ctypes.byref(status))
    assert rc == 0 and status.value == 0
    ref = torch.empty_like(job[1])
    bc_ntt.lde(job[0], ref, log_n, cols, log_b)
    assert bool((outs == ref).all())


def test_noalloc_batch_takes_other_splits_when_its_plans_do_not_fit(gpu_ctx):
    """505 jobs of 33 columns of 2^17 need more than the array with the shipped table's split, less with another: the
    batch is accepted and exact.  A plan that the caller imported is not replaced."""
    import torch

    import bc_ntt

    log_n, cols, log_b, count = 17, 33, 1, 505
    n = 1 << log_n
    (job,), _ = _jobs(np.random.default_rng(4), [(log_n, cols, log_b)])
    outs = torch.full((count, (cols * n) << log_b), 0x11, dtype=torch.int64, device="cuda")
    arr = (bc_ntt.LdeJob * count)()
    for i in range(count):
        arr[i] = bc_ntt.LdeJob(job[0].data_ptr(), outs.data_ptr() + 8 * i * outs.shape[1], n, n, cols * n, log_n, cols,
                               log_b, 0)

    def run():
        status = ctypes.c_uint32(0xFFFF)
        rc = bc_ntt.lib().bc_lde_batch_noalloc(ctypes.cast(arr, ctypes.c_void_p), count,
                                               torch.cuda.current_stream().cuda_stream, ctypes.byref(status))
        return rc, status.value

    try:
        bc_ntt.plan_table_import(f"{log_n} {log_b} 2 5 8 12 1\n")
        assert run()[0] == 1  # cudaErrorInvalidValue, nothing enqueued
        bc_ntt.plan_table_clear()
        assert bc_ntt.load_tuned_plans()
        assert run() == (0, 0)
        ref = torch.empty_like(job[1])
        bc_ntt.lde(job[0], ref, log_n, cols, log_b)
        assert all(bool((o == ref).all()) for o in outs)
    finally:
        bc_ntt.plan_table_clear()
        del outs
        torch.cuda.empty_cache()
