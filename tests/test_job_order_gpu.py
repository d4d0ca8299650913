"""Job arrays filled by a kernel on the stream right before the call.

The step kernels' launches may start before the kernel ahead of them has ended; what
that kernel wrote, the job array included, may be read only behind their wait.  The
array first holds other, valid jobs, so a kernel that read too early would work on
those."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CALLS = [("realspace", (24, 20, 18)), ("realspace", (30, 26)), ("realspace", (70,)), ("continuous", (64, 64, 64)), ("continuous", (96, 96, 96)),
         ("continuous", (32, 32, 32)), ("continuous", (31, 20, 18)), ("sweep", (1, 40, 36)), ("discrete", (64, 64, 64)),
         ("discrete", (48, 48, 48)), ("discrete", (31, 20, 18))]


@pytest.mark.parametrize("call,nx", CALLS, ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v)))
def test_jobs_written_just_before_the_call_are_the_ones_done(call, nx):
    import torch
    from langevinfts_b200.capi import Context, StepJob, check
    nj = 3
    ctx = Context(nx)
    M, Mc, L = ctx.M, ctx.Mc, ctx.lib
    stream = torch.cuda.Stream()
    rng = np.random.default_rng(sum(nx))
    if call == "realspace":
        dim = len(nx)
        tab = np.zeros(L.lfts_realspace_table_size(ctx.h))
        check(L.lfts_realspace_tables(ctx.h, 1.0, 0.02, dim, (C.c_double * dim)(*[3.0 / n for n in nx]), (C.c_int * (2 * dim))(), tab.ctypes.data))
        bond = half = ctx.upload(tab)
    else:
        bond, half = ctx.malloc(Mc * 8), ctx.malloc(Mc * 8)
        check(L.lfts_bond_tables(ctx.h, 1.0, 0.02, (C.c_double * 3)(3.0, 2.6, 3.4), bond, half))
    fac = ctx.upload(np.exp(-0.005 * rng.normal(0.0, 1.0, M)))
    spec = ctx.malloc(nj * 2 * max(M, 2 * Mc) * 8)
    sets = []
    for _ in range(2):  # the jobs that stand there before, and the ones to be done
        jobs = (StepJob * nj)()
        for j in range(nj):
            q = ctx.malloc(2 * M * 8)
            ctx.h2d(q, np.concatenate([1.0 + 0.3 * rng.random(M), np.full(M, -7.0)]))
            jobs[j] = StepJob(q, M, q + M * 8, M, fac, bond, half, spec + j * 2 * max(M, 2 * Mc) * 8)
        sets.append(jobs)
    new = torch.from_numpy(np.frombuffer(sets[1], dtype=np.int64).copy()).cuda()
    work = torch.randn(1 << 24, device="cuda")
    run = {"realspace": lambda p: L.lfts_step_realspace(ctx.h, p, nj, 0, len(nx)), "continuous": lambda p: L.lfts_step_continuous(ctx.h, p, nj, 0),
           "discrete": lambda p: L.lfts_step_discrete(ctx.h, p, nj, 0, 0, 1), "sweep": lambda p: L.lfts_sweep_continuous(ctx.h, p, nj, 0, 1)}[call]
    array = torch.from_numpy(np.frombuffer(sets[0], dtype=np.int64).copy()).cuda()
    torch.cuda.synchronize()
    check(L.lfts_ctx_set_stream(ctx.h, stream.cuda_stream))
    with torch.cuda.stream(stream):
        for _ in range(4):
            work.mul_(1.0001)
        torch.add(new, 0, out=array)
        check(run(array.data_ptr()))
    got = [[ctx.d2h(jobs[j].out, (M,), np.float64) for j in range(nj)] for jobs in sets]
    assert all(np.all(g == -7.0) for g in got[0])
    assert all(np.all(g != -7.0) and np.all(np.isfinite(g)) for g in got[1])
    check(L.lfts_ctx_set_stream(ctx.h, None))
    ctx.close()
