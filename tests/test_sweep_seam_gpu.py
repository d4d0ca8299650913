"""Sweeps of several steps against the same steps taken one by one.

Between two steps of a sweep one kernel does the end of the one and the start of
the next, for every kernel family that has it; the rounding differs only in the
second step's forward transform, so the results agree to a few units of round-off
per step (the step tests' tolerance).  Jobs whose flag is off stay untouched."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FAMILIES = [((16,) * 3, "cubic"), ((32,) * 3, "cubic"), ((48,) * 3, "cubic"), ((64,) * 3, "register-64"), ((64,) * 3, "cubic"),
            ((96,) * 3, "register-96"), ((96,) * 3, "cubic"), ((128,) * 3, "cubic"), ((20, 18, 14), "generic"), ((1, 300, 7), "generic")]


@pytest.mark.parametrize("discrete", [False, True], ids=["continuous", "discrete"])
@pytest.mark.parametrize("prec", [8, 4], ids=["fp64", "fp32"])
@pytest.mark.parametrize("nx,impl", FAMILIES, ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v)))
def test_sweep_equals_single_steps(nx, impl, prec, discrete):
    from langevinfts_b200.capi import Context, StepJob, check
    ctx = Context(nx, precision=prec)
    if ctx.lib.lfts_set_step_impl(ctx.h, impl.encode()) != 0:
        ctx.close()
        pytest.skip("not available for this grid and precision")
    dt, nsteps, njobs = (np.float64 if prec == 8 else np.float32), 3, 3
    rng = np.random.default_rng(sum(nx))
    bond, half = ctx.malloc(ctx.Mc * prec), ctx.malloc(ctx.Mc * prec)
    check(ctx.lib.lfts_bond_tables(ctx.h, 1.0, 0.02, (C.c_double * 3)(3.0, 2.6, 3.4), bond, half))
    active = ctx.upload(np.array([1, 0, 1], dtype=np.int32))
    jobs = (StepJob * njobs)()
    for j in range(njobs):
        fac = ctx.upload(np.exp(-0.005 * rng.normal(0.0, 1.0, ctx.M)).astype(dt))
        q = ctx.malloc((nsteps + 1) * ctx.M * prec)
        ctx.h2d(q, np.exp(rng.normal(0.0, 0.3, ctx.M)).astype(dt))
        jobs[j] = StepJob(q, ctx.M, q + ctx.M * prec, ctx.M, fac, bond, half, ctx.malloc(2 * ctx.Mc * 2 * prec), active, j, 0)
    jp = ctx.upload(np.frombuffer(jobs, dtype=np.uint8))
    out = []
    for sweep in (False, True):
        for j in range(njobs):
            ctx.h2d(jobs[j].in_ + ctx.M * prec, np.full(nsteps * ctx.M, -7.0, dt))
        if sweep:
            check(ctx.lib.lfts_sweep_discrete(ctx.h, jp, njobs, 0, nsteps, 0, 1) if discrete
                  else ctx.lib.lfts_sweep_continuous(ctx.h, jp, njobs, 0, nsteps))
        else:
            for s in range(nsteps):
                check(ctx.lib.lfts_step_discrete(ctx.h, jp, njobs, s, 0, 1) if discrete
                      else ctx.lib.lfts_step_continuous(ctx.h, jp, njobs, s))
        out.append([ctx.d2h(jobs[j].in_, (nsteps + 1, ctx.M), dt) for j in range(njobs)])
    tol = 1e-12 if prec == 8 else 2e-5
    for j in (0, 2):
        for s in range(1, nsteps + 1):
            assert np.max(np.abs(out[0][j][s] - out[1][j][s])) <= tol * s * np.max(np.abs(out[0][j][s]))
    assert np.all(out[1][1][1:] == -7.0)
    ctx.close()
