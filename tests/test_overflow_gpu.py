"""A value that overflows in the Richardson combination of a step comes out infinite,
where it is, and not as a NaN.

q is one large point and tables that leave it as it is; its branches stay finite, four
times the half-step branch does not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = [((1, 24, 10), "generic"), ((1, 24, 10), "cluster-4"), ((7, 9, 11), "generic"), ((7, 9, 11), "cluster-2"), ((16, 16, 16), "cubic"),
         ((64, 64, 64), "register-64"), ((96, 96, 96), "register-96"), ((2, 130, 128), "generic")]


@pytest.mark.parametrize("nsteps", [1, 2], ids=["last", "seam"])
@pytest.mark.parametrize("prec", [8, 4], ids=["fp64", "fp32"])
@pytest.mark.parametrize("nx,impl", FORMS, ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v)))
def test_overflow_is_infinite(nx, impl, prec, nsteps):
    from langevinfts_b200.capi import Context, StepJob, check
    ctx = Context(nx, precision=prec)
    check(ctx.lib.lfts_set_step_impl(ctx.h, impl.encode()))
    dt, big = (np.float64, 6e307) if prec == 8 else (np.float32, 1.2e38)
    M, at = ctx.M, ctx.M // 3
    q = np.zeros(M, dt)
    q[at] = big
    table = ctx.upload(np.full(ctx.Mc, 1.0 / M, dt))
    qd = ctx.malloc((nsteps + 1) * M * prec)
    ctx.h2d(qd, q)
    job = (StepJob * 1)(StepJob(qd, M, qd + M * prec, M, ctx.upload(np.ones(M, dt)), table, table, ctx.malloc(2 * ctx.Mc * 2 * prec)))
    check(ctx.lib.lfts_sweep_continuous(ctx.h, ctx.upload(np.frombuffer(job, dtype=np.uint8)), 1, 0, nsteps))
    got = ctx.d2h(qd, (nsteps + 1, M), dt)[1]
    assert np.isposinf(got[at])
    assert np.all(np.isfinite(np.delete(got, at)))
    ctx.close()
