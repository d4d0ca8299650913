"""The real-space sweeps are as close to extended precision as plain FP64 in the
reference's order of operations.

A rounding of a matrix entry is the same in every step, so it adds up over a chain:
at these lengths one extra (the reciprocal pivots folded into the off-diagonals) shows
as 1.20 (160 points) and 1.44 (200 points) times the error of the reference's order,
while that order with fused multiply-adds stays within 1 % of it (both restated on the
CPU).  The bound lies between."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NSTEPS, DS, BOX, LINES = 100, 1.0 / 60.0, 4.0, 24


def _tables(n, T):
    xf = T(1.0) * T(DS) / ((T(BOX) / T(n)) ** 2 * T(6.0))
    l, d, h = np.full(n, T(-0.5) * xf, T), np.full(n, T(1.0) + xf, T), np.full(n, T(-0.5) * xf, T)
    d[0] += l[0]  # reflecting
    l[0] = h[-1] = 0  # absorbing
    p, c = np.zeros(n, T), np.zeros(n, T)
    p[0] = d[0]
    for i in range(1, n):
        c[i - 1] = h[i - 1] / p[i - 1]
        p[i] = d[i] - l[i] * c[i - 1]
    return l, d, h, T(1.0) / p, c


def _chain(n, w, T):
    """NSTEPS steps of every column of w from q = 1, in precision T throughout."""
    l, d, h, rp, c = _tables(n, T)
    e = np.exp(-w.astype(T) * T(DS) / 2)
    q = np.ones(w.shape, T)
    for _ in range(NSTEPS):
        E = e * q
        r = (2 - d)[:, None] * E - l[:, None] * np.vstack([E[:1], E[:-1]]) - h[:, None] * np.vstack([E[1:], E[-1:]])
        x = np.empty_like(r)
        x[0] = r[0] * rp[0]
        for i in range(1, n):
            x[i] = (r[i] - l[i] * x[i - 1]) * rp[i]
        for i in range(n - 2, -1, -1):
            x[i] -= c[i] * x[i + 1]
        q = e * x
    return q


@pytest.mark.parametrize("n", [160, 200])
def test_error_is_that_of_the_reference_order(n):
    from langevinfts_b200.capi import Context, StepJob, check
    w = np.random.default_rng(1).normal(0.0, 1.0, (n, LINES))
    exact = _chain(n, w, np.longdouble)
    ctx = Context([n])
    tab = np.zeros(ctx.lib.lfts_realspace_table_size(ctx.h))
    check(ctx.lib.lfts_realspace_tables(ctx.h, 1.0, DS, 1, (C.c_double * 1)(BOX / n), (C.c_int * 2)(1, 2), tab.ctypes.data))
    tabd, jobs, q = ctx.upload(tab), (StepJob * LINES)(), ctx.malloc(LINES * (NSTEPS + 1) * n * 8)
    for j in range(LINES):
        fac = ctx.malloc(n * 8)
        check(ctx.lib.lfts_field_factors(ctx.h, ctx.upload(np.ascontiguousarray(w[:, j])), -DS / 4, fac))
        at = q + j * (NSTEPS + 1) * n * 8
        ctx.h2d(at, np.ones(n))
        jobs[j] = StepJob(at, n, at + n * 8, n, fac, tabd, tabd, ctx.malloc(2 * n * 8))
    jp = ctx.upload(np.frombuffer(jobs, dtype=np.uint8))
    for s in range(NSTEPS):
        check(ctx.lib.lfts_step_realspace(ctx.h, jp, LINES, s, 1))
    got = ctx.d2h(q, (LINES, NSTEPS + 1, n), np.float64)[:, -1].T
    ctx.close()

    def error(v):
        return float(np.linalg.norm((v - exact).ravel()) / np.linalg.norm(exact.ravel()))
    assert error(got) <= 1.12 * error(_chain(n, w, np.float64))
