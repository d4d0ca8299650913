"""Any-extent step kernels and cluster sweeps against the numpy oracle.

Extents at which they can go wrong: one plane, one row, one column and one
point along an axis, radices of every kind (2..13, 16, primes above 13 alone
and twice), odd and even extents (unpaired planes, Nyquist), columns and planes
that do not divide among the CTAs, and every cluster size the grid fits.  The
tolerance is the step tests' one: round-off of three transforms a step.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(1, 1, 24), (1, 1, 289), (1, 12, 10), (1, 84, 48), (1, 37, 9), (6, 1, 9), (5, 4, 3), (2, 2, 2), (16, 7, 2), (13, 11, 8),
         (17, 5, 4), (9, 10, 34), (31, 49, 23), (20, 18, 14), (33, 26, 25), (80, 60, 48), (3, 100, 110)]


def _setup(nx, prec, njobs, nsteps):
    from langevinfts_b200.capi import Context, StepJob, check
    from oracle import lfts_oracle as orc
    ctx = Context(nx, precision=prec)
    dt = np.float64 if prec == 8 else np.float32
    rng = np.random.default_rng(sum(nx) + njobs)
    lx, ds, b2 = [3.0, 2.6, 3.4], 0.02, 1.0
    bond, half = ctx.malloc(ctx.Mc * prec), ctx.malloc(ctx.Mc * prec)
    check(ctx.lib.lfts_bond_tables(ctx.h, b2, ds, (C.c_double * 3)(*lx), bond, half))
    tab = (orc.boltz_bond(nx, lx, b2, ds), orc.boltz_bond(nx, lx, b2 / 2, ds))
    jobs, q0, w = (StepJob * njobs)(), [], []
    for j in range(njobs):
        wj = rng.normal(0.0, 1.0, ctx.M)
        q = np.exp(rng.normal(0.0, 0.3, ctx.M)).astype(dt)
        fac = ctx.malloc(ctx.M * prec)
        check(ctx.lib.lfts_field_factors(ctx.h, ctx.upload(wj), -ds / 4, fac))
        d = ctx.malloc((nsteps + 1) * ctx.M * prec)
        ctx.h2d(d, q)
        jobs[j] = StepJob(d, ctx.M, d + ctx.M * prec, ctx.M, fac, bond, half, ctx.malloc(2 * ctx.Mc * 2 * prec))
        q0.append(q.astype(np.float64))
        w.append(wj)
    return ctx, jobs, ctx.upload(np.frombuffer(jobs, dtype=np.uint8)), q0, w, tab, lx, ds


def _check(ctx, jobs, q0, w, tab, lx, nx, ds, prec, nsteps, discrete):
    from oracle import lfts_oracle as orc
    g = orc.Grid(nx, lx)
    dt = np.float64 if prec == 8 else np.float32
    tol = 1e-12 if prec == 8 else 2e-5
    for j in range(len(q0)):
        got = ctx.d2h(jobs[j].in_, (nsteps + 1, ctx.M), dt)
        ref = q0[j]
        e = np.exp(-w[j] * ds / 4)
        for s in range(nsteps):
            ref = orc.step_discrete(g, ref, e, tab[0]) if discrete else orc.step_continuous(g, ref, e ** 2, e, tab[0], tab[1])
            assert np.max(np.abs(got[s + 1] - ref)) <= tol * (s + 1) * np.max(np.abs(ref)), (j, s)


@pytest.mark.parametrize("discrete", [False, True], ids=["continuous", "discrete"])
@pytest.mark.parametrize("prec", [8, 4], ids=["fp64", "fp32"])
@pytest.mark.parametrize("nx", GRIDS, ids=lambda n: "x".join(map(str, n)))
def test_steps_and_sweeps_match_the_oracle(nx, prec, discrete):
    from langevinfts_b200.capi import check
    nsteps = 3
    for njobs in (1, 3):
        ctx, jobs, jp, q0, w, tab, lx, ds = _setup(nx, prec, njobs, nsteps)
        for impl in ("generic", "cluster-1", "cluster-2", "cluster-4", "cluster-8", "cluster-16"):
            if ctx.lib.lfts_set_step_impl(ctx.h, impl.encode()) != 0:
                continue
            for j in range(njobs):  # what an earlier implementation wrote must not pass for this one's
                ctx.h2d(jobs[j].in_ + ctx.M * prec, np.full(nsteps * ctx.M, np.nan, np.float64 if prec == 8 else np.float32))
            if discrete:
                check(ctx.lib.lfts_sweep_discrete(ctx.h, jp, njobs, 0, nsteps, 0, 1))
            else:
                check(ctx.lib.lfts_sweep_continuous(ctx.h, jp, njobs, 0, nsteps))
            _check(ctx, jobs, q0, w, tab, lx, nx, ds, prec, nsteps, discrete)
        ctx.close()


def test_inactive_jobs_are_left_alone_by_sweeps():
    from langevinfts_b200.capi import check
    nx, nsteps = (1, 40, 36), 2
    ctx, jobs, _, q0, w, tab, lx, ds = _setup(nx, 8, 4, nsteps)
    active = ctx.upload(np.array([1, 0, 1, 0], dtype=np.int32))
    for j in range(4):
        jobs[j].active, jobs[j].replica = active, j
        ctx.h2d(jobs[j].in_ + ctx.M * 8, np.full(nsteps * ctx.M, -7.0))
    jp = ctx.upload(np.frombuffer(jobs, dtype=np.uint8))
    for impl in ("generic", "cluster-4"):
        check(ctx.lib.lfts_set_step_impl(ctx.h, impl.encode()))
        check(ctx.lib.lfts_sweep_continuous(ctx.h, jp, 4, 0, nsteps))
        for j in (1, 3):
            assert np.all(ctx.d2h(jobs[j].in_ + ctx.M * 8, (nsteps * ctx.M,), np.float64) == -7.0)
    for j in (0, 2):
        _check(ctx, [jobs[j]], [q0[j]], [w[j]], tab, lx, nx, ds, 8, nsteps, False)
    ctx.close()


def test_cluster_sizes_a_grid_does_not_fit_are_refused():
    from langevinfts_b200.capi import Context
    ctx = Context((96, 96, 80))
    assert ctx.lib.lfts_set_step_impl(ctx.h, b"cluster-16") != 0
    assert ctx.lib.lfts_set_step_impl(ctx.h, b"cluster-3") != 0
    assert ctx.lib.lfts_set_step_impl(ctx.h, b"generic") == 0
    ctx.close()
