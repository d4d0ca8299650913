"""Any-extent step kernels and cluster sweeps against the numpy oracle.

Extents at which they can go wrong: one plane, one row, one column and one
point along an axis, radices of every kind (2..13, 16, primes above 13 alone
and twice), odd and even extents (unpaired planes, Nyquist), columns and planes
that do not divide among the CTAs, every cluster size the grid fits (and there is one
for every small grid), extents whose plan needs three register radices (75, 98, 308),
planes stacked in a CTA with a remainder, and planes that only the
run-time-radix kernels hold.  The tolerance is the step tests' one: round-off of three
transforms a step.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(1, 1, 24), (1, 1, 289), (1, 12, 10), (1, 84, 48), (1, 37, 9), (6, 1, 9), (5, 4, 3), (2, 2, 2), (16, 7, 2), (13, 11, 8),
         (17, 5, 4), (9, 10, 34), (31, 49, 23), (20, 18, 14), (33, 26, 25), (80, 60, 48), (3, 100, 110),
         (1, 75, 10), (1, 6, 98), (1, 1, 308), (1, 338, 4), (75, 4, 6), (4, 98, 5)]


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
    nsteps, accepted = 3, set()
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
            accepted.add(impl)
        ctx.close()
    assert "generic" in accepted
    if np.prod(nx) <= 4032:  # one of the sizes holds the slabs and columns of so few points
        assert len(accepted) > 1, accepted


# Planes share a CTA when the launch still has two CTAs for each of 148 SMs: two planes (or
# pairs) from ceil(units / 2) * jobs >= 296 on, four from half as many.  Units are planes
# in the two-branch kernels and pairs in the others; these leave a remainder in both.
STACKED = [((1, 81, 7), 24), ((13, 5, 4), 150), ((27, 3, 10), 80)]


@pytest.mark.parametrize("discrete", [False, True], ids=["continuous", "discrete"])
@pytest.mark.parametrize("prec", [8, 4], ids=["fp64", "fp32"])
@pytest.mark.parametrize("nx,njobs", STACKED, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_stacked_planes_match_the_oracle(nx, njobs, prec, discrete):
    from langevinfts_b200.capi import check
    nsteps = 2
    ctx, jobs, jp, q0, w, tab, lx, ds = _setup(nx, prec, njobs, nsteps)
    check(ctx.lib.lfts_set_step_impl(ctx.h, b"generic"))
    if discrete:
        check(ctx.lib.lfts_sweep_discrete(ctx.h, jp, njobs, 0, nsteps, 0, 1))
    else:
        check(ctx.lib.lfts_sweep_continuous(ctx.h, jp, njobs, 0, nsteps))
    _check(ctx, jobs, q0, w, tab, lx, nx, ds, prec, nsteps, discrete)
    ctx.close()


# FP64 planes above about 14 500 points, which the any-extent kernels cannot hold
LARGE = [(3, 128, 130), (2, 126, 143), (5, 121, 122), (4, 128, 128)]


@pytest.mark.parametrize("discrete", [False, True], ids=["continuous", "discrete"])
@pytest.mark.parametrize("nx", LARGE, ids=lambda n: "x".join(map(str, n)))
def test_large_planes_match_the_oracle(nx, discrete):
    from langevinfts_b200.capi import check
    nsteps, njobs = 2, 2
    ctx, jobs, jp, q0, w, tab, lx, ds = _setup(nx, 8, njobs, nsteps)
    assert ctx.lib.lfts_set_step_impl(ctx.h, b"cluster-16") != 0
    if discrete:
        check(ctx.lib.lfts_sweep_discrete(ctx.h, jp, njobs, 0, nsteps, 0, 1))
    else:
        check(ctx.lib.lfts_sweep_continuous(ctx.h, jp, njobs, 0, nsteps))
    _check(ctx, jobs, q0, w, tab, lx, nx, ds, 8, nsteps, discrete)
    ctx.close()


@pytest.mark.parametrize("nx", LARGE, ids=lambda n: "x".join(map(str, n)))
def test_stress_and_transform_of_large_planes(nx):
    from langevinfts_b200.capi import Context, StepJob, StressJob, check
    from oracle import lfts_oracle as orc
    lx, nj = [3.0, 2.6, 3.4], 3
    ctx = Context(nx)
    M, Mc = ctx.M, ctx.Mc
    rng = np.random.default_rng(sum(nx))
    q1, q2 = rng.random((nj, M)), rng.random((nj, M))
    p1, p2, spec = ctx.upload(q1), ctx.upload(q2), ctx.malloc(2 * 2 * Mc * 16)
    basis, out = ctx.malloc(3 * Mc * 8), ctx.malloc(3 * nj * 8)
    check(ctx.lib.lfts_fourier_basis(ctx.h, (C.c_double * 3)(*lx), basis))
    jobs = (StressJob * nj)(*[StressJob(p1 + j * M * 8, p2 + j * M * 8, None, 1.0) for j in range(nj)])
    check(ctx.lib.lfts_stress(ctx.h, ctx.upload(np.frombuffer(jobs, dtype=np.uint8)), nj, basis, spec, 2, out))
    got, bas, g = ctx.d2h(out, (nj, 3), np.float64), orc.fourier_basis(nx, lx), orc.Grid(nx, lx)
    for j in range(nj):
        ref = orc.segment_stress(g, q1[j], q2[j], 1.0, bas, None)
        assert np.allclose(got[j], ref, rtol=1e-11, atol=1e-9 * np.max(np.abs(ref))), (j, got[j], ref)
    field = (StepJob * 1)(StepJob(p1, 0, p1, 0, None, None, None, spec))
    check(ctx.lib.lfts_fft_forward(ctx.h, ctx.upload(np.frombuffer(field, dtype=np.uint8)), 1))
    ref = np.fft.rfftn(q1[0].reshape(nx)).reshape(-1)
    assert np.max(np.abs(ctx.d2h(spec, (Mc,), np.complex128) - ref)) <= 1e-12 * np.max(np.abs(ref))
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
