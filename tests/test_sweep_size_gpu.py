"""A sweep's launch shape does not depend on earlier calls.

Cluster sizes differ in how planes pair up, hence in the last bits: a solver that
captures its propagation in two graphs must get the same kernels in both, and the
first call on a context must give what the tenth gives."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# the number of resident clusters lies next to these numbers of jobs
CASES = [((24, 24, 24), 8), ((24, 24, 24), 16), ((1, 84, 48), 32), ((20, 18, 14), 32), ((1, 128, 120), 16), ((40, 36, 30), 8)]


def _sweep(ctx, nx, nj, discrete, prec, nsteps=2):
    from langevinfts_b200.capi import StepJob, check
    dt = np.float64 if prec == 8 else np.float32
    rng = np.random.default_rng(sum(nx) + nj)
    bond, half = ctx.malloc(ctx.Mc * prec), ctx.malloc(ctx.Mc * prec)
    check(ctx.lib.lfts_bond_tables(ctx.h, 1.0, 0.02, (C.c_double * 3)(3.0, 2.6, 3.4), bond, half))
    jobs = (StepJob * nj)()
    for j in range(nj):
        fac = ctx.upload(np.exp(-0.005 * rng.normal(0.0, 1.0, ctx.M)).astype(dt))
        q = ctx.malloc((nsteps + 1) * ctx.M * prec)
        ctx.h2d(q, np.exp(rng.normal(0.0, 0.3, ctx.M)).astype(dt))
        jobs[j] = StepJob(q, ctx.M, q + ctx.M * prec, ctx.M, fac, bond, half, ctx.malloc(2 * ctx.Mc * 2 * prec))
    jp = ctx.upload(np.frombuffer(jobs, dtype=np.uint8))

    def run():
        check(ctx.lib.lfts_sweep_discrete(ctx.h, jp, nj, 0, nsteps, 0, 1) if discrete
              else ctx.lib.lfts_sweep_continuous(ctx.h, jp, nj, 0, nsteps))

    def read():
        return np.array([ctx.d2h(jobs[j].in_, (nsteps + 1, ctx.M), dt) for j in range(nj)])
    return run, read


@pytest.mark.parametrize("discrete", [False, True], ids=["continuous", "discrete"])
@pytest.mark.parametrize("prec", [8, 4], ids=["fp64", "fp32"])
@pytest.mark.parametrize("nx,nj", CASES, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_first_and_later_sweeps_agree_bit_for_bit(nx, nj, prec, discrete):
    from langevinfts_b200.capi import Context
    ctx = Context(nx, precision=prec)
    run, read = _sweep(ctx, nx, nj, discrete, prec)
    run()
    first = read()
    for _ in range(3):
        run()
        assert np.array_equal(read(), first)
    ctx.close()


def test_two_captures_of_one_sweep_agree_bit_for_bit():
    from langevinfts_b200.capi import Context, check
    nx, nj = (24, 24, 24), 8
    ctx = Context(nx)
    run, read = _sweep(ctx, nx, nj, False, 8)
    out = []
    for _ in range(2):
        graph = C.c_void_p()
        check(ctx.lib.lfts_graph_begin(ctx.h))
        run()
        check(ctx.lib.lfts_graph_end(ctx.h, C.byref(graph)))
        check(ctx.lib.lfts_graph_launch(ctx.h, graph))
        out.append(read())
        check(ctx.lib.lfts_graph_destroy(graph))
    assert np.array_equal(out[0], out[1])
    ctx.close()


@pytest.mark.parametrize("nx,nj", CASES, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_size_is_the_same_in_any_order_of_asking(nx, nj):
    from langevinfts_b200.capi import Context, check
    counts = [1, 2, 4, nj - 1, nj, nj + 1, 64, 256]
    seen = {}
    for order in (counts, counts[::-1], counts + counts):
        ctx = Context(nx)
        for n in order:
            for cont in (0, 1):
                size = C.c_int(-1)
                check(ctx.lib.lfts_sweep_size(ctx.h, cont, n, C.byref(size)))
                assert seen.setdefault((n, cont), size.value) == size.value
        ctx.close()
    assert seen[1, 1] in (0, 1, 2, 4, 8, 16)
