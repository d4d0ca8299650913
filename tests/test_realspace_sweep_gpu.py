"""The tiled real-space sweeps at the edges of their tiles: fewer lines than a
tile, one line more, axes of two points (the fewest a box may have) with every wall,
and along each axis an extent above 361, where the tile has 16 lines instead of 32,
with line counts that 16 does not divide.  Against the numpy restatement, to round-off
per step."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALLS = {"periodic": 0, "reflecting": 1, "absorbing": 2}
CASES = [([5, 4, 3], ["periodic"] * 6), ([3, 11, 33], ["periodic", "periodic", "reflecting", "absorbing", "periodic", "periodic"]),
         ([40, 6, 7], ["absorbing", "reflecting", "periodic", "periodic", "reflecting", "reflecting"]),
         ([33, 3], ["periodic"] * 4), ([12, 340], ["periodic", "periodic", "absorbing", "absorbing"]), ([350, 5], ["reflecting"] * 4),
         ([17], ["periodic"] * 2), ([700], ["reflecting", "absorbing"]), ([4, 3, 360], ["periodic"] * 6)]
P, R, A = ["periodic"] * 2, ["reflecting", "absorbing"], ["absorbing", "reflecting"]
CASES += [([361, 17], P + R), ([363, 17], P + R), ([370, 19], R + P), ([19, 370], P + A), ([4, 5, 370], P + R + A), ([370, 3, 7], R + P + P),
          ([3, 370, 6], A + R + P), ([500], P)]
CASES += [([2], P), ([2], R), ([2, 2], P + A), ([2, 33], R + P), ([2, 2, 2], P + R + A), ([5, 2, 3], A + P + R), ([3, 17, 2], P + P + P)]


@pytest.mark.parametrize("nx,bc", CASES, ids=lambda v: "x".join(map(str, v)) if isinstance(v[0], int) else v[-1])
def test_sweeps_match_the_restatement(nx, bc):
    from langevinfts_b200.capi import Context, StepJob, check
    from oracle import lfts_oracle as orc
    dim, lx, ds, njobs, nsteps = len(nx), [3.0 + 0.3 * d for d in range(len(nx))], 0.02, 2, 2
    ctx = Context(nx)
    M = ctx.M
    rng = np.random.default_rng(sum(nx))
    tab = np.zeros(ctx.lib.lfts_realspace_table_size(ctx.h))
    dx = (C.c_double * dim)(*[l / n for l, n in zip(lx, nx)])
    codes = (C.c_int * (2 * dim))(*[WALLS[b] for b in bc])
    check(ctx.lib.lfts_realspace_tables(ctx.h, 1.3, ds, dim, dx, codes, tab.ctypes.data))
    tabd, jobs, w, q0 = ctx.upload(tab), (StepJob * njobs)(), [], []
    for j in range(njobs):
        w.append(rng.normal(0.0, 1.0, M))
        q0.append(1.0 + 0.3 * rng.random(M))
        fac = ctx.malloc(M * 8)
        check(ctx.lib.lfts_field_factors(ctx.h, ctx.upload(w[j]), -ds / 4, fac))
        q = ctx.malloc((nsteps + 1) * M * 8)
        ctx.h2d(q, q0[j])
        jobs[j] = StepJob(q, M, q + M * 8, M, fac, tabd, tabd, ctx.malloc(2 * M * 8))
    jp = ctx.upload(np.frombuffer(jobs, dtype=np.uint8))
    for s in range(nsteps):
        check(ctx.lib.lfts_step_realspace(ctx.h, jp, njobs, s, dim))
    for j in range(njobs):
        got = ctx.d2h(jobs[j].in_, (nsteps + 1, M), np.float64)
        ref, e = q0[j], np.exp(-w[j] * ds / 2)
        for s in range(nsteps):
            ref = orc.step_realspace(nx, lx, ref, e, 1.3, ds, bc)
            assert np.max(np.abs(got[s + 1] - ref)) <= 1e-12 * (s + 1) * np.max(np.abs(ref)), (j, s)
    ctx.close()
