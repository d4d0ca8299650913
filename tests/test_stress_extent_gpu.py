"""Stress where the x-tile of the any-extent kernel meets the shared-memory limit.

848 rows of a 2D box in FP64: a tile of eight columns fills a block's shared memory
to within the bytes that the kernel's own reduction scratch takes; longer axes
need the next narrower tile, 440 rows the wider one.  The tolerance is the stress
test's of the other grids."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [(1, 848, 12), (1, 440, 10), (1, 896, 7), (848, 1, 9), (700, 2, 3)], ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("prec", [8, 4], ids=["fp64", "fp32"])
def test_stress_of_long_axes(nx, prec):
    from langevinfts_b200.capi import Context, StressJob, check
    from oracle import lfts_oracle as orc
    dt = np.float64 if prec == 8 else np.float32
    lx, nj = [3.0, 2.6, 3.4], 3
    ctx = Context(nx, precision=prec)
    M, Mc = ctx.M, ctx.Mc
    rng = np.random.default_rng(sum(nx))
    g = orc.Grid(nx, lx)
    q1, q2 = rng.random((nj, M)).astype(dt), rng.random((nj, M)).astype(dt)
    p1, p2 = ctx.upload(q1), ctx.upload(q2)
    basis = ctx.malloc(3 * Mc * 8)
    check(ctx.lib.lfts_fourier_basis(ctx.h, (C.c_double * 3)(*lx), basis))
    jobs = (StressJob * nj)(*[StressJob(p1 + j * M * prec, p2 + j * M * prec, None, 0.5 + j) for j in range(nj)])
    out = ctx.malloc(3 * nj * 8)
    check(ctx.lib.lfts_stress(ctx.h, ctx.upload(np.frombuffer(jobs, dtype=np.uint8)), nj, basis, ctx.malloc(2 * 2 * Mc * 2 * prec), 2, out))
    got = ctx.d2h(out, (nj, 3), np.float64)
    bas = orc.fourier_basis(nx, lx)
    for j in range(nj):
        ref = orc.segment_stress(g, q1[j].astype(np.float64), q2[j].astype(np.float64), 1.0, bas, None) * (0.5 + j)
        # FP32: the products of two spectra carry the transforms' round-off (2e-5 of a step)
        tol = 1e-9 if prec == 8 else 4e-5
        assert np.all(np.abs(got[j] - ref) <= tol * np.max(np.abs(ref))), (j, got[j], ref)
    ctx.close()
