"""lfts_bond_tables and lfts_fourier_basis refuse host memory before any launch, and write
device and pinned memory."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_host_memory_is_refused_and_pinned_memory_taken():
    from langevinfts_b200.capi import Context, check
    nx, lx = (16, 12, 10), (C.c_double * 3)(3.0, 2.5, 2.0)
    ctx = Context(nx)
    L, Mc = ctx.lib, ctx.Mc
    host = np.zeros(3 * Mc)
    dev = ctx.malloc(3 * Mc * 8)
    assert L.lfts_bond_tables(ctx.h, 1.0, 0.01, lx, host.ctypes.data, dev) != 0
    assert L.lfts_bond_tables(ctx.h, 1.0, 0.01, lx, dev, host.ctypes.data) != 0
    assert L.lfts_fourier_basis(ctx.h, lx, host.ctypes.data) != 0
    assert not host.any()
    ctx.sync()  # nothing was launched that could fail later
    pinned = C.c_void_p()
    check(L.lfts_malloc_host(ctx.h, C.byref(pinned), 3 * Mc * 8))
    check(L.lfts_fourier_basis(ctx.h, lx, dev))
    check(L.lfts_fourier_basis(ctx.h, lx, pinned))
    got = np.ctypeslib.as_array((C.c_double * (3 * Mc)).from_address(pinned.value)).copy()
    assert np.array_equal(got, ctx.d2h(dev, (3 * Mc,), np.float64))
    check(L.lfts_free_host(ctx.h, pinned))
    ctx.close()
