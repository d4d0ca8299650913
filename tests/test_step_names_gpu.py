"""Names of step implementations: what is set is what is reported, anything but the exact
names is refused, and "default" brings back the rule of a new context."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _name(ctx):
    from langevinfts_b200.capi import check
    buf = C.create_string_buffer(64)
    check(ctx.lib.lfts_step_impl(ctx.h, buf, 64))
    return buf.value.decode()


def _sizes(ctx):
    from langevinfts_b200.capi import check
    out, size = [], C.c_int()
    for cont in (0, 1):
        for nj in (1, 2, 16):
            check(ctx.lib.lfts_sweep_size(ctx.h, cont, nj, C.byref(size)))
            out.append(size.value)
    return out


@pytest.mark.parametrize("nx,family", [((1, 84, 48), "generic"), ((33, 40, 12), "generic"), ((32, 32, 32), "cubic"), ((64, 64, 64), "register-64"), ((96, 96, 96), "register-96")],
                         ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v)))
def test_names(nx, family):
    from langevinfts_b200.capi import Context
    ctx = Context(nx)
    set_ = lambda n: ctx.lib.lfts_set_step_impl(ctx.h, n.encode())
    assert _name(ctx) == family
    default = _sizes(ctx)
    for bad in ("cluster-0", "cluster-x", "cluster-", "cluster-16x", "cluster-3", "cluster-08", "cluster-32", "cluster--1", "cubic ", "none", ""):
        assert set_(bad) != 0, bad
        assert _name(ctx) == family and _sizes(ctx) == default
    accepted = 0
    for n in (1, 2, 4, 8, 16):
        if set_(f"cluster-{n}") == 0:
            accepted += 1
            assert _name(ctx) == f"cluster-{n}"
            assert set(_sizes(ctx)) <= {0, n} and n in _sizes(ctx)
    if nx == (1, 84, 48):
        assert accepted == 5  # the whole box fits one CTA's shared memory
    assert set_(family) == 0 and _name(ctx) == family and set(_sizes(ctx)) == {0}
    assert set_("default") == 0 and _name(ctx) == family and _sizes(ctx) == default
    ctx.close()


def test_small_boxes_sweep_in_clusters_by_default():
    from langevinfts_b200.capi import Context
    for nx in ((1, 84, 48), (1, 1, 256), (20, 18, 14)):
        ctx = Context(nx)
        assert all(s > 0 for s in _sizes(ctx)), nx
        ctx.close()
