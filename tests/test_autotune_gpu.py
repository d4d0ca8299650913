"""The autotuner times what a solver runs: sweeps, with seams between their steps and as
cluster launches where the rule has them, counted by the kernels it enqueues."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

STEPS, WARM, SETUP = 8, 2, 2  # steps a sweep, untimed sweeps, kernels that make factors and tables


@pytest.mark.parametrize("prec", [8, 4], ids=["fp64", "fp32"])
@pytest.mark.parametrize("nx", [(1, 84, 48), (31, 49, 23), (48, 48, 48)], ids=lambda n: "x".join(map(str, n)))
def test_candidates_are_timed_as_sweeps(nx, prec):
    from langevinfts_b200.capi import Context, check
    ctx, reps = Context(nx, precision=prec), 3
    size = C.c_int()
    check(ctx.lib.lfts_sweep_size(ctx.h, 1, 2, C.byref(size)))
    seams = 1 + 4 * STEPS  # first pass, then three and the seam (or the last) a step
    before = ctx.lib.lfts_ctx_launches(ctx.h)
    report = C.create_string_buffer(512)
    check(ctx.lib.lfts_autotune(ctx.h, 2, reps, report, 512))
    names = [c.split()[0] for c in report.value.decode().split(" -> ")[0].split("; ")]
    assert names == (["cubic", "generic"] if nx[0] == 48 else ["generic"])
    sweeps = {"cubic": seams, "generic": 1 if size.value else seams}
    assert ctx.lib.lfts_ctx_launches(ctx.h) - before == SETUP + (WARM + reps) * sum(sweeps[n] for n in names)
    ctx.close()


def test_a_named_choice_gives_way():
    from langevinfts_b200.capi import Context, check
    ctx, size = Context((1, 84, 48)), C.c_int()
    check(ctx.lib.lfts_set_step_impl(ctx.h, b"generic"))
    check(ctx.lib.lfts_sweep_size(ctx.h, 1, 2, C.byref(size)))
    assert size.value == 0
    check(ctx.lib.lfts_autotune(ctx.h, 2, 2, None, 0))
    check(ctx.lib.lfts_sweep_size(ctx.h, 1, 2, C.byref(size)))
    assert size.value > 0
    ctx.close()
