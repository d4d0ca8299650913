"""Langevin steps of boxes whose contour sweeps are cluster launches: the saddle loop as a
conditional node of the step's graph, with those launches in its body, gives what the
same loop driven from the host gives (as test_lfts_gpu for the cubic kernels)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _params(nx, chain, n):
    return {
        "nx": list(nx), "lx": [4.0, 3.6, 3.2][3 - len(nx):], "chain_model": chain, "ds": 1 / n,
        "segment_lengths": {"A": 1.0, "B": 1.0}, "chi_n": {"A,B": 17.0},
        "distinct_polymers": [{"volume_fraction": 1.0, "blocks": [{"type": "A", "length": 0.5}, {"type": "B", "length": 0.5}]}],
        "langevin": {"dt": 0.8, "nbar": 100}, "saddle": {"max_iter": 100, "tolerance": 1e-4},
        "am": {"max_hist": 20, "start_error": 5e-1, "mix_min": 0.01, "mix_init": 0.01},
    }


@pytest.mark.parametrize("platform", ["cuda", "cuda-fp32"])
@pytest.mark.parametrize("chain", ["continuous", "discrete"])
@pytest.mark.parametrize("nx", [(20, 18, 14), (24, 24, 24), (48, 40), (120,)], ids=lambda n: "x".join(map(str, n)))
def test_step_graph_equals_the_host_loop(nx, chain, platform):
    from langevinfts_b200.capi import Context, check
    from langevinfts_b200.lfts import BatchedLFTS
    seeds = [41, 42]
    prec = 8 if platform == "cuda" else 4
    ctx, size = Context(nx, precision=prec), C.c_int()
    check(ctx.lib.lfts_sweep_size(ctx.h, int(chain == "continuous"), 2 * len(seeds), C.byref(size)))
    assert size.value > 0
    ctx.close()
    runs = []
    for host, graph in ((True, False), (False, True)):
        sim = BatchedLFTS(_params(nx, chain, 20), seeds, platform=platform)
        sim.engine.set_host_control(host)
        sim.engine.set_step_graph(graph)
        rng = np.random.Generator(np.random.PCG64(5))
        st = sim.start([{t: rng.normal(0.0, 1.0, sim.M) for t in ("A", "B")} for _ in seeds])
        hist = [(list(st["iterations"]), sim.fields())]
        for _ in range(2):
            st = sim.step()
            assert not any(st["failed"])
            hist.append((list(st["iterations"]), sim.fields()))
        runs.append(hist)
    # one and the same kernels in both forms: the host test's tolerance in FP64, where only
    # the control's sums differ; FP32 propagators round those differences up to 2^-24 a sum
    tol = 1e-12 if prec == 8 else 1e-5
    for (ih, wh), (idv, wd) in zip(*runs):
        assert ih == idv
        assert np.max(np.abs(wd - wh)) <= tol * np.max(np.abs(wh))
