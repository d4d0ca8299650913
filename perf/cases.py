"""Performance cases: the work users of langevinfts_b200 have it do.

Kinds of cases, each through the entry points a user's program calls:

  statistics  one saddle-point or SCFT iteration driven from numpy, the calls
              of the reference's drivers: compute_propagators,
              compute_concentrations, total concentrations (and, where the box
              relaxes, the stress), 1D to 3D, continuous and discrete chains,
              linear and branched molecules, FP64 and FP32 propagators
  film        the same through the real-space solver, walls on the last axis
  scft        one iteration of the device-resident SCFT loop with box relaxation
  lfts        one Langevin step of a batch of replicas, saddle search included
  unet        inference of the learned saddle-point start's network
  conv        forward and backward of one of its convolution layers

A case is a dict of plain numbers and texts.  listed() gives the fixed ones,
draw(rng) one more of the same ranges, prepare/run one pass, work the bytes and
operations a pass cannot do without, and exact the same results by plain torch
in 64 bits.
"""
import math

import numpy as np
import torch

# Molecules: (volume fraction, [(monomer type, share of a unit chain, node v, node u), ...]);
# shares are sixtieths so that every contour length used below divides them.
MOLECULES = {
    # the symmetric AB diblock of the L-FTS studies and of the smallest test system
    "diblock": ([(1.0, [("A", 30, 0, 1), ("B", 30, 1, 2)])], {"A": 1.0, "B": 1.0}),
    # an ABA triblock with unequal statistical segment lengths
    "triblock": ([(1.0, [("A", 12, 0, 1), ("B", 36, 1, 2), ("A", 12, 2, 3)])], {"A": 1.2, "B": 0.9}),
    # a three-arm star, a comb with eight side chains and a homopolymer
    "mixture": ([(0.5, [("A", 20, 0, 1), ("B", 20, 0, 2), ("C", 20, 0, 3)]),
                 (0.3, [("B", 5, i, i + 1) for i in range(8)] + [("A", 6, i, 8 + i) for i in range(1, 9)]),
                 (0.2, [("A", 30, 0, 1)])], {"A": 1.0, "B": 1.0, "C": 1.0}),
}

# Convolution layers of the 24-channel network (padded channels in, out, level):
# network input, first level, pooled levels, and the concatenations on the way up.
CONV_LAYERS = [(16, 32, 0), (32, 32, 0), (32, 48, 1), (48, 48, 1), (48, 96, 2), (96, 96, 2), (144, 48, 1), (80, 32, 0)]


def listed():
    return [
        # 2D SCFT of a cylinder phase on a rectangular cell with stress: the smallest calls, all latency
        {"name": "plane_2d", "kind": "statistics", "nx": 84, "ny": 48, "nz": 0, "box": 4.0, "model": "continuous",
         "molecule": "triblock", "segments": 60, "platform": "cuda", "stress": True},
        # the small 3D system of single-chain studies, one saddle-point iteration
        {"name": "diblock_32", "kind": "statistics", "nx": 32, "ny": 32, "nz": 32, "box": 4.0, "model": "continuous",
         "molecule": "diblock", "segments": 120, "platform": "cuda", "stress": False},
        # three different odd extents with large prime factors: nothing divides the tiles
        {"name": "ragged_31", "kind": "statistics", "nx": 31, "ny": 49, "nz": 23, "box": 4.0, "model": "continuous",
         "molecule": "diblock", "segments": 60, "platform": "cuda", "stress": True},
        # a non-cubic cell as hexagonal and orthorhombic phases need, with stress
        {"name": "ortho_80", "kind": "statistics", "nx": 80, "ny": 60, "nz": 48, "box": 5.0, "model": "continuous",
         "molecule": "triblock", "segments": 60, "platform": "cuda", "stress": True},
        # discrete chains: stars, combs and a homopolymer mixed, many short propagators and junctions
        {"name": "mixture_48", "kind": "statistics", "nx": 48, "ny": 48, "nz": 48, "box": 5.0, "model": "discrete",
         "molecule": "mixture", "segments": 60, "platform": "cuda", "stress": True},
        # a film between a reflecting and an absorbing wall: the real-space solver
        {"name": "film_64", "kind": "film", "nx": 48, "ny": 48, "nz": 64, "box": 4.0, "molecule": "diblock", "segments": 60},
        # 3D SCFT on the device, the box relaxing: the ordinary research calculation
        {"name": "scft_64", "kind": "scft", "nx": 64, "ny": 64, "nz": 64, "box": 3.6, "segments": 100},
        # many small replicas in single precision: a parameter sweep
        {"name": "lfts_32_fp32", "kind": "lfts", "nx": 32, "ny": 32, "nz": 32, "box": 5.0, "replicas": 16,
         "platform": "cuda-fp32"},
        # the L-FTS study system in double precision, a few replicas at a time
        {"name": "lfts_64", "kind": "lfts", "nx": 64, "ny": 64, "nz": 64, "box": 7.3, "replicas": 6, "platform": "cuda"},
        # the large study system in single precision
        {"name": "lfts_96_fp32", "kind": "lfts", "nx": 96, "ny": 96, "nz": 96, "box": 8.0, "replicas": 4,
         "platform": "cuda-fp32"},
        # the learned start's prediction for a batch of replicas
        {"name": "unet_64", "kind": "unet", "nx": 64, "batch": 4},
        # its training: one of the widest layers, forward, input gradient and weight gradient
        {"name": "conv_80_32", "kind": "conv", "nx": 64, "batch": 4, "cin": 80, "cout": 32},
    ]


def _log_int(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def _extent(rng, lo, hi):
    """A grid extent a transform can have: even and smooth mostly, now and then odd or with a larger prime."""
    while True:
        n = _log_int(rng, lo, hi, 1 if rng.random() < 0.25 else 4)
        m = n
        for p in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31):
            while m % p == 0:
                m //= p
        if m == 1:
            return n


def draw(rng):
    kind = rng.choice(["statistics"] * 5 + ["film", "scft", "lfts", "lfts", "unet", "conv"])
    if kind == "statistics":
        dim = rng.choice([1, 2, 3, 3, 3])
        lo, hi = {1: (32, 512), 2: (24, 128), 3: (12, 72)}[dim]
        n = [_extent(rng, lo, hi) for _ in range(dim)]
        if dim == 3 and rng.random() < 0.3:
            n = [rng.choice([16, 32, 48, 64])] * 3
        molecule = rng.choice(["diblock", "triblock", "mixture"])
        model = "discrete" if molecule == "mixture" else rng.choice(["continuous", "continuous", "discrete"])
        platform = rng.choice(["cuda", "cuda", "cuda-fp32"])
        return {"kind": kind, "nx": n[0], "ny": n[1] if dim > 1 else 0, "nz": n[2] if dim > 2 else 0,
                "box": round(rng.uniform(3.0, 6.0), 2), "model": model, "molecule": molecule,
                "segments": 60 if molecule != "diblock" else rng.choice([60, 120]), "platform": platform,
                "stress": platform == "cuda" and rng.random() < 0.6}
    if kind == "film":
        return {"kind": kind, "nx": _log_int(rng, 12, 56), "ny": _log_int(rng, 12, 56), "nz": _log_int(rng, 16, 72),
                "box": round(rng.uniform(3.0, 6.0), 2), "molecule": rng.choice(["diblock", "triblock"]), "segments": 60}
    if kind == "scft":
        n = [rng.choice([32, 48, 64])] * 3 if rng.random() < 0.5 else [_extent(rng, 24, 64) for _ in range(3)]
        return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "box": round(rng.uniform(3.4, 4.4), 2), "segments": 100}
    if kind == "lfts":
        n = rng.choice([16, 24, 32, 40, 48, 64])
        most = max(1, int(6 * 64 ** 3 / n ** 3))
        return {"kind": kind, "nx": n, "ny": n, "nz": n, "box": round(rng.uniform(4.0, 7.5), 2),
                "replicas": _log_int(rng, 1, min(most, 32)), "platform": rng.choice(["cuda", "cuda-fp32"])}
    if kind == "unet":
        return {"kind": kind, "nx": _log_int(rng, 16, 64, 4), "batch": rng.randint(1, 4)}
    cin, cout, level = rng.choice(CONV_LAYERS)
    return {"kind": kind, "nx": _log_int(rng, 16, 64, 8) >> level, "batch": rng.randint(1, 4), "cin": cin, "cout": cout}


# ---------------------------------------------------------------- descriptions
def _grid(case):
    return [case[k] for k in ("nx", "ny", "nz") if case.get(k, 0)]


def _lengths(case):
    """Box lengths: the first axis has case["box"], the others the same up to 12 % (a cell in use is rarely cubic
    when its grid is not)."""
    n = _grid(case)
    if len(set(n)) == 1:
        return [case["box"]] * len(n)
    return [round(case["box"] * (1.0 - 0.06 * d), 4) for d in range(len(n))]


def _structure(shape):
    """A periodic composition pattern of unit amplitude (gyroid-like in 3D, a lamella in 1D)."""
    x = np.meshgrid(*[np.arange(n) * 2 * np.pi / n for n in shape], indexing="ij")
    d = len(shape)
    if d == 1:
        return np.cos(x[0]).reshape(-1)
    return sum(np.sin(x[i]) * np.cos(x[(i + 1) % d]) for i in range(d)).reshape(-1) / d


def _fields(case, seed, types):
    """Monomer fields as a running calculation has them: a composition pattern and noise."""
    shape = _grid(case)
    rng = np.random.Generator(np.random.PCG64(seed))
    g = _structure(shape)
    amp = {"A": 2.0, "B": -2.0, "C": 0.5}
    return {t: amp[t] * g + rng.normal(0.0, 1.0, g.size) for t in types}


def _boundary(case):
    return ["periodic"] * (2 * len(_grid(case)) - 2) + ["reflecting", "absorbing"]


def _scft_params(case):
    """The asymmetric diblock with conformational asymmetry whose box relaxes."""
    eps, f = 1.2, 0.36
    den = eps * eps * f + (1 - f)
    return {"nx": _grid(case), "lx": _lengths(case), "chain_model": "continuous", "ds": 1.0 / case["segments"],
            "segment_lengths": {"A": (eps * eps / den) ** 0.5, "B": (1.0 / den) ** 0.5}, "chi_n": {"A,B": 20.0},
            "distinct_polymers": [{"volume_fraction": 1.0, "blocks": [{"type": "A", "length": f},
                                                                      {"type": "B", "length": 1 - f}]}],
            "box_is_altering": True, "scale_stress": 1.0,
            "optimizer": {"name": "am", "max_hist": 20, "start_error": 1e-2, "mix_min": 0.1, "mix_init": 0.1}}


def _scft_fields(case, seed):
    g = _structure(_grid(case)) * len(_grid(case))
    rng = np.random.Generator(np.random.PCG64(seed))
    return {"A": 6.0 * g + 0.1 * rng.normal(0, 1, g.size), "B": -6.0 * g + 0.1 * rng.normal(0, 1, g.size)}


def _lfts_params(case):
    return {"nx": _grid(case), "lx": [case["box"]] * 3, "chain_model": "continuous", "ds": 1 / 90,
            "segment_lengths": {"A": 1.0, "B": 1.0}, "chi_n": {"A,B": 17.0},
            "distinct_polymers": [{"volume_fraction": 1.0, "blocks": [{"type": "A", "length": 0.5},
                                                                      {"type": "B", "length": 0.5}]}],
            "langevin": {"dt": 0.8, "nbar": 100}, "saddle": {"max_iter": 100, "tolerance": 1e-4},
            "am": {"max_hist": 20, "start_error": 5e-1, "mix_min": 0.01, "mix_init": 0.01}}


def _lfts_seeds(case, seed):
    return [1000 * seed + r for r in range(case["replicas"])]


def _lfts_initial(seed, M):
    rng = np.random.Generator(np.random.PCG64(seed))
    return {"A": rng.normal(0.0, 1.0, M), "B": rng.normal(0.0, 1.0, M)}


def _unet(seed):
    """The learned start's network with its initial weights, but for the last layer, which starts at zero and is small
    after training."""
    from langevinfts_b200.learned import UNet3D
    torch.manual_seed(seed)
    net = UNet3D(cin=3, cout=1, base=24)
    with torch.no_grad():
        net.out.weight.normal_(0.0, 0.2)
        net.out.bias.normal_(0.0, 0.05)
    return net


def _unet_input(case, seed):
    g = torch.Generator().manual_seed(seed)
    n = case["nx"]
    return torch.randn([case["batch"], 3, n, n, n], generator=g).cuda()


def _conv_data(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, ci, co = case["nx"], case["cin"], case["cout"]
    shape = [case["batch"], n, n, n]
    x = torch.randn(shape + [ci], generator=g, device="cuda").clamp_(min=0).to(torch.bfloat16)  # after a ReLU
    gy = (torch.randn(shape + [co], generator=g, device="cuda") * 1e-2).to(torch.bfloat16)
    w = (torch.randn([co, ci, 3, 3, 3], generator=g, device="cuda") * (2.0 / (27 * ci)) ** 0.5).to(torch.bfloat16).float()
    b = torch.randn([co], generator=g, device="cuda") * 0.1
    return x, gy, w, b


# ---------------------------------------------------------------- prepare and run
class _DeviceView:
    """Device memory of the engine as a CUDA array, without a copy; an array made from it keeps the owner alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8", "data": (int(ptr), False), "version": 3,
                                         "strides": None}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("statistics", "film"):
        from langevinfts_b200 import langevinfts as L
        polymers, bonds = MOLECULES[case["molecule"]]
        ds = 1.0 / case["segments"]
        factory = L.PlatformSelector.create_factory(case.get("platform", "cuda"), False)
        if kind == "film":
            box = factory.create_computation_box(_grid(case), _lengths(case), _boundary(case))
        else:
            box = factory.create_computation_box(_grid(case), _lengths(case))
        molecules = factory.create_molecules_information(case.get("model", "continuous"), ds, bonds)
        for fraction, blocks in polymers:
            molecules.add_polymer(fraction, [[t, share / 60, v, u] for t, share, v, u in blocks])
        analyzer = factory.create_propagator_analyzer(molecules, True)
        make = factory.create_realspace_solver if kind == "film" else factory.create_pseudospectral_solver
        solver = make(box, molecules, analyzer)
        return {"kind": kind, "solver": solver, "keep": (factory, box, molecules, analyzer), "types": sorted(bonds),
                "n_polymers": len(polymers),
                "record": np.float32 if case.get("platform") == "cuda-fp32" else np.float64, "w": _fields(case, seed, sorted(bonds)), "stress": case.get("stress", False)}
    if kind == "scft":
        from langevinfts_b200.scft import SCFT
        scft = SCFT(_scft_params(case))
        w = _scft_fields(case, seed)
        scft.engine.set_fields(np.array([w["A"], w["B"]]))
        scft.engine.reset()
        return {"kind": kind, "scft": scft}
    if kind == "lfts":
        from langevinfts_b200.lfts import BatchedLFTS
        seeds = _lfts_seeds(case, seed)
        sim = BatchedLFTS(_lfts_params(case), seeds, platform=case["platform"])
        sim.start([_lfts_initial(s, sim.M) for s in seeds])
        w = torch.as_tensor(_DeviceView(sim, sim.engine.w_aux_ptr(), (sim.R, sim.S, sim.M)), device="cuda")
        return {"kind": kind, "sim": sim, "w": w, "single": case["platform"] == "cuda-fp32"}
    if kind == "unet":
        from langevinfts_b200.learned import TcgenUNet
        return {"kind": kind, "net": TcgenUNet(_unet(seed).cuda()), "x": _unet_input(case, seed)}
    from langevinfts_b200.learned import pack_conv
    x, gy, w, b = _conv_data(case, seed)
    ci, co = case["cin"], case["cout"]
    conv = torch.nn.Conv3d(ci, co, 3, padding=1, padding_mode="circular").cuda()
    back = torch.nn.Conv3d(co, ci, 3, padding=1, padding_mode="circular", bias=False).cuda()
    with torch.no_grad():
        conv.weight.copy_(w)
        conv.bias.copy_(b)
        back.weight.copy_(w.flip(2, 3, 4).transpose(0, 1))  # the input gradient is a convolution with these
    return {"kind": kind, "x": x, "gy": gy, "forward": pack_conv(conv, list(range(ci)), ci),
            "backward": pack_conv(back, list(range(co)), co), "cin": ci, "cout": co}


def run(state):
    kind = state["kind"]
    if kind in ("statistics", "film"):
        solver = state["solver"]
        solver.compute_propagators(state["w"])
        solver.compute_concentrations()
        out = {"phi": [solver.get_total_concentration(t) for t in state["types"]],
               "partitions": np.array([solver.get_total_partition(p) for p in range(state["n_polymers"])], state["record"])}
        if state["stress"]:
            solver.compute_stress()
            out["stress"] = np.array(solver.get_stress())
        return out
    if kind == "scft":
        engine = state["scft"].engine
        stats = engine.evaluate()
        engine.update()
        return {"partitions": np.array(stats["partitions"]), "stress": np.array(stats["stress"]),
                "error_level": stats["error_level"], "phi": engine.get_concentrations(), "w": engine.get_fields()}
    if kind == "lfts":
        stats = state["sim"].step()
        energy = torch.tensor(stats["hamiltonian"], dtype=torch.float64)
        if state["single"]:  # single-precision runs keep single-precision records
            return {"w": state["w"].float(), "hamiltonian": energy.float()}
        return {"w": state["w"], "hamiltonian": energy}
    if kind == "unet":
        return state["net"](state["x"])
    from langevinfts_b200.capi import check, lib
    from langevinfts_b200.learned import conv3d_tcgen05
    x, gy, ci, co = state["x"], state["gy"], state["cin"], state["cout"]
    stream = torch.cuda.current_stream().cuda_stream
    y = conv3d_tcgen05(x, state["forward"], True)
    g, db = torch.empty_like(y), torch.zeros(co, device=x.device)
    check(lib().lfts_relu_grad_bf16(stream, gy.data_ptr(), y.data_ptr(), g.data_ptr(), db.data_ptr(), y.numel() // co, co, co))
    dx = conv3d_tcgen05(g, state["backward"], False)
    dw = torch.zeros(27, co, ci, device=x.device)
    b, d, h, w, _ = x.shape
    check(lib().lfts_conv3d_wgrad_bf16(stream, x.data_ptr(), g.data_ptr(), dw.data_ptr(), b, d, h, w, ci, co, 27))
    return {"y": y, "dx": dx, "dw": dw, "db": db}


# ---------------------------------------------------------------- work
def _steps(case):
    """Contour steps of all propagators of the molecules, equal arms counted once."""
    polymers, _ = MOLECULES[case["molecule"]]
    n = case["segments"]
    steps = 0
    for _, blocks in polymers:
        arms = {}
        for t, share, v, u in blocks:
            for a, b in ((v, u), (u, v)):
                arms[_arm(blocks, a, b)] = share * n // 60
        steps += sum(arms.values())
    return steps


def _arm(blocks, v, u):
    """Canonical text of the propagator from node v to node u."""
    for t, share, a, b in blocks:
        if (a, b) in ((v, u), (u, v)):
            inner = sorted(_arm(blocks, x if y == v else y, v) for s, _, x, y in blocks
                           if v in (x, y) and u not in (x, y))
            return "(" + "".join(inner) + ")" + t + str(share)
    raise KeyError((v, u))


def work(case):
    kind = case["kind"]
    if kind in ("statistics", "film", "scft", "lfts"):
        M = float(np.prod(_grid(case)))
        lg = math.log2(M)
        size = 4 if case.get("platform") == "cuda-fp32" else 8
        replicas, iterations, types = 1, 1, 2
        if kind == "lfts":
            steps, replicas, iterations = 4 * 45, case["replicas"], 40
        elif kind == "scft":
            steps = 2 * case["segments"]
        else:
            steps, types = _steps(case), len(MOLECULES[case["molecule"]][1])
        # operations of a contour step: real transforms at 2.5 M log2 M and about ten operations a point between them
        if kind == "film":
            per_step = 40.0 * M
        elif case.get("model", "continuous") == "continuous":
            per_step = 6 * 2.5 * M * lg + 20 * M
        else:
            per_step = 2 * 2.5 * M * lg + 5 * M
        points = steps * M * replicas * iterations
        flops = replicas * iterations * steps * per_step + 2 * points
        # every propagator slice is written once (the concentrations read them while they are made), fields in,
        # concentrations out
        nbytes = size * points + 8.0 * 2 * types * M * replicas * iterations
        if case.get("stress") or kind == "scft":
            flops += steps * (2.5 * M * lg + 4 * M)
        return {"bytes": nbytes, "flops": flops}
    n3 = float(case["nx"]) ** 3 * case["batch"]
    if kind == "conv":
        ci, co = case["cin"], case["cout"]
        return {"bytes": n3 * 2 * (2 * ci + 2 * co) + 4 * 27 * ci * co, "flops": 3 * 2 * 27 * n3 * ci * co}
    b = 24
    flops = 27 * (3 * b + b * b) + 27 * (2 * b * b + 4 * b * b) / 8 + 27 * (8 * b * b + 16 * b * b) / 64
    flops += 27 * (12 * b * b + 4 * b * b) / 8 + 27 * (3 * b * b + b * b) + b
    return {"bytes": n3 * 4 * (3 + 1) + 2e6, "flops": 2 * n3 * flops}


# ---------------------------------------------------------------- the same results in 64 bits
def _simpson(N):
    if N == 1:
        return [0.5, 0.5]
    if N == 3:
        return [3 / 8, 9 / 8, 9 / 8, 3 / 8]
    c = [0.0] * (N + 1)
    even = N if N % 2 == 0 else N - 3
    for i in range(0, even, 2):
        c[i] += 1 / 3
        c[i + 1] += 4 / 3
        c[i + 2] += 1 / 3
    if N % 2:
        for i, v in enumerate((3 / 8, 9 / 8, 9 / 8, 3 / 8)):
            c[N - 3 + i] += v
    return c


class _Chains:
    """Propagators, concentrations and stress of a mixture of tree molecules by torch.fft in float64."""

    def __init__(self, shape, lx, model, ds, polymers, bonds, walls=None):
        self.shape, self.lx, self.model, self.ds, self.polymers, self.bonds = list(shape), list(lx), model, ds, polymers, bonds
        self.dims = list(range(-len(shape), 0))
        self.walls = walls
        k = [torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device="cuda") * (2 * math.pi / l) for n, l in zip(shape, lx)]
        k[-1] = torch.arange(shape[-1] // 2 + 1, dtype=torch.float64, device="cuda") * (2 * math.pi / lx[-1])
        self.kk = []
        for d in range(len(shape)):
            view = [1] * len(shape)
            view[d] = -1
            self.kk.append((k[d] ** 2).reshape(view))
        k2 = sum(self.kk)
        self.bond = {t: torch.exp(-b * b * ds / 6 * k2) for t, b in bonds.items()}
        self.half = {t: torch.exp(-b * b * ds / 12 * k2) for t, b in bonds.items()}
        self.weight = torch.full([shape[-1] // 2 + 1], 2.0, dtype=torch.float64, device="cuda")
        self.weight[0] = 1.0
        if shape[-1] % 2 == 0:
            self.weight[-1] = 1.0
        if walls is not None:
            self.sweeps = {t: self._sweeps(b) for t, b in bonds.items()}

    def _conv(self, q, table):
        return torch.fft.irfftn(torch.fft.rfftn(q, dim=self.dims) * table, s=self.shape, dim=self.dims)

    def _sweeps(self, b):
        """Per axis the Crank-Nicolson operator and the inverse of one plus it, as dense matrices."""
        out = []
        for a, n in enumerate(self.shape):
            r = b * b * self.ds / (6.0 * (self.lx[a] / n) ** 2)
            m = torch.zeros(n, n, dtype=torch.float64)
            for i in range(n):
                m[i, i] += r
                for j, side in ((i - 1, 2 * a), (i + 1, 2 * a + 1)):
                    wall = self.walls[side]
                    if 0 <= j < n or wall == "periodic":
                        m[i, j % n] -= r / 2
                    elif wall == "reflecting":
                        m[i, i] -= r / 2
            inv = torch.linalg.inv(torch.eye(n, dtype=torch.float64) + m)
            out.append((m.cuda(), inv.cuda()))
        return out

    def _apply(self, m, q, axis):
        return torch.movedim(torch.tensordot(m, q, dims=([1], [axis])), 0, axis)

    def step(self, q, t):
        if self.model == "discrete":
            return self.e[t] * self._conv(q, self.bond[t])
        if self.walls is not None:
            e = self.e[t] ** 2
            p = e * q
            ops = self.sweeps[t]
            lp = [self._apply(m, p, a) for a, (m, _) in enumerate(ops)]
            x = self._apply(ops[0][1], p - lp[0] - 2 * sum(lp[1:], torch.zeros_like(p)), 0)
            for a in range(1, len(ops)):
                x = self._apply(ops[a][1], x + lp[a], a)
            return e * x
        e = self.e[t]  # a quarter step's field factor
        full = e ** 2 * self._conv(e ** 2 * q, self.bond[t])
        two = e ** 2 * self._conv(e * q, self.half[t])
        two = e * self._conv(two, self.half[t])
        return (4 * two - full) / 3

    def solve(self, w, stress=False):
        self.e = {t: torch.exp(-v * (self.ds / 4 if self.model == "continuous" else self.ds)) for t, v in w.items()}
        phi = {t: torch.zeros_like(v) for t, v in w.items()}
        Q, dq = [], []
        for fraction, blocks in self.polymers:
            alpha = sum(s for _, s, _, _ in blocks) / 60
            seg = {}
            for t, s, v, u in blocks:
                seg[(v, u)] = seg[(u, v)] = (t, int(round(s / 60 / self.ds)))
            q, start = {}, {}
            depth = {(v, u): _arm(blocks, v, u) for v, u in seg}

            def propagate(v, u):
                if (v, u) in q:
                    return
                t, N = seg[(v, u)]
                deps = [(a, b) for (a, b) in seg if b == v and a != u]
                for a, b in deps:
                    propagate(a, b)
                if self.model == "continuous":
                    s = torch.ones_like(w[t])
                    for d in deps:
                        s = s * q[d][-1]
                    line = [s]
                    for _ in range(N):
                        line.append(self.step(line[-1], t))
                else:
                    if deps:
                        s = torch.ones_like(w[t])
                        for d in deps:
                            s = s * self._conv(q[d][-1], self.half[seg[d][0]])
                        start[(v, u)] = s
                        first = self.e[t] * self._conv(s, self.half[t])
                    else:
                        first = self.e[t].clone()
                    line = [None, first]
                    for _ in range(N - 1):
                        line.append(self.step(line[-1], t))
                q[(v, u)] = line

            for v, u in seg:
                propagate(v, u)
            t, _, v, u = blocks[0]
            N = seg[(v, u)][1]
            if self.model == "continuous":
                total = (q[(v, u)][N] * q[(u, v)][0]).mean()
            else:
                total = (q[(v, u)][N] * q[(u, v)][1] / self.e[t]).mean()
            Q.append(total)
            sums = [0.0] * len(self.shape)

            def pair(a, b, table, scale):
                c = torch.fft.rfftn(a, dim=self.dims) * torch.fft.rfftn(b, dim=self.dims).conj()
                c = c.real * self.weight * scale
                if table is not None:
                    c = c * table
                for d in range(len(self.shape)):
                    sums[d] = sums[d] + (c * self.kk[d]).sum()

            for t, _, v, u in blocks:
                if len(depth[(v, u)]) > len(depth[(u, v)]):
                    v, u = u, v  # an odd count's 3/8 tail sits where the deeper propagator ends
                N, f, r = seg[(v, u)][1], q[(v, u)], q[(u, v)]
                b2 = self.bonds[t] ** 2
                if self.model == "continuous":
                    c = _simpson(N)
                    s = sum(c[n] * f[N - n] * r[n] for n in range(N + 1))
                    if stress:
                        for n in range(N + 1):
                            pair(f[N - n], r[n], None, b2 * c[n])
                else:
                    s = sum(f[N - n + 1] * r[n] for n in range(1, N + 1)) / self.e[t]
                    if stress:
                        for n in range(1, N):
                            pair(f[N - n], r[n], self.bond[t], b2)
                        if (v, u) in start:
                            pair(start[(v, u)], r[N], self.half[t], b2 / 2)
                        if (u, v) in start:
                            pair(f[N], start[(u, v)], self.half[t], b2 / 2)
                phi[t] = phi[t] + s * (self.ds * fraction / alpha / total)
            M = float(np.prod(self.shape))
            dq.append([x / (-3.0 * l * M * M / self.ds) * fraction / alpha / total for x, l in zip(sums, self.lx)])
        if not stress:
            return phi, Q, None
        return phi, Q, [sum(p[d] for p in dq) for d in range(len(self.shape))]


def _exact_statistics(case, seed):
    polymers, bonds = MOLECULES[case["molecule"]]
    shape = _grid(case)
    walls = _boundary(case) if case["kind"] == "film" else None
    c = _Chains(shape, _lengths(case), case.get("model", "continuous"), 1.0 / case["segments"], polymers, bonds, walls)
    w = {t: torch.from_numpy(v).cuda().reshape(shape) for t, v in _fields(case, seed, sorted(bonds)).items()}
    phi, Q, stress = c.solve(w, case.get("stress", False))
    out = {"phi": [phi[t].reshape(-1).cpu().numpy() for t in sorted(bonds)], "partitions": np.array([float(v) for v in Q])}
    if case.get("stress", False):
        out["stress"] = np.array([float(v) for v in stress])
    return out


def _exact_scft(case, seed):
    """One iteration from the start: statistics, residual, simple mixing of fields and box (the first step of Anderson
    mixing), every field's mean removed."""
    p = _scft_params(case)
    shape, lx = p["nx"], p["lx"]
    polymers = [(1.0, [("A", 21.6, 0, 1), ("B", 38.4, 1, 2)])]
    w0 = _scft_fields(case, seed)
    w = {t: torch.from_numpy(w0[t] - w0[t].mean()).cuda().reshape(shape) for t in ("A", "B")}
    phi, Q, stress = _Chains(shape, lx, "continuous", p["ds"], polymers, p["segment_lengths"]).solve(w, True)
    chi = p["chi_n"]["A,B"]
    half = (w["A"] - w["B"]) / 2  # the part of the fields the residual is taken of
    diff = {"A": chi * phi["B"] - half, "B": chi * phi["A"] + half}
    diff = {t: v - v.mean() for t, v in diff.items()}
    volume = float(np.prod(lx))
    dd = volume * sum((v ** 2).mean() for v in diff.values())
    ww = 1.0 + volume * sum((v ** 2).mean() for v in w.values())
    stress = torch.stack(stress)
    error = float(torch.sqrt(dd / ww) + torch.sqrt((stress ** 2).sum()))
    mix = p["optimizer"]["mix_init"] * 1.01
    new = {t: w[t] + mix * diff[t] for t in w}
    return {"partitions": np.array([float(Q[0])]), "stress": stress.cpu().numpy(), "error_level": error,
            "phi": np.array([phi[t].reshape(-1).cpu().numpy() for t in ("A", "B")]),
            "w": np.array([(new[t] - new[t].mean()).reshape(-1).cpu().numpy() for t in ("A", "B")])}


def _exact_lfts(case, seed):
    """The initial saddle-point search and one Langevin step of every replica: Leimkuhler-Matthews update of the
    exchange field, then Anderson mixing of the pressure field to the tolerance."""
    p = _lfts_params(case)
    shape, chi, am, R = p["nx"], p["chi_n"]["A,B"], p["am"], case["replicas"]
    M = int(np.prod(shape))
    polymers = [(1.0, [("A", 30, 0, 1), ("B", 30, 1, 2)])]
    chains = _Chains(shape, p["lx"], "continuous", p["ds"], polymers, p["segment_lengths"])
    seeds = _lfts_seeds(case, seed)
    w_out, h_out = [], []

    def statistics(wm, wp):
        phi, Q, _ = chains.solve({"A": wp + wm, "B": wp - wm})
        return phi["A"], phi["B"], Q[0]

    def saddle(wm, wp):
        ws, ds_, count, mix, old = [], [], -1, am["mix_init"], 1e20
        for it in range(1, p["saddle"]["max_iter"] + 1):
            a, b, Q = statistics(wm, wp)
            d = a + b - 1.0
            err = float(d.std(unbiased=False))
            if err < p["saddle"]["tolerance"]:
                break
            if err < am["start_error"] or count >= 0:
                count = min(count + 1, am["max_hist"])
                ws.insert(0, wp)
                ds_.insert(0, d)
                del ws[am["max_hist"] + 1:], ds_[am["max_hist"] + 1:]
            if count <= 0:
                mix = max(0.7 * mix, am["mix_min"]) if old < err else 1.01 * mix
                wp = wp + mix * d
            else:
                D = torch.stack([ds_[0] - v for v in ds_[1:count + 1]]).reshape(count, -1)
                coef = torch.linalg.solve(D @ D.T, D @ ds_[0].reshape(-1))
                new = ws[0] + ds_[0]
                for c, x, y in zip(coef, ws[1:], ds_[1:]):
                    new = new + c * (x + y - ws[0] - ds_[0])
                wp = new
            old = err
        energy = chi / 4 - wp.mean() + (wm ** 2).mean() / chi - torch.log(Q)
        return wp - wp.mean(), a, b, float(energy)

    sigma = math.sqrt(2 * p["langevin"]["dt"] * M / (float(np.prod(p["lx"])) * math.sqrt(p["langevin"]["nbar"])))
    for s in seeds:
        f = _lfts_initial(s, M)
        wm = torch.from_numpy((f["A"] - f["B"]) / 2).cuda().reshape(shape)
        wp = torch.from_numpy((f["A"] + f["B"]) / 2).cuda().reshape(shape)
        wp, a, b, _ = saddle(wm, wp)
        noise = np.random.Generator(np.random.PCG64(s)).normal(0.0, sigma, [1, M])
        noise = torch.from_numpy(noise).cuda().reshape(shape)
        wm = wm - (2 * wm / chi + a - b) * p["langevin"]["dt"] + 0.5 * noise
        wp, a, b, h = saddle(wm, wp)
        w_out.append(torch.stack([wm.reshape(-1), wp.reshape(-1)]))
        h_out.append(h)
    return {"w": torch.stack(w_out), "hamiltonian": torch.tensor(h_out, dtype=torch.float64)}


def _conv64(x, w, b=None):
    """Periodic 3^3 (or pointwise) convolution of a channels-last float64 array."""
    co, k = w.shape[0], w.shape[2]
    out = torch.zeros(list(x.shape[:-1]) + [co], dtype=torch.float64, device=x.device)
    for z in range(k):
        for y in range(k):
            for v in range(k):
                out += torch.roll(x, (k // 2 - z, k // 2 - y, k // 2 - v), (1, 2, 3)) @ w[:, :, z, y, v].T
    return out if b is None else out + b


def _exact_unet(case, seed):
    net = _unet(seed)

    def conv(m, x, relu=True):
        y = _conv64(x, m.weight.detach().cuda().to(torch.bfloat16).double(), m.bias.detach().cuda().double())
        return y.clamp_(min=0) if relu else y

    def block(name, x):
        m = getattr(net, name)
        return conv(m[2], conv(m[0], x))

    def pool(x):
        B, D, H, W, C = x.shape
        return x.reshape(B, D // 2, 2, H // 2, 2, W // 2, 2, C).mean((2, 4, 6))

    def up(x):
        return x.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)

    out = []
    for x in _unet_input(case, seed).split(1):
        h = x.permute(0, 2, 3, 4, 1).double()
        x1 = block("e1", h)
        x2 = block("e2", pool(x1))
        x3 = block("e3", pool(x2))
        y2 = block("d2", torch.cat([up(x3), x2], -1))
        y1 = block("d1", torch.cat([up(y2), x1], -1))
        out.append(conv(net.out, y1, False).permute(0, 4, 1, 2, 3))
    return torch.cat(out)


def _exact_conv(case, seed):
    x, gy, w, b = _conv_data(case, seed)
    ci, co = case["cin"], case["cout"]
    y, dx, dw, db = [], [], torch.zeros(27, co, ci, dtype=torch.float64, device="cuda"), 0.0
    w64 = w.double()
    back = w64.flip(2, 3, 4).transpose(0, 1)
    for xi, gi in zip(x.split(1), gy.split(1)):
        xi = xi.double()
        yi = _conv64(xi, w64, b.double()).clamp_(min=0)
        g = gi.double() * (yi > 0)
        y.append(yi)
        dx.append(_conv64(g, back))
        db = db + g.sum((0, 1, 2, 3))
        for t in range(27):
            s = torch.roll(xi, (1 - t // 9, 1 - t // 3 % 3, 1 - t % 3), (1, 2, 3))
            dw[t] += g.reshape(-1, co).T @ s.reshape(-1, ci)
    return {"y": torch.cat(y), "dx": torch.cat(dx), "dw": dw, "db": db}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("statistics", "film"):
        return _exact_statistics(case, seed)
    if kind == "scft":
        return _exact_scft(case, seed)
    if kind == "lfts":
        # beyond this the searches take longer than a check is worth
        if float(np.prod(_grid(case))) * case["replicas"] > 1.7e6:
            return None
        return _exact_lfts(case, seed)
    if kind == "unet":
        return _exact_unet(case, seed)
    return _exact_conv(case, seed)
