"""Performance cases: the work a user of this package has it do, through its public entry points.

Eight kinds of case.  Six are single passes or solves with a plain 64-bit counterpart or whole-number
results; ``crk_steps`` and ``ensemble`` are whole programs (an integrator loop, a batch of boxes).

  crk_steps     recorded CRKSPH integrator steps (``StepGraph``), the loop a blast-wave run spends its time in
  crk_rhs       one CRKSPH right-hand side issued from Python (``crkSPH_step``) on a list kept from the stage before
  compsph_rhs   the CompSPH pair passes of one right-hand side
  verlet        a neighbour search from scratch
  dfsph         one DFSPH pressure solve with a fixed iteration budget
  ensemble      a chunk of recorded steps of a batch of delta-SPH boxes
  mlp_forward   the warm-start network on one solve's feature rows
  mlp_grad      its training gradient on a batch

Particles are jittered periodic lattices in the memory order of the package's own case builders (x fastest in
2D), with smooth flow, energy and support fields whose phases and amplitudes come from the seed.  ``exact``
uses that order: the neighbours of lattice point k are the points at a fixed set of index offsets, so a pair
sum is a sum over offsets of rolled arrays in 64 bits.
"""
import math

import numpy as np
import torch

DEVICE = "cuda:0"
KERNELS = {"Wendland2": 1, "Wendland4": 2, "Wendland6": 3}
GAMMA = 5.0 / 3.0


# ---------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest run: 64^2 particles, where a step is a chain of short kernels and launches decide
        {"name": "crk_steps_2d_64", "kind": "crk_steps", "dim": 2, "side": 64, "neighbors": 32, "kernel": "Wendland4", "steps": 10},
        # the benchmark's workload: the 2D Sedov blast of 512^2 particles
        {"name": "crk_steps_2d_512", "kind": "crk_steps", "dim": 2, "side": 512, "neighbors": 32, "kernel": "Wendland4", "steps": 10},
        # an ordinary 2D right-hand side on an odd lattice, issued from Python (a user's own integrator)
        {"name": "crk_rhs_2d_777", "kind": "crk_rhs", "dim": 2, "side": 777, "neighbors": 20, "kernel": "Wendland2", "kahan": False},
        # the 3D blast's right-hand side with compensated sums and 128 neighbours: long rows, large records
        {"name": "crk_rhs_3d_96", "kind": "crk_rhs", "dim": 3, "side": 96, "neighbors": 128, "kernel": "Wendland4", "kahan": True},
        # the CompSPH scheme's pair passes on the benchmark's 2D size
        {"name": "compsph_rhs_2d_512", "kind": "compsph_rhs", "dim": 2, "side": 512, "neighbors": 32, "kernel": "Wendland4", "kahan": False},
        # neighbour searches: every third step or so in 2D, and the first step of every run
        {"name": "verlet_2d_512", "kind": "verlet", "dim": 2, "side": 512, "neighbors": 32, "h_spread": 0.05},
        {"name": "verlet_3d_101", "kind": "verlet", "dim": 3, "side": 101, "neighbors": 128, "h_spread": 0.05},
        # pressure solves: a dam-break-sized 3D density solve, and a small 2D divergence-free solve with varying supports
        {"name": "dfsph_density_3d_100", "kind": "dfsph", "solve": "density", "dim": 3, "side": 100, "neighbors": 40, "kernel": "Wendland2",
         "h_spread": 0.0, "iterations": 16},
        {"name": "dfsph_divergence_2d_96", "kind": "dfsph", "solve": "divergence", "dim": 2, "side": 96, "neighbors": 32, "kernel": "Wendland4",
         "h_spread": 0.05, "iterations": 16},
        # a quarter of the ensemble benchmark: 64 uneven boxes, one recorded chunk of six RK2 steps
        {"name": "ensemble_64", "kind": "ensemble", "boxes": 64, "nmin": 4096, "nmax": 65536},
        # inference on a large solve's particles, and the training gradient on the benchmark's batch
        {"name": "mlp_forward_16m", "kind": "mlp_forward", "samples": 1 << 24},
        {"name": "mlp_grad_4m", "kind": "mlp_grad", "samples": 1 << 22},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["crk_steps", "crk_rhs", "crk_rhs", "compsph_rhs", "verlet", "verlet", "dfsph", "dfsph", "ensemble", "mlp_forward",
                       "mlp_grad"])
    if kind == "mlp_forward":
        return {"kind": kind, "samples": _log_int(rng, 4000, 1 << 24)}
    if kind == "mlp_grad":
        return {"kind": kind, "samples": _log_int(rng, 4096, 1 << 22)}
    if kind == "ensemble":
        return {"kind": kind, "boxes": rng.randint(3, 64), "nmin": rng.choice([1024, 4096]), "nmax": rng.choice([16384, 40000, 65536])}
    kernel = rng.choice(list(KERNELS))
    if kind == "crk_steps":
        return {"kind": kind, "dim": 2, "side": _log_int(rng, 48, 512), "neighbors": rng.choice([20, 32, 50]), "kernel": kernel,
                "steps": rng.randint(4, 10)}
    dim = rng.choice([2, 3])
    if kind == "dfsph":
        return {"kind": kind, "solve": rng.choice(["density", "divergence"]), "dim": dim,
                "side": _log_int(rng, 40, 700) if dim == 2 else _log_int(rng, 16, 100), "neighbors": rng.choice([32, 50] if dim == 2 else [40, 60]),
                "kernel": kernel, "h_spread": rng.choice([0.0, 0.05]), "iterations": rng.randint(2, 16)}
    neighbors = rng.choice([20, 32, 50] if dim == 2 else [50, 64, 128])
    if kind == "verlet":
        return {"kind": kind, "dim": dim, "side": _log_int(rng, 40, 900) if dim == 2 else _log_int(rng, 20, 100), "neighbors": neighbors,
                "h_spread": rng.choice([0.0, 0.05, 0.15])}
    return {"kind": kind, "dim": dim, "side": _log_int(rng, 60, 800) if dim == 2 else _log_int(rng, 20, 96), "neighbors": neighbors,
            "kernel": kernel, "kahan": rng.choice([False, True])}


# ---------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _rand(g, *shape):
    return torch.rand(shape, device=DEVICE, generator=g, dtype=torch.float64)


def _support(side, neighbors, dim):
    v = neighbors / side ** dim
    return math.sqrt(v / math.pi) if dim == 2 else (0.75 * v / math.pi) ** (1.0 / 3.0)


def _lattice(side, dim):
    c = (torch.arange(side, device=DEVICE, dtype=torch.float64) + 0.5) / side - 0.5
    return torch.stack([a.reshape(-1) for a in torch.meshgrid(*([c] * dim), indexing="xy")], 1)


def _modes(g, x, count=4):
    """A smooth periodic field of unit amplitude: a few low Fourier modes with random phases."""
    k = torch.randint(1, 4, (count, x.shape[1]), device=DEVICE, generator=g).double()
    phase = 2 * math.pi * _rand(g, count)
    f = torch.zeros_like(x[:, 0])
    for a in range(count):
        f += torch.sin(2 * math.pi * (x * k[a]).sum(1) + phase[a]) / count
    return f


def _f32(t):
    return t.float().contiguous()


def _particles(case, seed):
    """Positions, supports, masses and smooth velocity and energy fields (32 bits; the 64-bit counterpart starts from these values)."""
    dim, side = case["dim"], case["side"]
    # the geometry is one jittered lattice, numbered from a point that the seed chooses: neighbour lists of
    # another seed are other lists with as many entries
    g = _gen(side)
    x = _lattice(side, dim)
    x = x + (_rand(g, *x.shape) - 0.5) * (0.2 / side)
    H = _support(side, case["neighbors"], dim) * (1.0 + case.get("h_spread", 0.03) * _modes(g, x))
    g = _gen(seed)
    shift = torch.randint(0, side, (dim,), device=DEVICE, generator=g).tolist()
    x, H = (torch.roll(f.reshape(*[side] * dim, -1), shift, tuple(range(dim))).reshape(f.shape) for f in (x, H))
    out = {"x": _f32(torch.remainder(x + 0.5, 1.0) - 0.5), "H": _f32(H)}
    out["m"] = _f32((1.0 + 0.05 * _modes(g, x)) / side ** dim)
    out["v"] = _f32(torch.stack([_modes(g, x) for _ in range(dim)], 1))
    out["u"] = _f32(1.0 + 0.5 * _modes(g, x))
    out["rho"] = _f32(1.0 + 0.05 * _modes(g, x))
    out["dvdt"] = _f32(torch.stack([0.2 * _modes(g, x) for _ in range(dim)], 1))
    out["p"] = _f32(0.1 + 0.05 * _modes(g, x))
    out["alpha"] = _f32(1.0 + 0.5 * _modes(g, x))
    return out


def _config(case):
    import warpsph_b200 as ws
    dim = case["dim"]
    cfg, integrator = ws.buildConfig(dim=dim, domain=ws.buildDomainDescription(1.0, dim, True, torch.device(DEVICE)),
                                     kernel=ws.KernelFunctions[case.get("kernel", "Wendland4")], targetNeighbors=case["neighbors"],
                                     integrationScheme=ws.IntegrationSchemeType.rungeKutta2, cflFactor=0.3, device=torch.device(DEVICE))
    return ws, cfg, integrator


def _network(g):
    """The warm-start network's parameter vector: W1 b1 W2 b2 W3 b3 w4 b4."""
    parts = []
    for rows, cols in ((64, 8), (64, 64), (64, 64), (1, 64)):
        parts.append(torch.randn((rows * cols,), device=DEVICE, generator=g) * math.sqrt(2.0 / cols))
        parts.append(torch.randn((rows,), device=DEVICE, generator=g) * 0.1)
    return torch.cat(parts).contiguous()


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def _prepare_crk_steps(case, seed):
    from warpsph_b200 import ops
    from warpsph_b200.stepgraph import StepGraph
    ws, cfg, integrator = _config(case)
    System, State, Config, _, step, *_ = ws.buildScheme("crkSPH")
    sch = Config()
    sch.gamma = GAMMA
    sch.viscositySwitchParams.scheme = ws.ViscositySwitch.CullenDehnen2010
    g = _gen(seed)
    energy = 0.5 + float(_rand(g, 1))
    system = ws.buildSedov(System, State, cfg, nx=case["side"], dim=2, domainExtent=1.0, E0=energy, p0=1e-6, gamma=GAMMA,
                           kernel=cfg.kernel, targetNeighbors=case["neighbors"], device=torch.device(DEVICE))
    S = system.state
    S.positions = _f32(torch.remainder(S.positions.double() + (_rand(g, *S.positions.shape) - 0.5) * (0.1 / case["side"]) + 0.5, 1.0) - 0.5)
    system.adjacency = None
    ops.release_device_lists()      # a simulation of its own: it shares no rows with another one of the same size
    sg = StepGraph(system, integrator, step, cfg, sch, dt=cfg.dt)
    names = ("positions", "velocities", "internalEnergies", "supports", "masses", "densities", "alpha0s", "alphas", "divergence")
    return {"graph": sg, "start": {k: getattr(sg.inputs.state, k).clone() for k in names}, "dt": sg.dt.clone(), "steps": case["steps"]}


def _prepare_crk_rhs(case, seed):
    from warpsph_b200 import ops
    ws, cfg, _ = _config(case)
    System, State, Config, _, step, *_ = ws.buildScheme("crkSPH")
    sch = Config()
    sch.gamma = GAMMA
    sch.viscositySwitchParams.scheme = ws.ViscositySwitch.CullenDehnen2010
    sch.compensatedSums = case["kahan"]
    q = _particles(case, seed)
    # the stage before left a list: built where the particles were a step ago, still valid
    before = _f32(torch.remainder(q["x"].double() - (0.02 / case["side"]) * q["v"].double() + 0.5, 1.0) - 0.5)
    adjacency = ops.buildVerletList(before, q["H"], ws.make_params(cfg, sch), cfg.verletScale)
    ones = torch.ones_like(q["H"])
    state = State(positions=q["x"], velocities=q["v"], supports=q["H"], masses=q["m"], densities=ones, internalEnergies=q["u"],
                  divergence=0.5 * (q["rho"] - 1.0), alpha0s=q["alpha"], alphas=q["alpha"])
    return {"step": step, "system": System(state=state, adjacency=adjacency, domain=cfg.domain), "dt": 1e-4, "config": cfg, "params": sch}


def _prepare_compsph_rhs(case, seed):
    from warpsph_b200 import ops
    ws, cfg, _ = _config(case)
    _, _, Config, *_ = ws.buildScheme("compSPH")
    sch = Config()
    sch.gamma = GAMMA
    sch.compensatedSums = case["kahan"]
    q = _particles(case, seed)
    q["c"] = torch.sqrt(q["u"] * (GAMMA * (GAMMA - 1.0)))
    q["P"] = q["rho"] * q["u"] * (GAMMA - 1.0)
    params = ws.make_params(cfg, sch)
    return {"q": q, "params": params, "adjacency": ops.buildVerletList(q["x"], q["H"], params, cfg.verletScale)}


def _prepare_verlet(case, seed):
    ws, cfg, _ = _config(case)
    q = _particles(case, seed)
    return {"x": q["x"], "H": q["H"], "params": ws.make_params(cfg), "scale": cfg.verletScale}


def _prepare_dfsph(case, seed):
    from warpsph_b200 import ops
    from warpsph_b200.configurations import IncompressibleSPHConfig
    ws, cfg, _ = _config(case)
    q = _particles(case, seed)
    scheme = IncompressibleSPHConfig()
    scheme.fluid.restDensity = 1.0
    for solver in (scheme.solverConfig.pressureSolver, scheme.solverConfig.divergenceFreeSolver):
        solver.minIterations = solver.maxIterations = case["iterations"]
    adjacency = ops.buildVerletList(q["x"], q["H"], ws.make_params(cfg), cfg.verletScale)
    state = ws.buildScheme("dfsph")[1](positions=q["x"], velocities=q["v"], supports=q["H"], masses=q["m"], densities=q["rho"], pressures=q["p"])
    return {"state": state, "dvdt": q["dvdt"], "config": cfg, "scheme": scheme, "adjacency": adjacency, "solve": case["solve"],
            "dt": 0.1 / case["side"]}


def _prepare_ensemble(case, seed):
    from warpsph_b200.ensemble import BoxSet, Ensemble, box_sizes
    sizes = box_sizes(case["boxes"], 0, case["nmin"], case["nmax"])
    E = Ensemble(BoxSet(sizes, [int(seed) % (1 << 28) + b for b in range(len(sizes))]), DEVICE)
    E.tile = (4, 128)               # the tile the autotuner settles on for these boxes
    E.advance(1)
    return {"ensemble": E}


def _prepare_mlp(case, seed):
    g = _gen(seed)
    theta = _network(g)
    feats = torch.randn((case["samples"], 8), device=DEVICE, generator=g)
    return {"theta": theta, "feats": feats, "target": torch.randn((case["samples"],), device=DEVICE, generator=g),
            "scale": 0.5 + torch.rand((1,), device=DEVICE, generator=g), "grad": case["kind"] == "mlp_grad"}


_PREPARE = {"crk_steps": _prepare_crk_steps, "crk_rhs": _prepare_crk_rhs, "compsph_rhs": _prepare_compsph_rhs, "verlet": _prepare_verlet,
            "dfsph": _prepare_dfsph, "ensemble": _prepare_ensemble, "mlp_forward": _prepare_mlp, "mlp_grad": _prepare_mlp}


# ---------------------------------------------------------------------------------------------- one pass
def run(state):
    from warpsph_b200 import ops
    if "graph" in state:
        # the state of the step before comes in, a few recorded steps follow.  The switch's alphas are not
        # returned: its limiter divides rounding by rounding where the divergence vanishes, and the CRK
        # right-hand side does not read them.
        sg = state["graph"]
        sg.load_state(state["start"])
        sg.dt.copy_(state["dt"])
        sg.replay(state["steps"])
        S = sg.system.state
        return {k: getattr(S, k) for k in ("positions", "velocities", "internalEnergies", "supports", "densities", "pressures", "soundspeeds")}
    if "step" in state:
        system = state["system"].initializeNewState()
        update, _, S = state["step"](system, state["dt"], state["config"], state["params"])
        return {"dvdt": update.dvdt, "dudt": update.dudt, "dEdt": update.dEdt, "drhodt": update.drhodt, "supports": S.supports,
                "densities": S.densities, "pressures": S.pressures, "soundspeeds": S.soundspeeds, "entropies": S.entropies,
                "divergence": S.divergence}
    if "q" in state:
        q, p, adj = state["q"], state["params"], state["adjacency"]
        omega, div, drhodt = ops.compsph_prep(p, q["x"], q["H"], q["m"], q["rho"], q["v"], adj)
        dvdt, dudt, dEdt, ap, av = ops.compsph_accel_dudt(p, q["x"], q["H"], q["m"], q["rho"], q["v"], q["c"], q["alpha"], q["P"], omega, adj)
        return {"omega": omega, "div": div, "drhodt": drhodt, "dvdt": dvdt, "dudt": dudt, "dEdt": dEdt, "ap_ij": ap, "av_ij": av}
    if "scale" in state and "x" in state:
        adj = ops.buildVerletList(state["x"], state["H"], state["params"], state["scale"])
        return {"offsets": adj.neighborOffsets, "counts": adj.numNeighbors, "interacting": adj.interCounts, "list": adj.neighborList,
                "sort": adj.sortIndex, "keys": adj.sortedKeys}
    if "solve" in state:
        from warpsph_b200.incompressible import solveDivergenceFree, solveIncompressible
        solve = solveIncompressible if state["solve"] == "density" else solveDivergenceFree
        acc, p, history, flags = solve(state["state"], state["config"], state["scheme"], state["adjacency"], state["dvdt"], state["dt"],
                                       device_history=True)
        return {"accel": acc, "pressure": p, "history": history, "iterations": flags[0], "status": flags[1]}
    if "ensemble" in state:
        E = state["ensemble"]
        E.advance(E.graph_steps)
        return {"x": E.x, "v": E.v, "rho": E.rho}
    if state["grad"]:
        grad, loss = ops.mlp_grad(state["theta"], state["feats"], state["target"])
        return {"grad": grad, "loss": loss}
    return ops.mlp_forward(state["theta"], state["feats"], state["scale"])


# ---------------------------------------------------------------------------------------------- least work
def work(case):
    """Bytes: each input read once and each output written once, with 4 bytes per neighbour index of a given list.
    Flops: the arithmetic of the pair bodies (a multiply-add counts two)."""
    kind = case["kind"]
    if kind in ("mlp_forward", "mlp_grad"):
        n, forward = case["samples"], 2.0 * (8 * 64 + 2 * 64 * 64 + 64)
        backward = 2 * (2 * 64 * 64) + 2 * (2 * 64 * 64 + 64 * 8) + 4 * 64
        return {"bytes": 36.0 * n + 4 * 8961, "flops": n * (forward + (backward if kind == "mlp_grad" else 0))}
    if kind == "ensemble":
        n = sum(int(round(math.sqrt(v))) ** 2 for v in np.exp(np.random.default_rng(0).uniform(math.log(case["nmin"]), math.log(case["nmax"]),
                                                                                           case["boxes"])))
        # 6 RK2 steps: two stages of two pair passes over 50 interacting neighbours
        return {"bytes": 6.0 * n * (2 * 20 + 12 + 4 * 50), "flops": 6.0 * n * 50 * 2 * (45 + 75)}
    d, k = case["dim"], float(case["neighbors"])
    n = float(case["side"]) ** d
    if kind == "verlet":
        entries = k * 2.0                       # the Verlet sphere: (2^(1/d))^d times the support's volume
        return {"bytes": n * (4 * d + 4 + 4 * entries + 20), "flops": n * entries * (3 * d + 2)}
    if kind == "dfsph":
        return {"bytes": n * (12 * d + 16 + 4 * d + 4 + 4 * k), "flops": n * k * (2 * case["iterations"] + 2) * (8 * d + 14)}
    if kind == "compsph_rhs":
        return {"bytes": n * (8 * d + 28 + 4 * d + 20 + k * (4 + 2 * 8 * d)), "flops": n * k * (30 * d + 120)}
    rhs = n * k * (20 + 20 + 20 + (14 + 8 * d * d + 3 * d ** 3) + (30 + 12 * d * d) + 30 + (110 + 24 * d * d + 20 * d) + 12)
    if kind == "crk_rhs":
        return {"bytes": n * (8 * d + 24 + 8 * d + 36 + 4 * k), "flops": rhs}
    state = 2 * (8 * d + 24)
    return {"bytes": case["steps"] * n * (state + 2 * 4 * k), "flops": case["steps"] * (2 * rhs + 2 * n * k * 6 * d)}


# ---------------------------------------------------------------------------------------------- 64 bits
def exact(case, seed):
    fn = {"crk_rhs": _exact_crk_rhs, "compsph_rhs": _exact_compsph_rhs, "dfsph": _exact_dfsph, "mlp_forward": _exact_mlp,
          "mlp_grad": _exact_mlp}.get(case["kind"])
    if fn is None:
        return None     # whole numbers (neighbour lists), or many steps of a whole program
    with torch.no_grad():
        return fn(case, seed)


_NORM = {(1, 2): 7 / math.pi, (2, 2): 9 / math.pi, (3, 2): 78 / (7 * math.pi), (1, 3): 21 / (2 * math.pi), (2, 3): 495 / (32 * math.pi),
         (3, 3): 1365 / (64 * math.pi)}
_SCALE = {(1, 2): 1.897366596, (2, 2): 2.171240593, (3, 2): 2.415229458, (1, 3): 1.936491673, (2, 3): 2.207940217, (3, 3): 2.449489743}


class _Sums:
    """Pair sums of a jittered periodic lattice: ``pairs()`` yields (x_ij, r, at) for every index offset within
    reach, at(f) being the neighbour's values of f."""

    def __init__(self, case, x, Hmax):
        self.d, self.side = case["dim"], case["side"]
        self.k = KERNELS[case["kernel"]]
        self.C = _NORM[(self.k, self.d)]
        self.scale = _SCALE[(self.k, self.d)]
        self.x = x
        w = 1.1 * Hmax * self.side + 0.4
        m = int(math.ceil(w))
        grid = np.stack([a.ravel() for a in np.meshgrid(*([np.arange(-m, m + 1)] * self.d))], 1)
        self.offsets = [tuple(int(v) for v in o) for o in grid if math.sqrt(float((o * o).sum())) < w]

    def pairs(self):
        shape = (self.side,) * self.d
        dims = tuple(range(self.d))
        for o in self.offsets:
            def at(f, o=o):
                return torch.roll(f.reshape(*shape, *f.shape[1:]), o, dims).reshape(f.shape)
            xij = self.x - at(self.x)
            xij = xij - torch.round(xij)
            yield xij, torch.sqrt((xij * xij).sum(1)), at

    def kp(self, q):
        t = (1 - q).clamp(min=0)
        if self.k == 1:
            return t ** 4 * (1 + 4 * q), 20 * t ** 3
        if self.k == 2:
            return t ** 6 * (1 + 6 * q + 35 / 3 * q * q), 56 / 3 * (1 + 5 * q) * t ** 5
        return t ** 8 * (1 + 8 * q + 25 * q * q + 32 * q ** 3), 22 * (1 + 7 * q + 16 * q * q) * t ** 7

    def W(self, r, H):
        return self.C / H ** self.d * self.kp(r / H)[0]

    def Ws(self, r, H):
        """W and s with grad W = s x_ij."""
        k, p = self.kp(r / H)
        c = self.C / H ** self.d
        return c * k, -c * p / (H * H)

    def WdH(self, r, H):
        q = r / H
        k, p = self.kp(q)
        c = self.C / H ** self.d
        return c * k, -c / H * (self.d * k - q * q * p)


def _mul(s, v):
    return s[:, None] * v


def _crk_gradient(x, W, s, A, B, gA, gB):
    bx = 1 + (B * x).sum(1)
    gbx = (gB * x[:, :, None]).sum(1)
    return _mul(A * bx * s, x) + _mul(A * W, B) + _mul(bx * W, gA) + _mul(A * W, gbx)


def _exact_crk_rhs(case, seed):
    q = {k: v.double() for k, v in _particles(case, seed).items()}
    d, x, H, m, v, u = case["dim"], q["x"], q["H"], q["m"], q["v"], q["u"]
    S = _Sums(case, x, float(H.max()))
    # one Newton iteration of the adaptive support (gather)
    rho, dh = torch.zeros_like(H), torch.zeros_like(H)
    for xij, r, at in S.pairs():
        W, g = S.WdH(r, H)
        mj = at(m)
        rho += mj * W
        dh += mj * g
    vol = case["neighbors"] * (m / rho)
    F = H - (torch.sqrt(vol / math.pi) if d == 2 else (vol / math.pi * 0.75) ** (1.0 / 3.0))
    omega = 1 + H / (rho * d) * dh
    lo, hi = H.min() / 4, H.max() * 4
    H = torch.minimum(torch.maximum(H - F / (omega + 1e-6), lo), hi)
    # apparent volumes and the linear corrections (scatter)
    V = torch.zeros_like(H)
    for xij, r, at in S.pairs():
        V += S.W(r, at(H))
    V = 1 / V
    n = H.shape[0]
    zero = lambda *s: torch.zeros((n, *s), device=H.device, dtype=torch.float64)    # noqa: E731
    m0, s0, m1, s1, dm0, m2, dm1, dm2 = zero(), zero(), zero(d), zero(d), zero(d), zero(d, d), zero(d, d), zero(d, d, d)
    eye = torch.eye(d, device=H.device, dtype=torch.float64)
    for xij, r, at in S.pairs():
        Vj, mj = at(V), at(m)
        W, s = S.Ws(r, at(H))
        g = _mul(s, xij)
        m0 += Vj * W
        s0 += mj * W
        m1 += _mul(Vj * W, xij)
        s1 += _mul(mj * W, xij)
        dm0 += _mul(Vj, g)
        xx = xij[:, :, None] * xij[:, None, :]
        m2 += (Vj * W)[:, None, None] * xx
        dm1 += Vj[:, None, None] * (xij[:, :, None] * g[:, None, :] + W[:, None, None] * eye)
        sym = xij[:, None, :, None] * eye[None, :, None, :] + xij[:, :, None, None] * eye[None, None, :, :]
        dm2 += Vj[:, None, None, None] * (xx[..., None] * g[:, None, None, :] + sym * W[:, None, None, None])
    inv = torch.linalg.inv(m2)
    B = -(inv @ m1[..., None])[..., 0]
    A = 1 / (m0 + (m1 * B).sum(1))
    gB = -(inv @ (dm1 + (dm2 * B[:, None, :, None]).sum(2)))
    gA = -(A * A)[:, None] * (dm0 + (dm1 * B[:, :, None]).sum(1) + (gB * m1[:, :, None]).sum(1))
    rho = A * (s0 + (B * s1).sum(1))
    P = (GAMMA - 1) * rho * u
    c = torch.sqrt(u.abs() * GAMMA * (GAMMA - 1))
    entropy = u * (GAMMA - 1) * rho ** (1 - GAMMA)
    # corrected velocity gradient (scatter)
    G = zero(d, d)
    for xij, r, at in S.pairs():
        W, s = S.Ws(r, at(H))
        gr = _crk_gradient(xij, W, s, A, B, gA, gB)
        G += (_mul(at(V), at(v) - v))[:, :, None] * gr[:, None, :]
    drhodt = -torch.diagonal(G, dim1=1, dim2=2).sum(1) * rho
    # momentum and energy (limited CRK viscosity)
    dvdt, dudt = zero(d), zero()
    ks = S.scale

    def side_terms(Hs):
        sm = Hs / ks
        return 1 / sm, 1e-7 * sm * sm

    inv_i, eps_i = side_terms(H)
    for xij, r, at in S.pairs():
        Hj, Vj, vj, rj, cj, Pj = at(H), at(V), at(v), at(rho), at(c), at(P)
        r2 = r * r
        inside = r < torch.maximum(H, Hj)
        eta = r * torch.minimum(1 / H, 1 / Hj)
        factor = torch.where(eta < 0.3333333, torch.exp(-(((eta - 0.3333333) / 0.2) ** 2)), torch.ones_like(eta))
        Gi = (G * xij[:, None, :]).sum(2)
        Gj = (at(G) * xij[:, None, :]).sum(2)
        gi, gj = 0.25 * (Gi * xij).sum(1), 0.25 * (Gj * xij).sum(1)
        pos = lambda t: torch.where(t >= 0, 1.0, -1.0)    # noqa: E731
        ri, rjj = gi / (pos(gj) * gj.abs()), gj / (pos(gi) * gi.abs())
        ri, rjj = torch.where(ri.isnan(), 1.0, ri), torch.where(rjj.isnan(), 1.0, rjj)
        t = torch.minimum(ri, rjj)
        vl = 2 / (1 + t.clamp(min=0))
        phi = torch.where(t <= 0, 0.0, t * vl * vl) * factor
        hp = 0.5 * phi.clamp(0, 1)
        vdi = v - _mul(hp, Gi)
        da, dd = vdi - (vj + _mul(hp, Gj)), vdi - (vj - _mul(hp, Gj))
        Wi, si = S.Ws(r, Hj)
        Wj, sj = S.Ws(r, H)
        gw = 0.5 * (_crk_gradient(xij, Wi, si, A, B, gA, gB) - _crk_gradient(-xij, Wj, sj, at(A), at(B), at(gA), at(gB)))
        inv_j, eps_j = side_terms(Hj)
        idi, idj = inv_i / (r2 * inv_i ** 2 + eps_i), inv_j / (r2 * inv_j ** 2 + eps_j)

        def Q(dv):
            s = (dv * xij).sum(1)
            mi, mj_ = (s * idi).clamp(max=0), (s * idj).clamp(max=0)
            return rho * (-c * mi + mi * mi) + rj * (-cj * mj_ + mj_ * mj_)

        w = torch.where(inside, Vj * (V / m), torch.zeros_like(V))
        dvdt += _mul(-(P + Pj + Q(da)) * w, gw)
        dudt += (Pj + 0.5 * Q(dd)) * ((v - vj) * gw).sum(1) * w
    dEdt = m * (v * dvdt).sum(1) + m * dudt
    return {"dvdt": dvdt, "dudt": dudt, "dEdt": dEdt, "drhodt": drhodt, "supports": H, "densities": rho, "pressures": P, "soundspeeds": c,
            "entropies": entropy, "divergence": -drhodt / rho}


def _exact_compsph_rhs(case, seed):
    q = _particles(case, seed)
    c32, P32 = torch.sqrt(q["u"] * (GAMMA * (GAMMA - 1.0))), q["rho"] * q["u"] * (GAMMA - 1.0)
    q = {k: t.double() for k, t in q.items()}
    c, P = c32.double(), P32.double()
    d, x, H, m, v, rho, al = case["dim"], q["x"], q["H"], q["m"], q["v"], q["rho"], q["alpha"]
    S = _Sums(case, x, float(H.max()))
    n = H.shape[0]
    zero = lambda *s: torch.zeros((n, *s), device=H.device, dtype=torch.float64)    # noqa: E731
    dh, div, con = zero(), zero(), zero()
    for xij, r, at in S.pairs():
        mj = at(m)
        dh += mj * S.WdH(r, H)[1]
        t = S.Ws(r, torch.maximum(H, at(H)))[1] * ((at(v) - v) * xij).sum(1)
        div += mj / at(rho) * t
        con += mj * t
    omega = 1 + H / (rho * d) * dh
    drhodt = -con / omega
    dvdt, dudt = zero(d), zero()
    pi_ = P / (rho * rho) / omega
    for xij, r, at in S.pairs():
        Hj, mj, rj, cj, aj, vj = at(H), at(m), at(rho), at(c), at(al), at(v)
        inside = r < torch.maximum(H, Hj)
        ux = ((v - vj) * xij).sum(1)
        rho_bar, hbar, coef = 0.5 * (rho + rj), 0.5 * (H + Hj), 0.5 * (al + aj)
        den = r + 1e-14 * hbar
        sfac = hbar / S.scale / den
        mu = ux / den * sfac

        def visc(cs, rs):
            val = rj / rho_bar * (coef * cs - 2.0 * coef * mu) * sfac
            return torch.where(ux > 0, 0.0, val) * (rho_bar / rs)

        vi, vjv = visc(c, rho), visc(cj, rj)
        gi, gj = _mul(S.Ws(r, H)[1], xij), _mul(S.Ws(r, Hj)[1], xij)
        gw = 0.5 * (gi + gj)
        pj = at(P) / (rj * rj) / at(omega)
        mup = -ux / (r + 1e-14 * H)
        Vj = mj / rj
        on = inside.double()
        dvdt += _mul(on * (-(pi_ + pj) * mj - 0.5 * (vi + vjv) * Vj * mup), gw)
        dotg = ((vj - v) * gi).sum(1)
        dudt += on * (-Vj * pi_ * rj * dotg - 0.5 * Vj * vi * mup * dotg)
    dEdt = m * (v * dvdt).sum(1) + m * dudt
    return {"omega": omega, "div": div, "drhodt": drhodt, "dvdt": dvdt, "dudt": dudt, "dEdt": dEdt, "ap_ij": None, "av_ij": None}


def _exact_dfsph(case, seed):
    q = {k: t.double() for k, t in _particles(case, seed).items()}
    d, x, H, m, rho = case["dim"], q["x"], q["H"], q["m"], q["rho"]
    dt = float(torch.tensor(0.1 / case["side"], dtype=torch.float32))
    density = case["solve"] == "density"
    vs = q["v"] + dt * q["dvdt"]
    S = _Sums(case, x, float(H.max()))
    V = m / rho
    n, N = H.shape[0], case["iterations"]
    div, sA, sB = torch.zeros_like(H), torch.zeros_like(x), torch.zeros_like(H)
    for xij, r, at in S.pairs():
        Vj = at(V)
        div += Vj * S.Ws(r, at(H))[1] * ((at(vs) - vs) * xij).sum(1)
        g = _mul(S.Ws(r, H)[1], xij)
        sA += _mul(Vj, g)
        sB += Vj * Vj / at(m) * (g * g).sum(1)
    div = -div
    alpha = -(V / m * (sA * sA).sum(1) + V * sB)
    if density:
        src, diag, p, dtf = 1.0 - (rho + dt * div).clamp(min=float(np.float32(0.9))), (dt * dt * alpha).clamp(max=-1e-6), torch.zeros_like(H), dt * dt
        tol = float(np.float32(5e-4))
    else:
        src, diag, p, dtf = -div, dt * alpha, 0.75 * q["p"], dt
    omega = float(np.float32(0.3))
    hist = torch.zeros((N, 4), device=H.device, dtype=torch.float64)

    def accel(p):
        a = torch.zeros_like(x)
        qi = p / (rho * rho)
        for xij, r, at in S.pairs():
            a -= _mul(at(m) * (qi + at(qi)) * S.Ws(r, at(H))[1], xij)
        return a

    for it in range(N):
        a = accel(p)
        s = torch.zeros_like(H)
        for xij, r, at in S.pairs():
            s += at(V) * S.Ws(r, at(H))[1] * ((at(a) - a) * xij).sum(1)
        res = src + dtf * s
        p = p + omega * res / diag
        if density:
            p = p.clamp(min=0)
            err, mu = (-res).clamp(min=-tol).mean(), 0.0
        else:
            err, mu = res.abs().mean(), p.mean()
        hist[it] = torch.stack([err, p.min() - mu, p.max() - mu, p.mean() - mu])
        p = p - mu
    return {"accel": accel(p), "pressure": p, "history": hist, "iterations": None, "status": None}


def _exact_mlp(case, seed):
    s = _prepare_mlp(case, seed)
    theta = s["theta"].double()
    n = case["samples"]
    shapes = [(64, 8), (64,), (64, 64), (64,), (64, 64), (64,), (1, 64), (1,)]
    grad, loss, out = torch.zeros_like(theta), torch.zeros(1, device=DEVICE, dtype=torch.float64), []
    for a in range(0, n, 1 << 19):
        with torch.enable_grad():
            t = theta.clone().requires_grad_(s["grad"])
            parts, o = [], 0
            for sh in shapes:
                parts.append(t[o:o + math.prod(sh)].reshape(sh))
                o += math.prod(sh)
            h = s["feats"][a:a + (1 << 19)].double()
            for k in range(3):
                h = torch.relu(h @ parts[2 * k].T + parts[2 * k + 1])
            y = (h @ parts[6].T + parts[7])[:, 0]
            if not s["grad"]:
                out.append(y.detach() * s["scale"].double())
                continue
            sq = ((y - s["target"][a:a + (1 << 19)].double()) ** 2).sum()
            grad += torch.autograd.grad(sq, t)[0] / n
            loss += sq.detach()
    return {"grad": grad, "loss": loss} if s["grad"] else torch.cat(out)
