"""Performance cases of the step path: what a user of the engine runs, sized
from the workloads (softflow_b200/workloads.py), the tests and the benchmark.

Every case is a plain dict.  `prepare` builds the initialized simulation (or
the network, or the marker arrays) a user's program holds before its loop,
`run` is one pass of that loop through the public API with the results such a
program reads, `work` the bytes and operations a pass cannot do without, and
`exact` the same results from plain torch in 64 bits.

Kinds of case:
  channel    one Simulation: `steps` steps, then its fields and markers
  ensemble   many channels in one Ensemble: `steps` steps, then every marker,
             the thermo records and (small ensembles) every channel's fields
  spread     the standalone marker-to-lattice spread on device arrays
  network    one training pass of the forcing network and its predictions
"""
import ctypes as C
import math

import numpy as np
import torch

import softflow_b200 as S
from softflow_b200.learned import MDFNetwork, harvest, train_network

COLLISION = {"bgk": S.CollisionModel.BGK, "mrt": S.CollisionModel.MRT,
             "reg": S.CollisionModel.REGULARIZED}
ELEM = {"fp64": 8, "fp32": 4, "fp16s": 2}
# capsules as in the workloads: (radius, nodes)
SIZES = {"skalak": (3.0, 24), "wlc": (6.0, 48)}


def channel(name=None, **kw):
    c = dict(kind="channel", nx=400, ny=80, precision="fp32", collision="reg", tau=0.8, fx=3e-5,
             sweeps=1, skalak=0, wlc=0, scalar=0.0, pillars=0, steps=100)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def ensemble(name=None, **kw):
    c = dict(kind="ensemble", channels=12, nx_min=200, nx_max=800, ny_min=40, ny_max=160,
             multiple=8, caps_min=5, caps_max=60, precision="fp16s", learned=False, fields=True,
             shapes=7, steps=50)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a test-sized double-precision run (the size of the smoke check):
        # every kernel of the step is tiny, so launches and latency are all
        channel("small_96x40_fp64", nx=96, ny=40, precision="fp64", skalak=2, sweeps=3, steps=50),
        # workload c0: a Poiseuille channel without capsules
        channel("poiseuille_400x80_fp32", steps=500),
        # workload c1: the channel with 30 capsules and five forcing sweeps,
        # the reference's everyday simulation
        channel("capsules_400x80_fp32", skalak=30, sweeps=5),
        # double precision (the mode that reproduces the reference) on a
        # coupled channel with both capsule kinds
        channel("capsules_512x200_fp64", nx=512, ny=200, precision="fp64", collision="bgk", fx=1e-5,
                skalak=40, wlc=20, sweeps=3, steps=50),
        # a pillar array (cell-type mask) driven by a body force, odd sizes
        channel("pillars_601x121_fp32", nx=601, ny=121, collision="mrt", pillars=12, fx=1e-5,
                steps=200),
        # solute transport beside capsules in FP16-shifted storage
        channel("scalar_512x160_fp16s", nx=512, ny=160, precision="fp16s", fx=3e-6, skalak=30,
                wlc=10, scalar=0.05),
        # workload c2's fluid: the plain stream-collide at full size
        channel("lattice_4096x1024_fp32", nx=4096, ny=1024, collision="mrt", fx=1e-6, steps=2000),
        # workload c2: 2,000 capsules of both kinds and the scalar
        channel("coupled_4096x1024_fp32", nx=4096, ny=1024, collision="mrt", fx=1e-5,
                skalak=1000, wlc=1000, scalar=0.05, steps=500),
        # a small ensemble whose channels have arbitrary (odd) sizes, plain
        # forcing sweeps
        ensemble("ensemble12_ragged_fp16s", nx_min=100, nx_max=400, ny_min=30, ny_max=120,
                 multiple=1, caps_max=20),
        # workload c3, the benchmark's: 256 channels with the learned forcing
        ensemble("ensemble256_learned_fp16s", channels=256, learned=True, fields=False,
                 steps=100),
        # a host code's own marker forces spread on its own field
        dict(name="spread_1000x700_fp64", kind="spread", nx=1000, ny=700, capsules=500, nodes=40),
        # the network's training on a harvested-size set, and its predictions
        dict(name="network_262144", kind="network", samples=262144, batch=8192, predict=204528),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    """A case of the same ranges: any size and remainder, any precision,
    collision operator, sweep count and capsule load."""
    k = rng.random()
    if k < 0.62:
        nx, ny = _log(rng, 64, 2048), _log(rng, 32, 512)
        if rng.random() < 0.6:                       # workload sizes are multiples of 8
            nx = max(64, nx // 8 * 8)
        room = (nx * (ny - 16)) // 900               # at most about 6 % of the area
        opt = rng.choice(["plain", "capsules", "capsules", "capsules", "scalar", "pillars"])
        c = channel(nx=nx, ny=ny, precision=rng.choice(["fp64", "fp32", "fp16s"]),
                    collision=rng.choice(["bgk", "mrt", "reg"]), tau=round(rng.uniform(0.6, 1.0), 3),
                    fx=min(3e-5, round(rng.uniform(0.01, 0.05) / (ny * ny), 9)),
                    steps=max(20, min(500, int(3e7 / (nx * ny)))))
        if opt == "pillars":
            c["pillars"] = rng.randint(1, 16)
        elif opt != "plain":
            c["sweeps"] = rng.choice([1, 3, 5])
            c["skalak"] = rng.randint(0, max(1, min(200, room // 2)))
            c["wlc"] = rng.randint(0, max(1, min(100, room // 8))) if ny >= 48 else 0
            c["steps"] = min(c["steps"], 100)
        if opt == "scalar":
            c["scalar"] = round(rng.uniform(0.01, 0.2), 3)
        return c
    if k < 0.82:
        n = _log(rng, 2, 128)
        return ensemble(channels=n, nx_min=64, nx_max=rng.randint(200, 800), ny_min=30,
                        ny_max=rng.randint(60, 160), multiple=rng.choice([1, 4, 8]),
                        caps_min=1, caps_max=rng.randint(4, 40),
                        precision=rng.choice(["fp64", "fp32", "fp16s"]), fields=n <= 12,
                        shapes=rng.randint(0, 1 << 20), learned=rng.random() < 0.25)
    if k < 0.92:
        nx, ny = _log(rng, 64, 2048), _log(rng, 32, 1024)
        return dict(kind="spread", nx=nx, ny=ny,
                    capsules=rng.randint(1, max(2, min(1000, nx * ny // 1500))),
                    nodes=rng.randint(12, 64))
    batch = 128 * _log(rng, 1, 128)
    return dict(kind="network", samples=batch * _log(rng, 1, 32) + rng.randint(0, 127),
                batch=batch, predict=_log(rng, 100, 300000))


# ------------------------------------------------------------------ inputs ----
def _place(rng, nx, ny, counts, margin=3.0, gap=3.5):
    """Capsule centres in a channel periodic in x, surfaces at least `gap` (the
    contact cut-off) apart and `margin` off the walls: (x, y, kind) rows."""
    out, X, Y, R = [], np.empty(0), np.empty(0), np.empty(0)
    for kind, n in counts:
        r = SIZES[kind][0]
        lo, hi = margin + 2.0 + r, ny - 3.0 - margin - r
        for _ in range(n):
            for _ in range(200):
                x, y = rng.uniform(0, nx), rng.uniform(lo, hi) if hi > lo else 0.5 * (ny - 1)
                d = np.abs(X - x)
                d = np.minimum(d, nx - d)
                if not np.any(d * d + (Y - y) ** 2 < (R + r + gap) ** 2):
                    out.append((x, y, kind))
                    X, Y, R = np.append(X, x), np.append(Y, y), np.append(R, r)
                    break
    return out


def _membrane(kind, G_s=0.06):
    if kind == "wlc":
        return S.MembraneParams(model=S.MembraneModel.WLC, G_s=G_s, k_bend=0.005,
                                use_helfrich_bending=True)
    return S.MembraneParams(model=S.MembraneModel.SKALAK, G_s=G_s, C_skalak=10.0, k_bend=0.0)


def _params(nx, ny, collision, tau, fx, sweeps, precision, scalar=0.0):
    p = S.SimulationParams(nx=nx, ny=ny, ibm_iterations=sweeps, precision=precision)
    p.fluid.boundary_type = S.BoundaryType.PERIODIC
    p.fluid.collision_model = COLLISION[collision]
    p.fluid.tau = tau
    p.fluid.body_force_x = fx
    if scalar:
        p.scalar.enabled = True
        p.scalar.diffusivity = [scalar]
    return p


def _pillars(case, seed):
    """Circular pillars (cx, cy, radius) off the walls and the seam."""
    rng = np.random.default_rng([seed, 3])
    r = max(2.0, min(case["nx"], case["ny"]) / 16.0)
    out = []
    for _ in range(case["pillars"]):
        out.append((float(rng.uniform(r + 2, case["nx"] - r - 3)),
                    float(rng.uniform(r + 2, case["ny"] - r - 3)), r))
    return out


def _fluid0(nx, ny, seed, device):
    """Populations of a developed flow: the equilibrium of a few long waves of
    small amplitude (weakly compressible speeds), [9][ny][nx] in 64 bits."""
    g = np.random.default_rng([seed, 1])
    y = torch.arange(ny, dtype=torch.float64, device=device)[:, None]
    x = torch.arange(nx, dtype=torch.float64, device=device)[None, :]
    prof = 4.0 * y * (ny - 1 - y) / (ny - 1.0) ** 2      # zero at the walls
    ux = torch.zeros((ny, nx), dtype=torch.float64, device=device)
    uy = torch.zeros_like(ux)
    rho = torch.ones_like(ux)
    for _ in range(4):
        kx, ky = int(g.integers(1, 5)), int(g.integers(1, 4))
        a, b, ph = g.uniform(-4e-3, 4e-3), g.uniform(-2e-3, 2e-3), g.uniform(0, 2 * math.pi)
        wave = torch.cos(2 * math.pi * kx * x / nx + ph) * torch.sin(math.pi * ky * y / (ny - 1))
        ux += a * wave
        uy += b * wave * prof
        rho += 0.1 * a * wave
    ux += float(g.uniform(0.005, 0.02)) * prof
    return _feq(rho, ux, uy), rho


def _gaussian(nx, ny, seed):
    g = np.random.default_rng([seed, 2])
    y, x = np.mgrid[0:ny, 0:nx]
    s = max(2.0, min(20.0, ny / 8.0))
    return np.exp(-((x - nx * g.uniform(0.3, 0.7)) ** 2 + (y - 0.5 * (ny - 1)) ** 2) / (2 * s * s))


def _shapes(case):
    """Channel shapes and constants of an ensemble (part of the case)."""
    rng = np.random.default_rng(case["shapes"])
    m = case["multiple"]
    out = []
    for _ in range(case["channels"]):
        nx = int(rng.integers(-(-case["nx_min"] // m), case["nx_max"] // m + 1)) * m
        ny = int(rng.integers(case["ny_min"], case["ny_max"] + 1))
        ny = max(32, ny // m * m)
        n = int(rng.integers(case["caps_min"], case["caps_max"] + 1))
        out.append((nx, ny, min(n, max(1, nx * (ny - 16) // 400)),
                    float(10.0 ** rng.uniform(-2, -1)), float(rng.uniform(0.6, 1.0)),
                    float(rng.uniform(1e-5, 3e-5))))
    return out


def _capsules(case, seed):
    """Per channel: placed capsules, (x, y, kind), and shear modulus."""
    if case["kind"] == "channel":
        rng = np.random.default_rng([seed, 0])
        return [(_place(rng, case["nx"], case["ny"],
                        (("wlc", case["wlc"]), ("skalak", case["skalak"]))), 0.06)]
    out = []
    for i, (nx, ny, n, G_s, _, _) in enumerate(_shapes(case)):
        out.append((_place(np.random.default_rng([seed, 0, i]), nx, ny, (("skalak", n),)), G_s))
    return out


def _ensemble(case, seed):
    ens = S.Ensemble(precision=case["precision"])
    for (nx, ny, _, _, tau, fx), (caps, G_s) in zip(_shapes(case), _capsules(case, seed)):
        i = ens.add_channel(_params(nx, ny, "reg", tau, fx, 5, case["precision"]))
        m = {k: _membrane(k, G_s) for k in SIZES}
        for x, y, kind in caps:
            ens.addCapsule(i, (x, y), SIZES[kind][0], SIZES[kind][1], m[kind])
    ens.initialize()
    return ens


def _network(seed):
    """A forcing network trained on a short plain run of a few channels."""
    small = _ensemble(ensemble(channels=24, precision="fp32"), seed + 1000)
    X, Y = harvest(small, at=[1, 2, 4, 8, 16, 32, 64, 128, 256, 512, 768, 1024, 1280, 1536])
    small.close()
    return train_network(X, Y, epochs=8, batch=4096, seed=1)[0]


def _rings(case, seed):
    """Marker rings of a host code: offsets, positions and forces."""
    rng = np.random.default_rng([seed, 4])
    n, k = case["capsules"], case["nodes"]
    r = 0.75 * k / (2 * math.pi)
    c = np.stack([rng.uniform(0, case["nx"], n), rng.uniform(2, case["ny"] - 3, n)], -1)
    th = 2 * math.pi * np.arange(k) / k + rng.uniform(0, 1, (n, 1))
    pos = c[:, None, :] + r * np.stack([np.cos(th), np.sin(th)], -1)
    pos[..., 0] %= case["nx"]
    pos[..., 1] = np.clip(pos[..., 1], 1.5, case["ny"] - 1.5)
    return (np.arange(n + 1, dtype=np.int32) * k, pos.reshape(-1, 2),
            rng.normal(0, 1e-3, (n * k, 2)))


def _samples(case, seed, n):
    """Features and corrections with the scales of harvested ones."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    scale = torch.tensor([1e-4, 1e-4, 1e-5, 1e-5, 0.05, 0.1, 0.02, 0.005], device="cuda")
    X = torch.randn((n, 8), generator=g, device="cuda") * scale
    Y = torch.stack([2.1 * X[:, 0] + 0.5 * X[:, 2] * torch.cos(X[:, 5]),
                     1.8 * X[:, 1] * (1 + X[:, 4]) + 0.4 * X[:, 3]], -1)
    return X, Y


def prepare(case, seed):
    if case["kind"] == "channel":
        p = _params(case["nx"], case["ny"], case["collision"], case["tau"], case["fx"],
                    case["sweeps"], case["precision"], case["scalar"])
        sim = S.Simulation(p)
        if case["pillars"]:
            b = S.ChannelBuilder(case["nx"], case["ny"]).addWalls()
            for cx, cy, r in _pillars(case, seed):
                b.addCirclePillar(cx, cy, r)
            b.setBoundaryType(S.BoundaryType.PERIODIC)
            sim.setChannelBuilder(b)
        for x, y, kind in _capsules(case, seed)[0][0]:
            sim.addCapsule((x, y), SIZES[kind][0], SIZES[kind][1], _membrane(kind))
        sim.initialize()
        f = _fluid0(case["nx"], case["ny"], seed, "cuda")[0]
        sim.field().set_distributions(f.cpu().numpy())
        if case["scalar"]:
            sim.advectionDiffusion().setConcentration(_gaussian(case["nx"], case["ny"], seed))
        return {"sim": sim, "case": case}
    if case["kind"] == "ensemble":
        net = _network(seed) if case["learned"] else None
        ens = _ensemble(case, seed)
        if net is not None:
            ens.setLearnedMDF(net)
        m = 2 * ens.num_markers()
        return {"ens": ens, "case": case, "pos": np.zeros(m), "vel": np.zeros(m)}
    if case["kind"] == "spread":
        off, pos, frc = _rings(case, seed)
        n = case["nx"] * case["ny"]
        return {"case": case, "off": torch.tensor(off, device="cuda"),
                "pos": torch.tensor(pos, device="cuda"), "frc": torch.tensor(frc, device="cuda"),
                "Fx": torch.zeros(n, dtype=torch.float64, device="cuda"),
                "Fy": torch.zeros(n, dtype=torch.float64, device="cuda")}
    X, Y = _samples(case, seed, case["samples"])
    net = MDFNetwork(0, seed=int(seed))
    net.fit_normalization(X.cpu().numpy(), Y.cpu().numpy())
    return {"case": case, "net": net, "X": X, "Y": Y, "P": _samples(case, seed + 1, case["predict"])[0]}


# -------------------------------------------------------------------- pass ----
_THERMO = ("max_speed", "mean_rho", "mean_velocity", "kinetic_energy", "min_rho", "max_rho",
           "mean_deformation", "max_deformation", "fluid_cells", "first_nonfinite",
           "capped_nodes", "num_capsules")


def _dptr(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def run(state):
    case = state["case"]
    if case["kind"] == "channel":
        sim = state["sim"]
        sim.run(case["steps"])
        out = dict(zip(("rho", "ux", "uy", "Fx", "Fy"), sim.field().macroscopic()))
        if case["skalak"] + case["wlc"]:
            caps = sim.capsules()
            out["pos"], out["vel"] = caps.positions(), caps.velocities()
        if case["scalar"]:
            out["C"] = sim.advectionDiffusion().concentration()
        return out
    if case["kind"] == "ensemble":
        ens = state["ens"]
        ens.run(case["steps"])
        lib, ctx = S.load_library(), ens.context()
        if lib.sfg_get_all_markers(ctx._h, _dptr(state["pos"]), _dptr(state["vel"])):
            raise RuntimeError(lib.sfg_last_error().decode())
        out = {"pos": state["pos"], "vel": state["vel"],
               "thermo": np.array([[t[k] for k in _THERMO] for t in ens.thermo()], dtype=float),
               "shapes": ctx.thermo()[1]}
        if case["fields"]:
            out["fields"] = [ens.field(i).macroscopic()[:3] for i in range(case["channels"])]
        return out
    if case["kind"] == "spread":
        state["Fx"].zero_()
        state["Fy"].zero_()
        lib = S.load_library()
        if lib.sfg_spread_forces(case["nx"], case["ny"], case["capsules"],
                                 state["off"].data_ptr(), state["pos"].data_ptr(),
                                 state["frc"].data_ptr(), state["Fx"].data_ptr(),
                                 state["Fy"].data_ptr(), case["capsules"] * case["nodes"],
                                 C.c_void_p(torch.cuda.current_stream().cuda_stream)):
            raise RuntimeError(lib.sfg_last_error().decode())
        return state["Fx"], state["Fy"]
    net = state["net"]
    loss = net.train(state["X"], state["Y"], epochs=1, batch=case["batch"], seed=net.steps())
    return {"loss": loss, "params": net.params(), "y": net.forward(state["P"])}


def work(case):
    if case["kind"] == "spread":
        m, n = case["capsules"] * case["nodes"], case["nx"] * case["ny"]
        return {"bytes": 32.0 * m + 32.0 * n, "flops": 160.0 * m}
    if case["kind"] == "network":
        n = case["samples"] // case["batch"] * case["batch"]
        mac = 8 * 64 + 64 * 64 + 64 * 2
        return {"bytes": 40.0 * (n + case["predict"]), "flops": 6.0 * mac * n + 2.0 * mac * case["predict"]}
    if case["kind"] == "channel":
        chans = [(case["nx"], case["ny"], case["skalak"] * 24 + case["wlc"] * 48, case["sweeps"])]
        read, scalar = 5, case["scalar"]
    else:
        chans = [(nx, ny, 24 * n, 5) for nx, ny, n, _, _, _ in _shapes(case)]
        read, scalar = (3 if case["fields"] else 0), 0.0
    e, real = ELEM[case["precision"]], 8 if case["precision"] == "fp64" else 4
    cells = sum(nx * ny for nx, ny, _, _ in chans)
    # per step: every population (and scalar population) read and written
    # once; per marker its position, velocity and reference state
    per_step = cells * 18 * (e + (real if scalar else 0)) + 96 * sum(m for _, _, m, _ in chans)
    flops = cells * (200 + (60 if scalar else 0)) + sum(m * (400 + 450 * k) for _, _, m, k in chans)
    return {"bytes": float(case["steps"] * per_step + cells * 8 * read),
            "flops": float(case["steps"] * flops)}


# ------------------------------------------------- the same in plain torch ----
_CX = [0, 1, 0, -1, 0, 1, -1, -1, 1]
_CY = [0, 0, 1, 0, -1, 1, 1, -1, -1]
_OPP = [0, 3, 4, 1, 2, 7, 8, 5, 6]
_W = [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4
# moments of the multiple-relaxation-time operator: density, energy, energy
# squared, x flux, x energy flux, y flux, y energy flux, normal and shear stress
_M = [[1] * 9, [-4, -1, -1, -1, -1, 2, 2, 2, 2], [4, -2, -2, -2, -2, 1, 1, 1, 1],
      [0, 1, 0, -1, 0, 1, -1, -1, 1], [0, -2, 0, 2, 0, 1, -1, -1, 1],
      [0, 0, 1, 0, -1, 1, 1, -1, -1], [0, 0, -2, 0, 2, 1, 1, -1, -1],
      [0, 1, -1, 1, -1, 0, 0, 0, 0], [0, 0, 0, 0, 0, 1, -1, 1, -1]]


def _vec(v, like):
    return torch.tensor(v, dtype=torch.float64, device=like.device)[:, None, None]


def _feq(rho, ux, uy):
    eu = _vec(_CX, rho) * ux + _vec(_CY, rho) * uy
    return _vec(_W, rho) * rho * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * (ux * ux + uy * uy))


class _Channel:
    """One channel, periodic in x between resting walls, in 64 bits: lattice
    Boltzmann with Guo forcing, elastic rings coupled by the four-point
    kernel with repeated direct forcing, soft contact, and a scalar."""

    def __init__(self, nx, ny, collision, tau, fx, sweeps, caps, G_s=0.06, f=None, solid=None,
                 scalar=0.0, C0=None, device="cpu"):
        self.nx, self.ny, self.coll, self.om, self.fx, self.K = nx, ny, collision, 1 / tau, fx, sweeps
        z = dict(dtype=torch.float64, device=device)
        self.f = f if f is not None else _feq(torch.ones((ny, nx), **z), torch.zeros((ny, nx), **z),
                                              torch.zeros((ny, nx), **z))
        if solid is None:
            solid = torch.zeros((ny, nx), dtype=torch.bool, device=device)
        solid = solid.clone()
        solid[0] = solid[-1] = True
        self.solid = solid
        self.into = [torch.roll(solid, (-_CY[q], -_CX[q]), (0, 1)) for q in range(9)]
        self.F = torch.zeros((2, ny, nx), **z)
        self.cx, self.cy = _vec(_CX, self.f), _vec(_CY, self.f)
        self.M = torch.tensor(_M, **z)
        self.Mi = torch.linalg.inv(self.M)
        r = torch.linspace(0, 2, 1025, **z)                # the kernel's 1024-bin table
        root = torch.sqrt(torch.clamp(torch.where(r <= 1, 1 + 4 * r - 4 * r * r,
                                                  -7 + 12 * r - 4 * r * r), min=0))
        self.tab = 0.125 * torch.where(r <= 1, 3 - 2 * r + root, 5 - 2 * r - root)
        # rings, grouped by node count
        self.rings, at, self.X, cap = [], 0, torch.zeros((0, 2), **z), []
        for c, (x, y, kind) in enumerate(caps):
            rad, n = SIZES[kind]
            th = 2 * math.pi * torch.arange(n, **z) / n
            X = torch.stack([x + rad * torch.cos(th), y + rad * torch.sin(th)], -1)
            self.X = torch.cat([self.X, X])
            cap += [c] * n
            if not self.rings or self.rings[-1]["kind"] != kind:
                self.rings.append({"kind": kind, "at": at, "n": n, "count": 0})
            self.rings[-1]["count"] += 1
            at += n
        self.V = torch.zeros_like(self.X)
        self.cap = torch.tensor(cap, device=device)
        self.G_s = G_s
        for g in self.rings:
            e = self._edges(g)[0]
            L = e.norm(dim=-1)
            g["L0"], g["A0"], g["P0"], g["prev"] = L, self._area(g)[0].abs() / 2, L.sum(1), None
            ep = torch.roll(e, 1, 1)
            g["ang"] = torch.atan2(ep[..., 0] * e[..., 1] - ep[..., 1] * e[..., 0], (ep * e).sum(-1))
            g["ds"] = 0.5 * (L + torch.roll(L, 1, 1))
        self.scalar = scalar
        if scalar:
            self.C = torch.tensor(C0, **z)
            self.g = _vec(_W, self.f) * self.C

    # -- rings
    def _image(self, d):
        d = d.clone()
        x = d[..., 0]
        d[..., 0] = torch.where(x > 0.5 * self.nx, x - self.nx, torch.where(x < -0.5 * self.nx, x + self.nx, x))
        return d

    def _of(self, g, A):
        return A[g["at"]:g["at"] + g["n"] * g["count"]].reshape(g["count"], g["n"], 2)

    def _edges(self, g):
        X = self._of(g, self.X)
        return self._image(torch.roll(X, -1, 1) - X), X

    def _area(self, g):
        e, X = self._edges(g)
        U = torch.cat([X[:, :1], X[:, :1] + torch.cumsum(e, 1)[:, :-1]], 1)
        N = torch.roll(U, -1, 1)
        return (U[..., 0] * N[..., 1] - U[..., 1] * N[..., 0]).sum(1), e

    def _membrane(self):
        out = []
        for g in self.rings:
            sa, e = self._area(g)
            L = e.norm(dim=-1)
            t, L0 = e / L[..., None], g["L0"]
            if g["kind"] == "skalak":
                lam = L / L0
                T = self.G_s * lam * (lam * lam - 1) * (1 + 10.0)
            else:
                x0, Lm = 1 / 2.2, 2.2 * L0[:, :1]
                kp = self.G_s * Lm / (L0[:, :1] * (1 / (2 * (1 - x0) ** 3) + 1))
                kw = kp * (1 / (4 * (1 - x0) ** 2) - 0.25 + x0) * L0[:, :1]
                x = torch.clamp(L / (2.2 * L0), max=0.99)
                T = kp * (1 / (4 * (1 - x) ** 2) - 0.25 + x) - kw / L
            T = T + 0.1 * (L.sum(1) - g["P0"])[:, None] / g["P0"][:, None]     # perimeter
            if g["prev"] is not None:                                            # viscosity
                T = T + 0.05 * (L - g["prev"]) / L0
            g["prev"] = L
            F = T[..., None] * t
            F = F - torch.roll(F, 1, 1)
            ep = torch.roll(e, 1, 1)
            if g["kind"] == "wlc":
                dth = torch.atan2(ep[..., 0] * e[..., 1] - ep[..., 1] * e[..., 0], (ep * e).sum(-1)) - g["ang"]
                c = (-0.005 * dth / g["ds"])[..., None]
                gn = torch.stack([-e[..., 1], e[..., 0]], -1) / (e * e).sum(-1, True) * c
                gp = torch.stack([-ep[..., 1], ep[..., 0]], -1) / (ep * ep).sum(-1, True) * c
                F = F - gn - gp + torch.roll(gn, 1, 1) + torch.roll(gp, -1, 1)
            A = 0.5 * sa.abs()
            o = torch.stack([ep[..., 1] + e[..., 1], -ep[..., 0] - e[..., 0]], -1)
            o = o / o.norm(dim=-1, keepdim=True) * torch.where(sa >= 0, 1.0, -1.0)[:, None, None]
            F = F + o * (-0.5 * (A - g["A0"]) / g["A0"])[:, None, None]
            out.append((F - 0.01 * self._of(g, self.V)).reshape(-1, 2))
        return torch.cat(out)

    def _contact(self):
        X = self.X
        near = []
        for a in range(0, len(X), 4096):                     # rows of the pair table
            d = X[a:a + 4096, None, 0] - X[None, :, 0]
            d = d - self.nx * torch.round(d / self.nx)
            r2 = d * d + (X[a:a + 4096, None, 1] - X[None, :, 1]) ** 2
            i, j = torch.nonzero((r2 < 3.5 ** 2) & (self.cap[a:a + 4096, None] != self.cap[None]), as_tuple=True)
            near.append((i + a, j))
        i, j = (torch.cat(v) for v in zip(*near))
        F = torch.zeros_like(X)

        def push(d):
            r = d.norm(dim=-1, keepdim=True)
            return torch.where(r < 3.5, 0.05 * r ** -4 * d / r, torch.zeros_like(d))

        F.index_add_(0, i, push(self._image(X[i] - X[j])))
        for wall in (0.5, self.ny - 1.5):
            d = torch.zeros_like(X)
            d[:, 1] = X[:, 1] - wall
            F += torch.where(d[:, 1:].abs() < 1e-15, torch.zeros_like(d), push(d))
        return F

    # -- coupling
    def _phi(self, r):
        a = r.abs() * 512
        i = torch.clamp(a.long(), max=1023)
        w = a - i
        return torch.where(a >= 1024, torch.zeros_like(a), self.tab[i] * (1 - w) + self.tab[i + 1] * w)

    def _stencil(self):
        b = torch.floor(self.X).long()[:, None] + torch.arange(-1, 3, device=self.X.device)[None, :, None]
        w = self._phi(self.X[:, None] - b)                   # [m, 4, 2]
        rows = b[:, :, 1]
        W = w[:, :, None, 1] * w[:, None, :, 0]              # [m, y, x]
        W = torch.where(((rows >= 0) & (rows < self.ny))[:, :, None] & (W > 1e-15), W, torch.zeros_like(W))
        cell = rows.clamp(0, self.ny - 1)[:, :, None] * self.nx + (b[:, :, 0] % self.nx)[:, None, :]
        return W.reshape(len(self.X), 16), cell.reshape(len(self.X), 16)

    def _spread(self, F, frc, ds, st):
        W, cell = st
        for k in range(2):
            F[k].view(-1).index_add_(0, cell.reshape(-1), (W * (frc[:, k] * ds)[:, None]).reshape(-1))

    def _moments(self):
        rho = torch.where(self.solid, torch.ones_like(self.f[0]), self.f.sum(0))
        return rho, (self.cx * self.f).sum(0), (self.cy * self.f).sum(0)

    def _velocity(self, m, F):
        rho, jx, jy = m
        z = torch.zeros_like(rho)
        return torch.where(self.solid, z, (jx + 0.5 * F[0]) / rho), torch.where(self.solid, z, (jy + 0.5 * F[1]) / rho)

    def _interp(self, u, st):
        W, cell = st
        return torch.stack([(W * c.reshape(-1)[cell]).sum(1) for c in u], -1)

    def step(self):
        m = self._moments()
        G = self.F                                            # last step's force
        F = torch.zeros_like(self.F)
        if len(self.X):
            frc = self._membrane() + self._contact()
            ds = torch.cat([0.5 * (lambda L: L + torch.roll(L, 1, 1))(self._edges(g)[0].norm(dim=-1)).reshape(-1)
                            for g in self.rings])
            st = self._stencil()
            self._spread(F, frc, ds, st)
        if self.K > 1:
            G = F.clone()
        if len(self.X):
            near = (self.X + 0.5).long()
            at = near[:, 1].clamp(0, self.ny - 1) * self.nx + near[:, 0] % self.nx
            # SOLID nodes count as zero density
            rho_at = torch.where(self.solid, torch.zeros_like(m[0]), m[0]).reshape(-1)[at]
            for _ in range(1, self.K):
                G = F.clone()
                d = self.V - self._interp(self._velocity(m, F), st)
                self._spread(F, 2 * rho_at[:, None] * d, ds, st)
        F[0] += torch.where(self.solid, torch.zeros_like(F[0]), torch.full_like(F[0], self.fx))
        size = (F * F).sum(0)
        F = torch.where(size > 1e-4, F * 0.01 / torch.sqrt(size.clamp(min=1e-300)), F)
        ux, uy = self._velocity(m, G)
        f = self._collide(m[0], ux, uy, F)
        new = torch.stack([torch.roll(f[q], (_CY[q], _CX[q]), (0, 1)) for q in range(9)])
        for q in range(1, 9):
            new[_OPP[q]] = torch.where(self.into[q], f[q], new[_OPP[q]])
        self.f, self.F = new, F
        u = self._velocity(self._moments(), F)
        if self.scalar:
            eu = self.cx * u[0] + self.cy * u[1]
            g = self.g - (self.g - _vec(_W, self.f) * self.C * (1 + 3 * eu)) / (3 * self.scalar + 0.5)
            g = torch.where(self.solid, self.g, g)
            new = torch.stack([torch.roll(g[q], (_CY[q], _CX[q]), (0, 1)) for q in range(9)])
            for q in range(1, 9):
                new[_OPP[q]] = torch.where(self.into[q], g[q], new[_OPP[q]])
            self.g = torch.where(self.solid, self.g, new)
            self.C = self.g.sum(0)
        if len(self.X):
            self.V = self._interp(u, st)
            X = self.X + self.V
            X[:, 0] %= self.nx
            X[:, 1] = X[:, 1].clamp(1.5, self.ny - 1.5)
            self.X = X

    def _collide(self, rho, ux, uy, F):
        om = self.om
        fe = _feq(rho, ux, uy)
        if self.coll == "mrt":
            uu, uF = ux * ux + uy * uy, ux * F[0] + uy * F[1]
            z = torch.zeros_like(rho)
            mom = (self.M @ self.f.reshape(9, -1)).reshape(self.f.shape)
            eq = torch.stack([mom[0], rho * (-2 + 3 * uu), rho * (1 - 3 * uu), mom[3], -rho * ux, mom[5],
                              -rho * uy, rho * (ux * ux - uy * uy), rho * ux * uy])
            src = torch.stack([z, 6 * uF, -6 * uF, F[0], -F[0], F[1], -F[1],
                               2 * (ux * F[0] - uy * F[1]), ux * F[1] + uy * F[0]])
            s = _vec([0, 1.4, 1.4, 0, 1.4, 0, 1.4, om, om], rho)
            mom = mom - s * (mom - eq) + (1 - 0.5 * s) * src
            return (self.Mi @ mom.reshape(9, -1)).reshape(self.f.shape)
        eu = self.cx * ux + self.cy * uy
        src = (1 - 0.5 * om) * _vec(_W, rho) * (3 * ((self.cx - ux) * F[0] + (self.cy - uy) * F[1])
                                               + 9 * eu * (self.cx * F[0] + self.cy * F[1]))
        ne = self.f - fe
        if self.coll == "reg":
            cx, cy = self.cx, self.cy
            pxx, pxy, pyy = ((ne * c).sum(0) for c in (cx * cx, cx * cy, cy * cy))
            ne = _vec(_W, rho) * (3 * (cx * (ne * cx).sum(0) + cy * (ne * cy).sum(0)) + 4.5 * (
                (cx * cx - 1 / 3) * pxx + 2 * cx * cy * pxy + (cy * cy - 1 / 3) * pyy))
        return fe + (1 - om) * ne + src

    def fields(self):
        m = self._moments()
        u = self._velocity(m, self.F)
        rho = torch.where(self.solid, torch.zeros_like(m[0]), m[0])
        return [a.cpu().numpy() for a in (rho, u[0], u[1], self.F[0], self.F[1])]


def _seconds(nx, ny, sweeps, markers, steps, gpu):
    cells = nx * ny * (1.5e-9 if gpu else 5e-7) + (2e-2 if gpu else 6e-3) * (0.3 + 0.1 * sweeps)
    return steps * (cells + markers * markers * (1e-10 if gpu else 1.5e-8) + markers * sweeps * 1e-6)


def exact(case, seed):
    if case["kind"] == "spread":
        off, pos, frc = _rings(case, seed)
        n, k = case["capsules"], case["nodes"]
        ref = _Channel(case["nx"], case["ny"], "bgk", 0.8, 0.0, 1, [])
        ref.X = torch.tensor(pos)
        X = ref.X.reshape(n, k, 2)
        L = ref._image(torch.roll(X, -1, 1) - X).norm(dim=-1)
        F = torch.zeros((2, case["ny"], case["nx"]), dtype=torch.float64)
        ref._spread(F, torch.tensor(frc), (0.5 * (L + torch.roll(L, 1, 1))).reshape(-1), ref._stencil())
        return F[0].reshape(-1), F[1].reshape(-1)
    if case["kind"] == "network":
        # training in mixed precision has no 64-bit value of its own; the
        # loss, the weights and the predictions follow from it
        return None
    if case["kind"] == "channel":
        nx, ny, steps = case["nx"], case["ny"], case["steps"]
        caps = _capsules(case, seed)[0][0]
        gpu = torch.cuda.is_available() and nx * ny > 50000
        if _seconds(nx, ny, case["sweeps"], sum(SIZES[c[2]][1] for c in caps), steps, gpu) > 15:
            return None
        dev = "cuda" if gpu else "cpu"
        f = _fluid0(nx, ny, seed, "cuda" if torch.cuda.is_available() else "cpu")[0].to(dev)
        y, x = torch.meshgrid(torch.arange(ny, device=dev), torch.arange(nx, device=dev), indexing="ij")
        solid = torch.zeros((ny, nx), dtype=torch.bool, device=dev)
        for cx, cy, r in (_pillars(case, seed) if case["pillars"] else []):
            solid |= (x - cx) ** 2 + (y - cy) ** 2 <= r * r
        ref = _Channel(nx, ny, case["collision"], case["tau"], case["fx"], case["sweeps"], caps, f=f,
                       solid=solid, scalar=case["scalar"], device=dev,
                       C0=_gaussian(nx, ny, seed) if case["scalar"] else None)
        for _ in range(steps):
            ref.step()
        out = dict(zip(("rho", "ux", "uy", "Fx", "Fy"), ref.fields()))
        if case["skalak"] + case["wlc"]:
            out["pos"], out["vel"] = ref.X.cpu().numpy(), ref.V.cpu().numpy()
        if case["scalar"]:
            C0 = ref.C.clone()
            out["C"] = C0.cpu().numpy()
        return out
    chans = list(zip(_shapes(case), _capsules(case, seed)))
    cost = sum(_seconds(nx, ny, 5, 24 * n, case["steps"], False) for (nx, ny, n, _, _, _), _ in chans)
    if case["learned"] or not case["fields"] or cost > 15:
        return None
    out = {"pos": [], "vel": [], "thermo": None, "shapes": None, "fields": []}
    for (nx, ny, _, _, tau, fx), (caps, G_s) in chans:
        ref = _Channel(nx, ny, "reg", tau, fx, 5, caps, G_s)
        for _ in range(case["steps"]):
            ref.step()
        out["pos"].append(ref.X.reshape(-1).numpy())
        out["vel"].append(ref.V.reshape(-1).numpy())
        out["fields"].append(tuple(ref.fields()[:3]))
    out["pos"], out["vel"] = np.concatenate(out["pos"]), np.concatenate(out["vel"])
    return out
