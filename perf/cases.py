"""What is timed of this framework: the calls that its users make, over the range of sizes they make them.

Five kinds of work, each through the package's public entry points:

* ``rhs``       ``update_diagnostics``: one right-hand side, for callers that bring their own integrator;
                ``sparse``: the call also updates the elastic and sea-surface convolutions.
* ``couple``    a coupled ice-sheet model: sets its ice thickness, steps the integrator, reads the fields back.
* ``cycle``     a prescribed ice history with the elastic, viscous and sea-surface solves on, stepped through the
                coupling calls: the caller's displacement goes in, a step is taken, the fields come back.
* ``ensemble``  members of mixed grid sizes and mean viscosities stepped together.
* ``predict`` / ``train``  the surrogate of a macro-step: inference, and one training step with its gradients.

Grid sizes are 32 to 1024 cells a side (the configurations use 64 to 350, and 1024 for high resolution), square
and rectangular, with lengths that have factors other than 2, 3, 5 and 7 among them; surrogate grids are 32 to 256.
Every field is seeded here; ``exact`` is the same mathematics in 64 bits with torch.
"""
import math
import pathlib

import numpy as np
import torch

import __graft_entry__

__graft_entry__.load_package()
import fastiso_b200 as F  # noqa: E402

ROOT = pathlib.Path(__file__).resolve().parents[1]
SIDES = (64, 96, 128, 192, 256)  # member grids of an ensemble
T_END = 1e7                      # far beyond any sequence of passes


def listed():
    return [
        # the smallest call: one right-hand side on the smallest configured grid (latency, copies, launches)
        {"name": "rhs_64", "kind": "rhs", "nx": 64, "ny": 64, "cell": 46875.0, "sparse": False},
        # a right-hand side with both convolutions on the glacial-cycle grid
        {"name": "rhs_350_sparse", "kind": "rhs", "nx": 350, "ny": 350, "cell": 17142.0, "sparse": True},
        # an ice-sheet model coupled every 10 yr on a coarse grid: few attempts, so the call itself counts
        {"name": "couple_64", "kind": "couple", "nx": 64, "ny": 64, "cell": 46875.0, "years": 10.0, "form": "fp32"},
        # the same on a regional rectangular grid whose sides have factors 11 and 13
        {"name": "couple_165x130", "kind": "couple", "nx": 165, "ny": 130, "cell": 25000.0, "years": 10.0,
         "form": "fp32"},
        # the double-precision form, which runs the other rheologies and is the accuracy baseline
        {"name": "couple_128_fp64", "kind": "couple", "nx": 128, "ny": 128, "cell": 30000.0, "years": 10.0,
         "form": "fp64"},
        # the glacial-cycle grid, the configuration that throughput is quoted on
        {"name": "cycle_350", "kind": "cycle", "nx": 350, "ny": 350, "cell": 17142.0, "years": 20.0, "form": "fp32"},
        # high resolution
        {"name": "cycle_1024", "kind": "cycle", "nx": 1024, "ny": 1024, "cell": 5859.0, "years": 0.5, "form": "fp32"},
        # 128 members of mixed sizes, the ensemble configuration
        {"name": "ensemble_128", "kind": "ensemble", "members": 128, "years": 10.0},
        # surrogate rollouts: one member, and a screening pool's batch
        {"name": "predict_64_b1", "kind": "predict", "side": 64, "batch": 1},
        {"name": "predict_128_b32", "kind": "predict", "side": 128, "batch": 32},
        # surrogate training: the configured step, and a small ragged one
        {"name": "train_128_b32", "kind": "train", "side": 128, "batch": 32},
        {"name": "train_96_b7", "kind": "train", "side": 96, "batch": 7},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rhs", "couple", "cycle", "ensemble", "predict", "train"])
    if kind in ("rhs", "couple", "cycle"):
        nx = _log_int(rng, 32, 700)
        ny = nx if rng.random() < 0.4 else max(24, min(700, int(nx * rng.uniform(0.6, 1.6))))
        cell = float(round(rng.uniform(0.8, 1.5) * max(6e6 / max(nx, ny), 8000.0)))
        case = {"kind": kind, "nx": nx, "ny": ny, "cell": cell}
        if kind == "rhs":
            case["sparse"] = rng.random() < 0.5
        else:
            # some tens of attempts where the cells are small (the stable step falls with the cube of the cell)
            case["years"] = float("%.2g" % min(10.0, 6.0 * (cell / 17142.0) ** 3))
            case["form"] = "fp64" if kind == "couple" and max(nx, ny) <= 256 and rng.random() < 0.3 else "fp32"
        return case
    if kind == "ensemble":
        return {"kind": kind, "members": _log_int(rng, 2, 96), "years": float(rng.choice([5.0, 10.0]))}
    side = 32 * rng.randint(1, 8)
    most = max(1, 32 * 128 * 128 // (side * side))
    return {"kind": kind, "side": side, "batch": _log_int(rng, 1, min(most, 64))}


# ---------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------


def _random_field(nx, ny, cell, length, rng):
    """Gaussian random field of the given correlation length, zero mean and unit deviation, [nx, ny]."""
    w = np.fft.rfft2(rng.standard_normal((nx, ny)))
    kx = 2 * np.pi * np.fft.fftfreq(nx, d=cell)
    ky = 2 * np.pi * np.fft.rfftfreq(ny, d=cell)
    w *= np.exp(-(kx[:, None] ** 2 + ky[None, :] ** 2) * length ** 2 / 4)
    g = np.fft.irfft2(w, s=(nx, ny))
    g -= g.mean()
    return g / g.std()


def _earth(nx, ny, cell, rng, mean_log_eta=21.0, thickness=None):
    """Viscosity, lithosphere thickness and ice thickness, distributed as in the glacial-cycle configuration."""
    log_eta = np.clip(mean_log_eta + 0.5 * _random_field(nx, ny, cell, 500e3, rng), 19, 23)
    if thickness is None:
        thick = np.clip(120e3 + 40e3 * _random_field(nx, ny, cell, 500e3, rng), 50e3, 250e3)
    else:
        thick = np.full((nx, ny), thickness)
    ice = np.clip(1500 * np.maximum(_random_field(nx, ny, cell, 800e3, rng), 0), 0, 4000)
    return 10.0 ** log_eta, thick, ice


def _history(ice):
    """Ice switched on over the first year, then the rising limb of the sawtooth, one snapshot a kyr."""
    return [0.0, 1.0, 1000.0, 2000.0, 3000.0], [np.zeros_like(ice)] + [f * ice for f in (0.5, 0.51, 0.52, 0.53)]


def _inputs(case, seed):
    """The members' fields and options of a solver case: a list of dicts."""
    rng = np.random.Generator(np.random.PCG64(seed))
    if case["kind"] == "ensemble":
        out = []
        sides = np.random.Generator(np.random.PCG64(case["members"])).choice(SIDES, case["members"])
        for n in (int(v) for v in sides):
            eta, thick, ice = _earth(n, n, 30e3, rng, rng.uniform(20.0, 22.0), 100e3)
            out.append({"nx": n, "ny": n, "cell": 30e3, "eta": eta, "thick": thick, "ice": ice, "history": True,
                        "geoid": False, "form": "fp32"})
        return out
    nx, ny, cell = case["nx"], case["ny"], case["cell"]
    eta, thick, ice = _earth(nx, ny, cell, rng)
    m = {"nx": nx, "ny": ny, "cell": cell, "eta": eta, "thick": thick, "ice": ice, "geoid": True,
         "history": case["kind"] != "couple", "form": case.get("form", "fp32")}
    if case["kind"] in ("rhs", "cycle"):
        m["u"] = -60.0 * np.clip(_random_field(nx, ny, cell, 800e3, rng), -3, 3)
    return [m]


def _simulation(m):
    nx, ny = m["nx"], m["ny"]
    domain = F.RegionalDomain(0.5 * nx * m["cell"], 0.5 * ny * m["cell"], nx, ny)
    earth = F.SolidEarth(domain, layer_boundaries=m["thick"].reshape(nx, ny, 1),
                         layer_viscosities=m["eta"].reshape(nx, ny, 1))
    if m["history"]:
        t, h = _history(m["ice"])
        bcs = F.BoundaryConditions(domain, ice_thickness=F.TimeInterpolatedIceThickness(t, h, domain, flat_bc=True))
    else:
        bcs = F.BoundaryConditions(domain, ice_thickness=F.ExternallyUpdatedIceThickness())
    surface = F.LaterallyVariableSeaSurface() if m["geoid"] else F.LaterallyConstantSeaSurface()
    return F.Simulation(domain, bcs, F.RegionalSeaLevel(surface=surface), earth, (0.0, T_END), form=m["form"])


LIFT, MODES, WIDTH, HIDDEN, LAYERS = 6, 512, 32, 128, 4  # the surrogate's fixed shape


def _net_parameters(rng):
    """A network as training leaves it in size: pointwise layers 1/sqrt(fan in), spectral weights decaying."""
    def uniform(n, a):
        return rng.uniform(-a, a, n).astype(np.float32)

    parts = [uniform(WIDTH * LIFT, LIFT ** -0.5), uniform(WIDTH, LIFT ** -0.5)]
    for _ in range(LAYERS):
        parts += [uniform(MODES * 2 * WIDTH * WIDTH, 0.05), uniform(WIDTH * WIDTH, WIDTH ** -0.5),
                  uniform(WIDTH, WIDTH ** -0.5)]
    parts += [uniform(HIDDEN * WIDTH, WIDTH ** -0.5), uniform(HIDDEN, WIDTH ** -0.5),
              uniform(HIDDEN, HIDDEN ** -0.5), uniform(1, HIDDEN ** -0.5)]
    return np.concatenate(parts)


def _net_data(case, seed):
    """Parameters, and a batch: smooth displacement, ice, viscosity and thickness fields, and the coordinates."""
    s, b = case["side"], case["batch"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = 2 * math.pi * torch.fft.fftfreq(s, device="cuda", dtype=torch.float64) * s / 3.0
    low = torch.exp(-(k[:, None] ** 2 + k[None, :] ** 2) * 0.3 ** 2 / 4)
    f = torch.randn((b, 5, s, s), generator=g, device="cuda", dtype=torch.float64)
    f = torch.fft.ifft2(torch.fft.fft2(f) * low).real
    f = f / f.std(dim=(-2, -1), keepdim=True)
    c = torch.linspace(-1, 1, s, device="cuda", dtype=torch.float64)
    xy = torch.stack([c.expand(s, s), c[:, None].expand(s, s)]).expand(b, 2, s, s)
    x = torch.cat([f[:, :1], f[:, 1:2].clamp_min(0), f[:, 2:4], xy], dim=1).float().contiguous()
    target = (0.3 * f[:, 4]).float().contiguous()
    weights = (0.5 + torch.rand(b, generator=g, device="cuda")).contiguous()
    return _net_parameters(np.random.Generator(np.random.PCG64(seed))), x, target, weights


# ---------------------------------------------------------------------------------------------------------------
# the passes
# ---------------------------------------------------------------------------------------------------------------

LEARNING_RATE = 1e-4


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("predict", "train"):
        params, x, target, weights = _net_data(case, seed)
        net = F.FNO(S=case["side"], max_batch=case["batch"], seed=0)
        net.set_params(params)
        state = {"kind": kind, "net": net, "x": x, "target": target, "weights": weights}
        if kind == "train":
            state["grads"] = net.grads_tensor()
        return state
    members = _inputs(case, seed)
    sims = [_simulation(m) for m in members]
    state = {"kind": kind, "sims": sims, "years": case.get("years")}
    if kind == "rhs":
        sims[0].init_problem()
        # a time that opens the gate of the sparse update in every pass, or in none
        state.update(u=members[0]["u"], dudt=np.zeros_like(members[0]["u"]), t=9e6 if case["sparse"] else 5.0)
    elif kind == "ensemble":
        state["ensemble"] = F.Ensemble(sims)
    else:
        state["integrator"] = F.init_integrator(sims[0])
        if kind == "cycle":
            state["u"] = members[0]["u"]
        else:  # the ice model's margin goes forth and back from one exchange to the next
            state["ice"] = [members[0]["ice"], 0.8 * members[0]["ice"]]
    return state


def run(state):
    kind = state["kind"]
    if kind == "predict":
        return state["net"].forward(state["x"])
    if kind == "train":
        loss = state["net"].train_step(state["x"], state["target"], LEARNING_RATE, weights=state["weights"])
        return {"loss": loss, "grads": state["grads"].clone()}  # the view lives only as long as the network
    if kind == "rhs":
        F.update_diagnostics(state["dudt"], state["u"], state["sims"][0], state["t"])
        return {"u": state["u"], "dudt": state["dudt"]}
    if kind == "ensemble":
        status = state["ensemble"].step(state["years"])
        if any(status):
            raise RuntimeError("members failed: %s" % status)
        by_side = {}
        for sim in state["sims"]:
            by_side.setdefault(sim.domain.nx, []).append(sim.get_field("u"))
        return {"u_%d" % n: np.stack(u) for n, u in sorted(by_side.items())}
    sim = state["sims"][0]
    if kind == "cycle":
        sim.now.u = state["u"]
    else:
        sim.now.H_ice = state["ice"][0]
        state["ice"].reverse()
    F.step(state["integrator"], state["years"])
    return {"u": sim.now.u, "ue": sim.now.ue, "dz_ss": sim.now.dz_ss}


def work(case):
    kind = case["kind"]
    if kind in ("predict", "train"):
        s, b = case["side"], case["batch"]
        pixels = b * s * s
        params = 4 * (WIDTH * (LIFT + 1) + LAYERS * (MODES * 2 * WIDTH * WIDTH + WIDTH * (WIDTH + 1))
                      + HIDDEN * (WIDTH + 2) + 1)
        # multiply-adds of a pass forward: the truncated transforms both ways, the modes' channel mixing, the
        # pointwise layers, lift and projection
        layer = 2 * (pixels * WIDTH * 32 + b * WIDTH * 16 * 2 * s * 64) + b * MODES * 4 * WIDTH * WIDTH \
            + pixels * WIDTH * WIDTH
        forward = 2 * (LAYERS * layer + pixels * (LIFT * WIDTH + WIDTH * HIDDEN + HIDDEN))
        if kind == "predict":
            return {"bytes": params // 2 + 4 * pixels * (LIFT + 1), "flops": forward}
        # masters, both moments and the gradient read and written once
        return {"bytes": 8 * params + 4 * pixels * (LIFT + 1), "flops": 3 * forward}

    def rhs(nx, ny, geoid, sparse):
        n, pad = nx * ny, 4 * nx * ny
        flops = n * (120 + 10 * math.log2(n))
        moved = 48 * n
        if sparse:
            flops += (1 + geoid) * pad * 10 * math.log2(pad)
            moved += (1 + geoid) * (20 * pad + 8 * n)
        return moved, flops

    if kind == "rhs":
        moved, flops = rhs(case["nx"], case["ny"], 1, case["sparse"])
        return {"bytes": moved + 24 * case["nx"] * case["ny"], "flops": flops}
    if kind == "ensemble":
        per = [(n, n, 30e3, 1.2e20, 0) for n in SIDES for _ in range(max(1, case["members"] // len(SIDES)))]
    else:
        per = [(case["nx"], case["ny"], case["cell"], 2e20, 1)]
    total = {"bytes": 0.0, "flops": 0.0}
    for nx, ny, cell, eta, geoid in per:
        # attempts: the stable step of the flexure term, D k^3 / (2 eta), for the shortest wave on stiff ground
        rate = 1.2e25 * (2.0 / cell) ** 3 / (2 * eta) * 3.15576e7
        attempts = max(1.0, case["years"] * rate / 2.5)
        moved, flops = rhs(nx, ny, geoid, False)
        extra, more = rhs(nx, ny, geoid, True)
        updates = case["years"] / 10.0
        total["bytes"] += 3 * attempts * moved + updates * (extra - moved) + 24 * nx * ny
        total["flops"] += 3 * attempts * flops + updates * (more - flops)
    return total


# ---------------------------------------------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------------------------------------------


def _elastic_green(nx, ny, cell):
    """Elastic Green's function integrated over each cell, 4 x 4 Gauss-Legendre points on the Farrell table."""
    table = torch.from_numpy(np.loadtxt(ROOT / "fastisostasy.jl_b200/data/elasticgreencoeffs_farrell1972.txt")).cuda()
    rm, coeff = table[:, 1].contiguous(), table[:, 2].contiguous()
    points, weights = np.polynomial.legendre.leggauss(4)
    p = (torch.arange(nx, device="cuda", dtype=torch.float64) - nx // 2) * cell
    q = (torch.arange(ny, device="cuda", dtype=torch.float64) - ny // 2) * cell
    green = torch.zeros((ny, nx), device="cuda", dtype=torch.float64)
    for a, wa in zip(points, weights):
        for b, wb in zip(points, weights):
            x, y = p + 0.5 * cell * (a + 1), q + 0.5 * cell * (b + 1)
            r = torch.sqrt(x[None, :] ** 2 + y[:, None] ** 2)
            hi = torch.searchsorted(rm, r.contiguous(), right=True).clamp(1, rm.numel() - 1)
            w = (r - rm[hi - 1]) / (rm[hi] - rm[hi - 1])
            v = ((1 - w) * coeff[hi - 1] + w * coeff[hi]) / (r * 1e12)
            v = torch.where(r < 0.01, coeff[0] / (rm[1] * 1e12), v)
            v = torch.where(r > rm[-1], torch.zeros_like(v), v)
            green += v * wa * wb * (0.5 * cell) ** 2
    return green


def _fast_length(n):
    while True:
        r = n
        for p in (2, 3, 5, 7):
            while r % p == 0:
                r //= p
        if r == 1:
            return n
        n += 1


class _Reference:
    """Members of one grid, in 64 bits, [member, y, x]: the laterally variable ELVA right-hand side and the BS3
    integrator with its PI step-size control."""

    g, rho_ice, rho_sea, rho_litho, rho_mantle, nu = 9.8, 910.0, 1023.0, 3200.0, 3400.0, 0.28
    year, r_pole, mass = 60.0 ** 2 * 24 * 365.25, 6357e3, 5.972e24
    reltol, abstol, sparse_every = float(np.float32(1e-5)), 1e-6, 10.0

    def __init__(self, members):
        m = members[0]
        self.nx, self.ny, self.cell, self.geoid = m["nx"], m["ny"], m["cell"], m["geoid"]

        def stack(f):
            return torch.from_numpy(np.stack([np.ascontiguousarray(f(q).T) for q in members])).cuda()

        self.rigidity = 6.6e10 * stack(lambda q: q["thick"]) ** 3 / (12 * (1 - self.nu ** 2))
        self.eta = stack(lambda q: q["eta"]) * (1.5 / 1.28)
        ice = stack(lambda q: q["ice"])
        if m["history"]:
            self.times = _history(m["ice"])[0]
            self.snapshots = torch.stack([torch.zeros_like(ice)] + [f * ice for f in (0.5, 0.51, 0.52, 0.53)])
            self.external = None
        else:
            self.external = torch.zeros_like(ice)
        zero = torch.zeros_like(ice)
        wx, wy = 0.5 * self.nx * self.cell, 0.5 * self.ny * self.cell
        ix = torch.arange(self.nx // 2 + 1, device="cuda", dtype=torch.float64)
        iy = torch.fft.fftfreq(self.ny, device="cuda", dtype=torch.float64).abs() * self.ny
        k = torch.sqrt((math.pi / wx * ix[None, :]) ** 2 + (math.pi / wy * iy[:, None]) ** 2)
        k[0, 0] = 1.0
        self.inverse_k = 1.0 / k
        self.inverse_k[0, 0] = 0.0  # the corner condition takes a constant out again
        self.pad = (_fast_length(2 * self.ny - 1), _fast_length(2 * self.nx - 1))
        self.green_e = torch.fft.rfft2(_elastic_green(self.nx, self.ny, self.cell), s=self.pad)
        x = -wx + (torch.arange(self.nx, device="cuda", dtype=torch.float64) + 1) * self.cell
        y = -wy + (torch.arange(self.ny, device="cuda", dtype=torch.float64) + 1) * self.cell
        r = torch.sqrt(x[None, :] ** 2 + y[:, None] ** 2)
        cap = self.r_pole / (2 * self.mass * math.sin(self.cell / 2 / (2 * self.r_pole)))
        green = self.r_pole / (2 * self.mass * torch.sin(r / (2 * self.r_pole)))
        self.green_g = torch.fft.rfft2(green.clamp(max=cap), s=self.pad)
        b = len(members)
        self.u, self.ue, self.dz = zero, zero.clone(), zero.clone()
        self.load, self.full = zero.clone(), zero.clone()
        self.count = torch.zeros(b, device="cuda", dtype=torch.float64)
        self.t = torch.zeros(b, device="cuda", dtype=torch.float64)
        self.rhs(self.u, self.t, torch.ones(b, dtype=torch.bool, device="cuda"))

    @staticmethod
    def pick(on, a, b):
        return torch.where(on.reshape(-1, *[1] * (a.ndim - 1)), a, b)

    @staticmethod
    def corners(v):
        return v - 0.25 * (v[:, :1, :1] + v[:, :1, -1:] + v[:, -1:, :1] + v[:, -1:, -1:])

    def convolve(self, v, green):
        full = torch.fft.irfft2(torch.fft.rfft2(v, s=self.pad) * green, s=self.pad)
        full = self.corners(full[:, :2 * self.ny - 1, :2 * self.nx - 1])
        i, j = (self.nx - 1) // 2, (self.ny - 1) // 2  # the crop window of a same-size convolution
        return full[:, j:j + self.ny, i:i + self.nx]

    def ice(self, t):
        if self.external is not None:
            return self.external
        times = torch.tensor(self.times, device="cuda", dtype=torch.float64)
        hi = torch.searchsorted(times, t).clamp(1, len(self.times) - 1)
        w = ((t - times[hi - 1]) / (times[hi] - times[hi - 1])).clamp(0, 1)[:, None, None]
        rows = torch.arange(t.numel(), device="cuda")
        a, b = self.snapshots[hi - 1, rows], self.snapshots[hi, rows]
        return a + (b - a) * w

    def second(self, v, dim):
        inner = v.narrow(dim, 2, v.shape[dim] - 2) - 2 * v.narrow(dim, 1, v.shape[dim] - 2) \
            + v.narrow(dim, 0, v.shape[dim] - 2)
        return torch.cat([inner.narrow(dim, 0, 1), inner, inner.narrow(dim, inner.shape[dim] - 1, 1)],
                         dim) / self.cell ** 2

    def first(self, v, dim):
        n = v.shape[dim]
        inner = (v.narrow(dim, 2, n - 2) - v.narrow(dim, 0, n - 2)) / 2
        left = v.narrow(dim, 1, 1) - v.narrow(dim, 0, 1)
        right = v.narrow(dim, n - 1, 1) - v.narrow(dim, n - 2, 1)
        return torch.cat([left, inner, right], dim) / self.cell

    def rhs(self, u, t, on):
        """(u with its corner condition, du/dt) of the members that are on, with the call's effects on their state."""
        u = self.corners(u)
        bed = 1e6 + self.ue + u
        ice = self.ice(t)
        gate = on & (t / self.sparse_every >= self.count)
        if bool(gate.any()):
            self.ue = self.pick(gate, self.convolve(self.load, self.green_e), self.ue)
            if self.geoid:
                self.dz = self.pick(gate, self.convolve(self.full * self.cell ** 2, self.green_g), self.dz)
            self.count = self.count + gate
        above = (ice + (bed - self.dz).clamp(max=0) * (self.rho_sea / self.rho_ice)).clamp_min(0)
        load = self.rho_ice * above
        full = load + self.rho_litho * self.ue + self.rho_mantle * u
        self.load, self.full = self.pick(on, load, self.load), self.pick(on, full, self.full)
        uxx, uyy = self.second(u, 2), self.second(u, 1)
        uxy = self.first(self.first(u, 2), 1)
        mxx = -self.rigidity * (self.nu * uyy + uxx)
        myy = -self.rigidity * (self.nu * uxx + uyy)
        mxy = -self.rigidity * (1 - self.nu) * uxy
        f = -self.g * full + self.second(mxx, 2) + 2 * self.first(self.first(mxy, 2), 1) + self.second(myy, 1)
        f = torch.fft.irfft2(torch.fft.rfft2(f / (2 * self.eta)) * self.inverse_k, s=(self.ny, self.nx))
        return u, self.corners(f * self.year)

    def rms(self, v):
        return torch.sqrt((v ** 2).mean(dim=(1, 2)))

    def start(self):
        """The first derivative and the step to begin with."""
        on = torch.ones_like(self.t, dtype=torch.bool)
        self.u, self.k1 = self.rhs(self.u, self.t, on)
        _, f0 = self.rhs(self.u, self.t, on)
        sk = self.abstol + self.u.abs() * self.reltol
        d0, d1 = self.rms(self.u / sk), self.rms(f0 / sk)
        small = (d0 < 1e-5) | (d1 < 1e-5)
        first = torch.where(small, torch.full_like(d0, 1e-6), d0 / d1.clamp_min(1e-300) / 100)
        _, f1 = self.rhs(self.u + first[:, None, None] * f0, self.t + first, on)
        d2 = self.rms((f1 - f0) / sk) / first
        most = torch.maximum(d1, d2)
        second = torch.where(most <= 1e-15, (first * 1e-3).clamp_min(1e-6),
                             10 ** (-(2 + torch.log10(most.clamp_min(1e-300))) / 3))
        same = ((f1 == f0).flatten(1)).all(dim=1)
        self.dt = torch.where(same, 100 * first, torch.minimum(100 * first, second))
        self.last = torch.full_like(self.t, 1e-4)

    def advance(self, years):
        """BS3 steps of every member from its time to `years` later."""
        stop = self.t + years
        col = lambda v: v[:, None, None]  # noqa: E731
        while True:
            on = self.t < stop
            if not bool(on.any()):
                return
            dt = torch.where(on, torch.minimum(self.dt, stop - self.t), self.dt)
            _, k2 = self.rhs(self.u + col(dt * 0.5) * self.k1, self.t + 0.5 * dt, on)
            _, k3 = self.rhs(self.u + col(dt * 0.75) * k2, self.t + 0.75 * dt, on)
            new = self.u + col(dt) * (2 / 9 * self.k1 + 1 / 3 * k2 + 4 / 9 * k3)
            new, k4 = self.rhs(new, self.t + dt, on)
            err = col(dt) * (-5 / 72 * self.k1 + 1 / 12 * k2 + 1 / 9 * k3 - 1 / 8 * k4)
            err = self.rms(err / (self.abstol + torch.maximum(self.u.abs(), new.abs()) * self.reltol))
            power = err ** (7 / 30)
            q = torch.where(err == 0, torch.full_like(err, 0.1),
                            (power / self.last ** (2 / 15) / 0.9).clamp(0.1, 5.0))
            accepted = on & (err <= 1)
            rejected = on & ~accepted
            self.t = torch.where(accepted, torch.where(stop - (self.t + dt) < 1e-9, stop, self.t + dt), self.t)
            self.last = torch.where(accepted, err.clamp_min(1e-4), self.last)
            self.dt = torch.where(accepted, dt / q, torch.where(rejected, dt / (power / 0.9).clamp(max=5.0), self.dt))
            self.u = self.pick(accepted, new, self.u)
            self.k1 = self.pick(accepted, k4, self.k1)


def _exact_net(case, seed):
    params, x, target, weights = _net_data(case, seed)
    s, b = case["side"], case["batch"]
    p = torch.from_numpy(params).cuda().double().requires_grad_(case["kind"] == "train")
    at = 0

    def take(*shape):
        nonlocal at
        n = math.prod(shape)
        at += n
        return p[at - n:at].reshape(shape)

    ky = torch.tensor([k if k < 16 else s - 32 + k for k in range(32)], device="cuda")
    v = torch.einsum("ci,biyx->bcyx", take(WIDTH, LIFT), x.double()) + take(WIDTH)[:, None, None]
    for layer in range(LAYERS):
        w = take(16, 32, 2, WIDTH, WIDTH)
        local, bias = take(WIDTH, WIDTH), take(WIDTH)
        modes = torch.fft.rfft2(v)[:, :, ky, :16]
        mixed = torch.einsum("bcyx,xyco->boyx", modes, torch.complex(w[:, :, 0], w[:, :, 1]))
        half = torch.zeros((b, WIDTH, s, 16), device="cuda", dtype=torch.complex128).index_copy(2, ky, mixed)
        half = torch.nn.functional.pad(half, (0, s // 2 + 1 - 16))
        z = torch.fft.irfft(torch.fft.ifft(half, dim=2), n=s, dim=3) + bias[:, None, None] \
            + torch.einsum("oc,bcyx->boyx", local, v)
        v = torch.nn.functional.gelu(z) if layer < LAYERS - 1 else z
    a = torch.einsum("jc,bcyx->bjyx", take(HIDDEN, WIDTH), v) + take(HIDDEN)[:, None, None]
    y = torch.einsum("j,bjyx->byx", take(HIDDEN), torch.nn.functional.gelu(a)) + take(1)
    if case["kind"] == "predict":
        return y.detach()
    loss = (weights.double()[:, None, None] * (y - target.double()) ** 2).mean()
    loss.backward()
    return {"loss": float(loss.detach()), "grads": p.grad}


def exact(case, seed):
    if case["kind"] in ("predict", "train"):
        return _exact_net(case, seed)
    members = _inputs(case, seed)
    out = lambda v: v.transpose(-1, -2).contiguous().cpu().numpy()  # noqa: E731
    if case["kind"] == "ensemble":
        result = {}
        for n in SIDES:
            group = [m for m in members if m["nx"] == n]
            if group:
                ref = _Reference(group)
                ref.start()
                ref.advance(case["years"])
                result["u_%d" % n] = out(ref.u)
        return result
    ref = _Reference(members)
    if case["kind"] == "rhs":
        u = torch.from_numpy(np.ascontiguousarray(members[0]["u"].T)).cuda()[None]
        t = torch.full_like(ref.t, 9e6 if case["sparse"] else 5.0)
        u, dudt = ref.rhs(u, t, torch.ones_like(t, dtype=torch.bool))
        return {"u": out(u[0]), "dudt": out(dudt[0])}
    ref.start()
    if case["kind"] == "cycle":
        ref.u = torch.from_numpy(np.ascontiguousarray(members[0]["u"].T)).cuda()[None]
        ref.u, ref.k1 = ref.rhs(ref.u, ref.t, torch.ones_like(ref.t, dtype=torch.bool))
    else:
        ref.external = torch.from_numpy(np.ascontiguousarray(members[0]["ice"].T)).cuda()[None]
    ref.advance(case["years"])
    return {"u": out(ref.u[0]), "ue": out(ref.ue[0]), "dz_ss": out(ref.dz[0])}
