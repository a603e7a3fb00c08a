"""Performance cases: blocks of time steps as a simulation program runs them.

A program creates a lattice, uploads its initial state, and then advances it in blocks of
some hundred to some thousand steps, reading the hydrodynamic fields (and the particles)
back after each block.  `prepare` is everything before the first block, `run` is one block
and its read-back, `exact` is the same block in plain FP64 torch.

    listed()  the cases;  draw(rng)  one more of the same ranges
    prepare(case, seed), run(state), exact(case, seed)
    work(case)  the bytes and operations a block cannot do without
    tolerance(case)  how far another correct implementation may be off
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ch4-project_b200"))

import ch4b200  # noqa: E402
from ch4b200 import abi  # noqa: E402

STORES = {"f64": abi.STORE_F64, "f32": abi.STORE_F32, "f16": abi.STORE_F16}
BYTES = {"f64": 8, "f32": 4, "f16": 2}
W = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
CX = [0, 1, -1, 0, 0, 0, 0, 1, 1, -1, -1, 1, -1, 1, -1, 0, 0, 0, 0]
CY = [0, 0, 0, 1, -1, 0, 0, 1, -1, 1, -1, 0, 0, 0, 0, 1, 1, -1, -1]
CZ = [0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, 1, -1, -1, 1, -1, 1, -1]
INV = [[i for i in range(19) if (CX[i], CY[i], CZ[i]) == (-CX[q], -CY[q], -CZ[q])][0] for q in range(19)]
VK = [(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (0, 1, 1), (1, 0, 1)]  # HIT forcing modes
PI2 = 2 * 3.14159265359  # the solver's constant


def listed():
    return [
        # the smallest served request: a 32^3 Kolmogorov cube, every step a launch
        _case("kolmogorov_32_f32", "kolmogorov", 32, 32, 32, "f32", 1000),
        # the validation run: 64^3 Kolmogorov flow in FP64, tau 0.6, 2000 steps
        _case("kolmogorov_64_f64", "kolmogorov", 64, 64, 64, "f64", 2000),
        # Rayleigh-Benard convection at the headline size and Rayleigh number
        _case("rb_256x256x128_f32", "rb", 256, 256, 128, "f32", 1000, Ra=1e8),
        # a parity run in FP64 on a ragged lattice
        _case("rb_129x97x75_f64", "rb", 129, 97, 75, "f64", 500, Ra=1e6),
        # the half-precision population store
        _case("rb_200x150x90_f16", "rb", 200, 150, 90, "f16", 1000, Ra=1e6),
        # temperature and a scalar carried together (three population sets)
        _case("rb_scalar_110x96x100_f32", "rb", 110, 96, 100, "f32", 600, Ra=1e6, scalar=True),
        # served Rayleigh-Benard cube with Smagorinsky LES
        _case("rb_les_128_f32", "rb", 128, 128, 128, "f32", 800, Ra=1e6, les=True),
        # served Kolmogorov cube with Smagorinsky LES and tracers
        _case("kolmogorov_les_96_tracers_f32", "kolmogorov", 96, 96, 96, "f32", 600, les=True, particles=40000),
        # forced turbulence with two-way coupled inertial particles, one per 16 cells
        _case("hit_160_twoway_f32", "hit", 160, 160, 160, "f32", 600, particles=250000, twoway=True),
        # the same physics in FP64 on a small ragged lattice, as a parity study runs it
        _case("hit_60x50x70_twoway_f64", "hit", 60, 50, 70, "f64", 400, particles=15000, twoway=True),
        # a parameter sweep: 48 quasi-2-D convection cells of mixed sizes advanced together
        _ensemble("ensemble_48_f32", 48, 4, "f32", 1200),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["kolmogorov", "rb", "rb", "rb_scalar", "rb_les", "tracers", "hit", "ensemble"])
    if kind == "ensemble":
        return _ensemble(None, rng.randint(8, 48), rng.randint(5, 1 << 20), "f32", rng.randint(300, 1200))
    nx, ny, nz = size(24, 180), size(24, 180), size(24, 180)
    while nx * ny * nz > 3000000:
        nx, ny, nz = size(24, 180), size(24, 180), size(24, 180)
    steps = rng.randint(300, 1000)
    flow = "kolmogorov" if kind == "tracers" else kind.split("_")[0]
    storage = rng.choice(["f64", "f32", "f32", "f16"] if kind in ("kolmogorov", "rb") else ["f32", "f32", "f64"])
    more = {}
    if flow == "rb":
        more["Ra"] = 10 ** rng.uniform(4, 2 * math.log10(12.5 * ny))  # nu >= 0.004
    if kind == "rb_scalar":
        more["scalar"] = True
    if kind in ("rb_les", "tracers"):
        more["les"] = True
    if kind == "tracers":
        more["particles"] = size(5000, 60000)
    if kind == "hit":
        more.update(particles=max(1000, nx * ny * nz // rng.randint(12, 30)), twoway=True)
        steps = min(steps, 700)
    return _case(None, flow, nx, ny, nz, storage, steps, **more)


def _case(name, flow, nx, ny, nz, storage, steps, Ra=0.0, les=False, scalar=False, particles=0, twoway=False):
    c = {"flow": flow, "NX": nx, "NY": ny, "NZ": nz, "storage": storage, "steps": steps, "Ra": float(Ra), "les": les,
         "scalar": scalar, "particles": particles, "twoway": twoway}
    return dict(c, name=name) if name else c


def _ensemble(name, lattices, sizes, storage, steps):
    c = {"flow": "ensemble", "lattices": lattices, "sizes": sizes, "storage": storage, "steps": steps}
    return dict(c, name=name) if name else c


def _members(case):
    """The lattices of an ensemble: 64 x 64 .. 512 x 256 log-uniform, Ra 1e5 .. 1e7."""
    rng = np.random.default_rng(case["sizes"])
    out = []
    for _ in range(case["lattices"]):
        nx = int(round(math.exp(rng.uniform(math.log(64), math.log(512)))))
        ny = int(round(math.exp(rng.uniform(math.log(64), math.log(256)))))
        ra = math.exp(rng.uniform(math.log(1e5), math.log(min(1e7, (12.5 * ny) ** 2))))
        out.append(_case(None, "rb", nx, ny, 1, case["storage"], case["steps"], Ra=ra))
    return out


# ---- the programs' configurations and inputs --------------------------------

def _config(case, seed):
    c = ch4b200.default_config()
    c.NX, c.NY, c.NZ = case["NX"], case["NY"], case["NZ"]
    c.SX, c.SY, c.SZ = float(c.NX), float(c.NY), float(c.NZ)
    c.time_dt = c.time_dt_lagr_factor = 1.0
    c.storage = STORES[case["storage"]]
    c.C_smag = 0.17
    c.seed = 1 + seed % (1 << 30)
    names = ["LB_FLUID", "LB_FLUID_FORCING"]
    if case["flow"] == "kolmogorov":  # F_x = 1e-5 sin(2 pi y / L)
        names.append("LB_FLUID_FORCING_KOLMOGOROV")
        c.tau_u = 0.6
        c.Amp_x = 1e-5 / ((c.tau_u - 0.5) / 3.0 * (PI2 / c.NY) ** 2)
    elif case["flow"] == "rb":  # free-fall velocity 0.05, Pr 1
        names += ["LB_FLUID_BC_Y", "LB_TEMPERATURE", "LB_TEMPERATURE_BUOYANCY", "LB_TEMPERATURE_BC_Y"]
        bg = 0.05 ** 2 / c.NY
        nu = (bg * c.NY ** 3 / case["Ra"]) ** 0.5
        c.tau_u = c.tau_t = 0.5 + 3 * nu
        c.beta_t, c.gravity_y, c.T_bot, c.T_top, c.T_ref = 1.0, bg, 1.0, 0.0, 0.0
        c.deltaT = 1.0
        if case["scalar"]:  # a second component, fresher on top, stabilising
            names += ["LB_SCALAR", "LB_SCALAR_BUOYANCY", "LB_SCALAR_BC_Y"]
            c.tau_s, c.beta_s = 0.5 + 0.6 * (c.tau_u - 0.5), 0.3
            c.S_bot, c.S_top, c.S_ref, c.deltaS = 0.0, 1.0, 0.0, 1.0
    else:  # forced homogeneous isotropic turbulence
        names.append("LB_FLUID_FORCING_HIT")
        c.tau_u = 0.51
        c.Amp_x = c.Amp_y = c.Amp_z = 5e-6
    if case["les"]:
        names.append("LB_FLUID_LES")
    if case["particles"]:
        names += ["LAGRANGE", "LAGRANGE_WRAP"]
    if case["twoway"]:
        names += ["LAGRANGE_GRADIENT", "LAGRANGE_ADDEDMASS", "LAGRANGE_TWOWAY", "LAGRANGE_TWOWAY_MOMENTUM"]
    abi.set_flags(c, names)
    c.nu = (c.tau_u - 0.5) / 3.0
    c.kappa = (c.tau_t - 0.5) / 3.0
    c.chi = (c.tau_s - 0.5) / 3.0
    return c


def _inputs(case, seed):
    """Populations as (19, NZ, NY, NX) FP64 tensors on the GPU, and the particle records."""
    nx, ny, nz = case["NX"], case["NY"], case["NZ"]
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def rand(*shape):
        return torch.rand(*shape, generator=gen, device="cuda", dtype=torch.float64)

    def line(n):
        return (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n

    x, y, z = line(nx)[None, None, :], line(ny)[None, :, None], line(nz)[:, None, None]
    u = 1e-4 * (2 * rand(3, nz, ny, nx) - 1)
    pops = {}
    if case["flow"] == "rb":  # the conductive profile, a convection roll and noise
        ph = 2 * math.pi * rand(1)
        u[0] += 0.02 * torch.sin(2 * math.pi * x + ph) * torch.sin(2 * math.pi * y)
        u[1] += 0.02 * ny / nx * torch.cos(2 * math.pi * x + ph) * (torch.cos(2 * math.pi * y) - 1)
        pops["g"] = (1.0 - y) + 1e-3 * (2 * rand(nz, ny, nx) - 1)
        if case["scalar"]:
            pops["h"] = y + 1e-3 * (2 * rand(nz, ny, nx) - 1)
    elif case["flow"] == "hit":  # large-scale solenoidal modes
        for a, b, pos in ((0, 1, y), (1, 2, z), (2, 0, x), (0, 2, z), (1, 0, x), (2, 1, y)):
            u[a] += 0.01 * torch.sin(2 * math.pi * pos + 2 * math.pi * rand(1))
    u2 = (u * u).sum(0)
    moments = dict(p=1.0, **pops)
    pops = {k: torch.empty(19, nz, ny, nx, device="cuda", dtype=torch.float64) for k in moments}
    for q in range(19):
        cu = CX[q] * u[0] + CY[q] * u[1] + CZ[q] * u[2]
        poly = W[q] * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * u2)
        for k, m in moments.items():
            pops[k][q] = m * poly
    n = case["particles"]
    rec = None
    if n:
        rng = np.random.default_rng(seed)
        rec = np.zeros((n, len(abi.PARTICLE_FIELDS)))  # name, tau_drag, beta_coeff, x, y, z, ...
        rec[:, 0] = np.arange(n)
        rec[:, 3:6] = rng.random((n, 3)) * (nx, ny, nz)
        if case["twoway"]:  # tracers and nine Stokes classes (beta, tau_p)
            kind = np.arange(n) % 10
            stokes = kind > 0
            rec[stokes, 2] = np.array([0.0, 1.0, 3.0])[(kind[stokes] - 1) % 3]
            tau = np.array([4.0, 8.0, 12.0])[(kind[stokes] - 1) // 3]
            # (larger bubbles: the explicit two-way coupling is unstable)
            rec[stokes, 1] = np.where(rec[stokes, 2] == 3.0, 4.0, tau)
    return pops, rec


def _aos(t):
    return t.permute(1, 2, 3, 0).contiguous().cpu().numpy()


def prepare(case, seed):
    if case["flow"] == "ensemble":
        ens = ch4b200.Ensemble(STORES[case["storage"]])
        slots = []
        for i, m in enumerate(_members(case)):
            s = ens.add(_config(m, seed))
            for k, v in _inputs(m, 1000 * seed + i)[0].items():
                ens.set_pop(s, k, _aos(v))
            ens.initialize(s)
            slots.append(s)
        ens.tune()
        return {"case": case, "ens": ens, "slots": slots}
    cfg = _config(case, seed)
    pops, rec = _inputs(case, seed)
    sim = ch4b200.Simulation(cfg)
    for k in list(pops):
        sim.set_pop(k, _aos(pops.pop(k)))
    if rec is not None:
        sim.set_particles((abi.Particle * len(rec)).from_buffer(rec))
    sim.initialize()
    return {"case": case, "sim": sim}


# the particle state a program keeps of the records.  (Not the accelerations: differences
# of consecutive velocities, with a rounding some hundred times theirs; the velocities,
# integrated from them, carry them.)
COLUMNS = {"velocity": ["vx", "vy", "vz"], "fluid_velocity": ["ux", "uy", "uz"]}
COLUMNS_TWOWAY = dict(COLUMNS, gradient=["dx_ux", "dy_ux", "dz_ux", "dx_uy", "dy_uy", "dz_uy", "dx_uz", "dy_uz",
                                         "dz_uz"])


def run(state):
    case = state["case"]
    if case["flow"] == "ensemble":
        ens = state["ens"]
        ens.step(case["steps"])
        fields = [ens.fields(s) for s in state["slots"]]
        return {k: np.concatenate([f[k].reshape(-1) for f in fields]) for k in ("dens", "u", "t")}
    sim = state["sim"]
    sim.step(case["steps"])
    f = sim.fields()
    out = {k: f[k] for k in _names(case)}
    if case["particles"]:
        rec = np.frombuffer(sim.get_particles(case["particles"]), dtype=np.float64)
        rec = rec.reshape(case["particles"], len(abi.PARTICLE_FIELDS))
        for k, cols in (COLUMNS_TWOWAY if case["twoway"] else COLUMNS).items():
            i = abi.PARTICLE_FIELDS.index(cols[0])
            out[k] = rec[:, i:i + len(cols)]
        i = abi.PARTICLE_FIELDS.index("x")
        out["position"] = _circle(rec[:, i:i + 3], (case["NX"], case["NY"], case["NZ"]))
    return out


def _circle(x, size):
    """Positions in the periodic box as two triangle waves per axis, which (unlike x) are
    continuous where a particle leaves through one face and enters through the other."""
    s = x / np.array(list(size), dtype=np.float64)
    a = np.abs(s - 0.5)
    s += 0.25
    s -= np.floor(s)
    return np.concatenate([a, np.abs(s - 0.5)], axis=1)


def _names(case):
    return ["dens", "u"] + (["t"] if case["flow"] == "rb" else []) + (["s"] if case["scalar"] else [])


def work(case):
    """Per step every population once in and once out (and the particles' state); the
    fields out once.  Operations: some 300 per cell for the fluid, 120 for a passive set."""
    if case["flow"] == "ensemble":
        each = [work(m) for m in _members(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    cells, steps = case["NX"] * case["NY"] * case["NZ"], case["steps"]
    sets = len(_names(case)) - 1
    particle = (2 * 15 + 2) * 8 if case["twoway"] else (2 * 6 + 2) * 8
    return {"bytes": steps * (cells * 2 * 19 * BYTES[case["storage"]] * sets + case["particles"] * particle)
            + 8 * cells * (sets + 3),
            "flops": steps * (cells * (300.0 + 120.0 * (sets - 1) + (150.0 if case["les"] else 0.0))
                              + case["particles"] * 600.0)}


def tolerance(case):
    """About four times what the solver is off `exact` (below)."""
    if case["storage"] == "f64":
        return {"rel": 4e-12}
    if case["storage"] == "f16":
        return {"rel": 6e-3}
    return {"rel": 1e-3 if case.get("twoway") else 3e-4}


# ---- the same block in plain FP64 torch -------------------------------------

def exact(case, seed):
    if case["flow"] == "ensemble":
        parts = [_Exact(m, seed, 1000 * seed + i).block() for i, m in enumerate(_members(case))]
        return {k: np.concatenate([p[k].reshape(-1) for p in parts]) for k in ("dens", "u", "t")}
    if case["NX"] * case["NY"] * case["NZ"] * case["steps"] > 5e9:
        return None  # some 20 seconds
    return _Exact(case, seed, seed).block()


class _Exact:
    """The lattice-Boltzmann step (BGK, Guo forcing with the force of the previous step in
    the velocity, halfway walls on y) and the particles, as array operations."""

    def __init__(self, case, seed, input_seed):
        self.case, self.cfg = case, _config(case, seed)
        pops, rec = _inputs(case, input_seed)
        self.f, self.g, self.h = pops["p"], pops.get("g"), pops.get("h")
        self.shape = (case["NZ"], case["NY"], case["NX"])
        d = dict(device="cuda", dtype=torch.float64)
        self.d = d
        self.C = torch.tensor([CX, CY, CZ], **d)
        self.w = torch.tensor(W, **d)[:, None, None, None]
        self.T = None if self.g is None else self.g.sum(0)
        self.S = None if self.h is None else self.h.sum(0)
        self.rng = ((self.cfg.seed & 0xFFFFFFFF) << 16) | 0x330E
        self.tables = None
        if case["flow"] == "hit":
            self.phi = [[self.uniform() for _ in range(3)] for _ in VK]
            self.tables = self.walk()
        self.kol = None
        if case["flow"] == "kolmogorov":
            y = torch.arange(case["NY"], **d) + 0.5
            self.kol = 1e-5 * torch.sin(PI2 * y / case["NY"])[None, :, None]
        self.part = None if rec is None else _ExactParticles(self, rec)
        self.dep = self.dep_prev = None

    def uniform(self):  # drand48
        self.rng = (0x5DEECE66D * self.rng + 0xB) & ((1 << 48) - 1)
        return self.rng / float(1 << 48)

    def gauss(self):
        while True:
            a, b = -1 + 2 * self.uniform(), -1 + 2 * self.uniform()
            r = a * a + b * b
            if 0 < r < 1:
                return a * math.sqrt(-2 * math.log(r) / r)

    def walk(self):
        """One step of the phases' random walk; the force component along each axis pair."""
        turn = self.case["NX"] / 0.1
        noise = math.sqrt(2.0 * 0.01 / turn)
        for p in self.phi:
            for a in range(3):
                p[a] += -p[a] / turn + self.gauss() * noise
        n = [self.case["NX"], self.case["NY"], self.case["NZ"]]
        phi, k = torch.tensor(self.phi, **self.d), torch.tensor(VK, **self.d)
        amp = 5e-6 * k.square().sum(1) ** (-1 / 3)
        view = [(1, 1, n[0]), (1, n[1], 1), (n[2], 1, 1)]
        s = []
        for a in range(3):
            x = (torch.arange(n[a], **self.d) + 0.5) / n[a]
            s.append((amp[:, None] * torch.sin(PI2 * (k[:, a:a + 1] * x + phi[:, a:a + 1]))).sum(0).reshape(view[a]))
        return s

    def force(self, T, S, tables, dep):
        F = [torch.zeros((), **self.d)] * 3
        if self.kol is not None:
            F[0] = F[0] + self.kol
        if tables is not None:
            F = [F[0] + tables[1] + tables[2], F[1] + tables[0] + tables[2], F[2] + tables[1] + tables[0]]
        c = self.cfg
        if T is not None:
            F[1] = F[1] + c.beta_t * (T - 0.5 * (c.T_bot + c.T_top)) * c.gravity_y
        if S is not None:
            F[1] = F[1] + c.beta_s * (S - 0.5 * (c.S_bot + c.S_top)) * c.gravity_y
        F = torch.stack([v.expand(self.shape) for v in F])
        return F if dep is None else F + dep

    def velocity(self, F):
        rho = self.f.sum(0)
        return rho, (self.C @ self.f.reshape(19, -1)).reshape(3, *self.shape) / rho + 0.5 * F

    def smagorinsky(self, u):
        g = []
        for axis in (2, 1, 0):  # x, y, z
            d = (torch.roll(u, -1, axis + 1) - torch.roll(u, 1, axis + 1)) / 2
            if axis == 1 and self.case["flow"] == "rb":  # one-sided at the walls
                d[:, :, 0] = -1.5 * u[:, :, 0] + 2 * u[:, :, 1] - 0.5 * u[:, :, 2]
                d[:, :, -1] = 1.5 * u[:, :, -1] - 2 * u[:, :, -2] + 0.5 * u[:, :, -3]
            g.append(d)
        s = sum((g[b][a] + g[a][b]).square() for a in range(3) for b in range(3))
        return 3 * (self.cfg.C_smag ** 2 * torch.sqrt(0.5 * s) + self.cfg.nu) + 0.5

    def stream(self, post, wall):
        out = torch.empty_like(post)
        for q in range(19):
            out[q] = torch.roll(post[q], (CZ[q], CY[q], CX[q]), (0, 1, 2)) if q else post[q]
        if self.case["flow"] == "rb":
            for q in range(19):
                if CY[q]:
                    row = -1 if CY[q] > 0 else 0
                    out[INV[q]][:, row] = wall(q, row)
        return out

    def step(self):
        c, f = self.cfg, self.f
        tables = self.walk() if self.tables is not None else None
        Fp = self.force(self.T, self.S, self.tables, self.dep_prev)
        T = None if self.g is None else self.g.sum(0)
        S = None if self.h is None else self.h.sum(0)
        F = self.force(T, S, tables, self.dep)
        rho, u = self.velocity(Fp)
        om = 1.0 / (self.smagorinsky(u) if self.case["les"] else c.tau_u)
        k = 1.0 - 0.5 / c.tau_u
        poly = (self.C.T @ u.reshape(3, -1)).reshape(19, *self.shape)  # c.u
        cF = (self.C.T @ F.reshape(3, -1)).reshape(19, *self.shape)
        cF.mul_(9 * poly + 3).sub_(3 * (u * F).sum(0)).mul_(rho * k).mul_(self.w)
        poly = (4.5 * poly).add_(3.0).mul_(poly).add_(1 - 1.5 * (u * u).sum(0)).mul_(self.w)
        post = f + om * (rho * poly - f) + cF
        self.f = self.stream(post, lambda q, r: post[q][:, r])
        for name, t, tau, lo, hi in (("g", T, c.tau_t, c.T_bot - c.T_ref, c.T_top - c.T_ref),
                                     ("h", S, c.tau_s, c.S_bot - c.S_ref, c.S_top - c.S_ref)):
            a = getattr(self, name)
            if a is None:
                continue
            post = a + (t * poly - a) / tau
            setattr(self, name, self.stream(post, lambda q, r: post[INV[q]][:, r] + W[q] * 2 * (
                (hi if r else lo) - t[:, r])))
        self.T, self.S, self.tables, self.dep_prev = T, S, tables, self.dep

    def block(self):
        if self.part is None and self.tables is None:  # every step the same launches: record one
            self.step()
            fields = ("f", "g", "h", "T", "S")
            held = {k: getattr(self, k) for k in fields if getattr(self, k) is not None}
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                self.step()
                for k, v in held.items():
                    v.copy_(getattr(self, k))
            for k, v in held.items():
                setattr(self, k, v)
            for _ in range(self.case["steps"] - 1):
                graph.replay()
            return self.outputs()
        for n in range(self.case["steps"]):
            if n and self.case["twoway"]:
                self.dep = self.part.deposit()
            self.step()
            if self.part is not None:
                self.part.move(self.velocity(self.force(self.T, self.S, self.tables, self.dep))[1], n == 0)
        return self.outputs()

    def outputs(self):
        dens, u = self.velocity(self.force(self.T, self.S, self.tables, self.dep))
        out = {"dens": dens, "u": u.permute(1, 2, 3, 0)}
        if self.g is not None:
            out["t"] = self.g.sum(0)
        if self.h is not None:
            out["s"] = self.h.sum(0)
        if self.part is not None:
            p = self.part
            out.update(velocity=p.v, fluid_velocity=p.u)
            if self.case["twoway"]:
                out["gradient"] = p.grad.reshape(-1, 9)
        out = {k: np.ascontiguousarray(v.cpu().numpy()) for k, v in out.items()}
        if self.part is not None:
            out["position"] = _circle(self.part.x.cpu().numpy(), reversed(self.shape))
        return out


class _ExactParticles:
    """Tracers and Stokes particles with added mass in a periodic box: trilinear u and grad u
    (one-sided on a stencil's halo cells), Adams-Bashforth, trilinear momentum deposit."""

    def __init__(self, flow, rec):
        d = flow.d
        self.n = torch.tensor([flow.case["NX"], flow.case["NY"], flow.case["NZ"]], device="cuda")
        self.L = self.n.to(torch.float64)
        rec = torch.tensor(rec, **d)
        self.tau, self.beta, self.x = rec[:, 1:2], rec[:, 2:3], rec[:, 3:6].clone()
        self.v, self.u, self.a, self.Dt = (torch.zeros_like(self.x) for _ in range(4))
        self.v_old, self.u_old, self.a_old = (torch.zeros_like(self.x) for _ in range(3))
        self.grad = torch.zeros(len(rec), 3, 3, **d)
        self.twoway = flow.case["twoway"]
        r2 = 3.0 * flow.cfg.nu * self.beta * self.tau
        self.vol = (4.0 / 3.0) * 3.14159265359 * r2 ** 1.5
        self.ratio = (3.0 - self.beta) / (2.0 * self.beta)

    def index(self, c):
        c = torch.remainder(c, self.n)
        return (c[:, 2] * self.n[1] + c[:, 1]) * self.n[0] + c[:, 0]

    def corners(self):
        lo = torch.floor(self.x - 0.5).to(torch.int64)
        far = self.x - (lo + 0.5)
        for k in range(8):
            e = torch.tensor([k & 1, k >> 1 & 1, k >> 2], device="cuda")
            yield lo + e, torch.where(e > 0, far, 1 - far).prod(1, keepdim=True)

    def move(self, u, first):
        flat = u.reshape(3, -1).T.contiguous()
        self.u, self.grad = torch.zeros_like(self.u), torch.zeros_like(self.grad)
        for c, w in self.corners():
            here = flat[self.index(c)]
            self.u += w * here
            if self.twoway:
                for b in range(3):
                    e = torch.zeros(3, device="cuda", dtype=torch.int64)
                    e[b] = 1
                    lo, hi = (c[:, b] == -1)[:, None], (c[:, b] == self.n[b])[:, None]
                    up, dn = flat[self.index(c + e)], flat[self.index(c - e)]
                    up2, dn2 = flat[self.index(c + 2 * e)], flat[self.index(c - 2 * e)]
                    one = torch.where(lo, -1.5 * here + 2 * up - 0.5 * up2, 1.5 * here - 2 * dn + 0.5 * dn2)
                    self.grad[:, :, b] += w * torch.where(lo | hi, one, (up - dn) / 2)
        tracer, u = self.tau == 0, self.u
        v = torch.where(tracer, u, self.v)
        v_old = torch.where(tracer, v, self.v_old) if first else self.v_old
        self.x = self.x + (v if first else 0.5 * (3 * v - v_old))
        rel = u - v
        u_old = u if first else self.u_old
        Dt = u - u_old + (self.grad @ rel[:, :, None])[:, :, 0]
        drag = ~tracer
        added = drag & (self.beta != 0)
        a = torch.where(tracer, v - v_old, rel / torch.where(drag, self.tau, 1.0))
        if self.twoway:
            a = torch.where(added, a + self.beta * Dt, a)
            self.Dt = torch.where(added, Dt, self.Dt)
        self.v = torch.where(drag, v + (a if first else 0.5 * (3 * a - self.a_old)), v)
        self.v_old, self.u_old, self.a, self.a_old = v, u, a, torch.where(drag, a, self.a_old)
        self.x = self.x - torch.floor(self.x / self.L) * self.L

    def deposit(self):
        live = (self.vol > 0) & (self.beta != 0)
        force = torch.where(live, self.vol * (self.Dt - self.ratio * self.a), 0.0)
        out = torch.zeros(int(self.n.prod()), 3, device="cuda", dtype=torch.float64)
        for c, w in self.corners():
            inside = ((c >= 0) & (c < self.n)).all(1, keepdim=True)  # halo cells take nothing
            out.index_add_(0, self.index(c), torch.where(inside, w * force, 0.0))
        return out.T.reshape(3, *(int(v) for v in self.n.flip(0)))
