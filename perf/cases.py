"""The work whose speed is followed: SPH runs as a user's program makes them.

Every case goes through the public Python host side (`BodySystem`,
`Ensemble`).  Four ways of use (`mode`):

  run       load particles that live in device tensors, advance by the
            initial iteration and `steps` leapfrog steps (`step`), take the
            state back as device tensors: one output interval of a run;
  calls     the same iterations driven call by call, as a host code with its
            own driver loop does (the C++ hydro driver's sequence);
  io        a running system whose inputs and results are host arrays, every
            step through `step_io`;
  ensemble  many independent 2D problems stepped together.

Sizes, physics and options are those of the repository's configurations and
tests: Sod, Noh, Sedov, Kelvin-Helmholtz and a self-gravitating polytrope, in
two and three dimensions, plain FP64 and mixed precision, Wendland and spline
kernels, constant and Cullen-Dehnen viscosity.  Particle sets are lattices
with a 1 % jitter (the polytrope: sampled radii), drawn from the seed, on the
GPU.
"""
import math

import torch

from flecsph_gb300.abi import (EOS_POLYTROPIC, KERNEL_CUBIC_SPLINE, KERNEL_WENDLAND_C4,
                               KERNEL_WENDLAND_C6, PRECISION_FP64, PRECISION_MIXED,
                               Params, VISC_CULLEN, make_view_tensors)
from flecsph_gb300.sph import BodySystem, Ensemble

DEV = torch.device("cuda", 0)
F64 = torch.float64
KERNELS = {"wendland_c6": KERNEL_WENDLAND_C6, "wendland_c4": KERNEL_WENDLAND_C4,
           "cubic_spline": KERNEL_CUBIC_SPLINE}
# h = eta * 2 * dx and the dimension of each problem
ETA = {"sod2d": 1.5, "noh2d": 1.5, "sod3d": 1.5, "sedov3d": 1.495, "kh3d": 1.44,
       "polytrope3d": 1.2}


# ------------------------------------------------------------------ cases --
def _case(problem, size, mode="run", precision="mixed", kernel="wendland_c6",
          viscosity="constant", steps=2, members=0, name=None):
    c = dict(problem=problem, size=size, mode=mode, precision=precision, kernel=kernel,
             viscosity=viscosity, steps=steps, members=members)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest problems of a parameter study (2,250 particles): every
        # kernel is a fraction of a wave, launches and latency are the time
        _case("sod2d", 15, steps=16, name="sod2d_2k"),
        # an ordinary 2D problem with the adaptive viscosity
        _case("noh2d", 199, viscosity="cullen", steps=4, name="noh2d_31k_cullen"),
        # the reference's 3D tube at a test's size, a spline kernel (not the
        # float-float passes), driven call by call by a host code
        _case("sod3d", 20, mode="calls", kernel="cubic_spline", steps=4,
              name="sod3d_32k_calls"),
        # the blast at an ordinary, odd size
        _case("sedov3d", 51, steps=4, name="sedov3d_133k"),
        # the blast at the benchmark's size
        _case("sedov3d", 128, steps=3, name="sedov3d_2m"),
        # the same blast with host arrays in and out of every step
        _case("sedov3d", 100, mode="io", steps=1, name="sedov3d_1m_io"),
        # self-gravity, varying h: a small star and the benchmark's
        _case("polytrope3d", 50000, steps=2, name="polytrope_50k"),
        _case("polytrope3d", 4194304, steps=2, name="polytrope_4m"),
        # periodic shear flow at the benchmark's size, the largest run
        _case("kh3d", 256, steps=1, name="kh3d_17m"),
        # the plain FP64 method, which follows the reference to rounding
        _case("noh2d", 100, precision="fp64", kernel="wendland_c4", steps=4,
              name="noh2d_8k_fp64"),
        _case("sedov3d", 45, precision="fp64", steps=2, name="sedov3d_91k_fp64"),
        # a parameter study: 32 tubes of 2k to 50k particles side by side
        _case("sod2d", 50000, mode="ensemble", steps=8, members=32,
              name="ensemble_32"),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["small2d", "mid2d", "tube", "blast", "blast", "io", "star", "shear",
                       "fp64_2d", "fp64_3d", "ensemble"])
    kernel = rng.choice(["wendland_c6", "wendland_c6", "wendland_c4", "cubic_spline"])
    wendland = rng.choice(["wendland_c6", "wendland_c4"])
    visc = rng.choice(["constant", "constant", "cullen"])
    if kind == "small2d":
        return _case("sod2d", logint(10, 40), steps=rng.randint(8, 16), kernel=kernel)
    if kind == "mid2d":
        return _case("noh2d", logint(60, 700), steps=rng.randint(2, 6), viscosity=visc)
    if kind == "tube":
        return _case("sod3d", logint(8, 40), mode=rng.choice(["run", "calls"]), kernel=kernel,
                     steps=rng.randint(2, 6))
    if kind == "blast":
        return _case("sedov3d", logint(16, 140), kernel=wendland, steps=rng.randint(1, 4))
    if kind == "io":
        return _case("sedov3d", logint(24, 110), mode="io", steps=1)
    if kind == "star":
        return _case("polytrope3d", logint(5000, 2500000), steps=rng.randint(1, 3))
    if kind == "shear":
        return _case("kh3d", logint(20, 180), steps=rng.randint(1, 3))
    if kind == "fp64_2d":
        return _case("noh2d", logint(40, 400), precision="fp64", kernel=kernel, viscosity=visc,
                     steps=rng.randint(2, 4))
    if kind == "fp64_3d":
        return _case("sedov3d", logint(16, 56), precision="fp64", kernel=wendland,
                     steps=rng.randint(1, 3))
    return _case("sod2d", logint(8000, 60000), mode="ensemble", steps=8,
                 members=rng.randint(8, 40))


# -------------------------------------------------------- particle states --
def _params(case, dx):
    problem = case["problem"]
    p = Params.defaults(dimension=2 if problem.endswith("2d") else 3,
                        sph_kernel=KERNELS[case["kernel"]], sph_eta=ETA[problem],
                        poly_gamma=1.4 if problem.startswith("sod") else 5.0 / 3.0,
                        adaptive_timestep=1, timestep_cfl_factor=0.25,
                        initial_dt={"polytrope3d": 1e-5, "noh2d": 0.02 * dx}.get(
                            problem, 0.1 * dx))
    p.precision_mode = PRECISION_MIXED if case["precision"] == "mixed" else PRECISION_FP64
    if case["viscosity"] == "cullen":
        p.sph_viscosity = VISC_CULLEN
    if problem == "kh3d":
        p.periodic_boundary_x = p.periodic_boundary_y = p.periodic_boundary_z = 1
        p.box_length = p.box_width = p.box_height = 1.0
    if problem == "polytrope3d":
        p.eos_type, p.poly_gamma = EOS_POLYTROPIC, 2.0
        p.enable_fmm, p.fmm_macangle, p.gravity_order = 1, 0.5, 2
        p.thermokinetic_formulation = 0
        p.max_neighbors = 512
    return p


def _lattice(ns, dx, gen, disc=False):
    """Cell centres of a box of ns cells centred on the origin, x fastest,
    (those of the disc of radius 0.5 only,) with the jitter."""
    axes = [(torch.arange(n, dtype=F64, device=DEV) + 0.5 - 0.5 * n) * dx for n in ns]
    grid = torch.meshgrid(*reversed(axes), indexing="ij")
    pos = torch.stack([g.reshape(-1) for g in reversed(grid)], 1)
    if disc:
        pos = pos[pos.norm(dim=1) < 0.5]
    return pos + 0.01 * dx * torch.randn(pos.shape, generator=gen, dtype=F64, device=DEV)


def _polytrope_positions(n, gen):
    """Radii of the n = 1 polytrope by inverting its enclosed mass, isotropic
    directions."""
    t = torch.rand(n, generator=gen, dtype=F64, device=DEV)
    lo, hi = torch.zeros_like(t), torch.ones_like(t)
    for _ in range(50):
        mid = 0.5 * (lo + hi)
        below = torch.sin(math.pi * mid) - math.pi * mid * torch.cos(math.pi * mid) < math.pi * t
        lo, hi = torch.where(below, mid, lo), torch.where(below, hi, mid)
    r = 0.5 * (lo + hi)
    d = torch.randn((n, 3), generator=gen, dtype=F64, device=DEV)
    return r, r[:, None] * d / d.norm(dim=1, keepdim=True)


def _state(case, seed):
    """(dict of device tensors, Params) of a case's particles."""
    problem, size = case["problem"], case["size"]
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    D = 2 if problem.endswith("2d") else 3
    vel = None
    if problem == "polytrope3d":
        dx = size ** (-1.0 / 3.0)
        r, pos = _polytrope_positions(size, gen)
        rho_c = math.pi / 4.0
        rho = rho_c * torch.sin(math.pi * r) / (math.pi * r)
        rho = torch.clamp(rho, min=1e-2 * rho_c)
        m = torch.full_like(r, 1.0 / size)
        K = 2.0 / math.pi
        P, u = K * rho ** 2, K * rho
        h = ETA[problem] * 2.0 * (m / rho) ** (1.0 / 3.0)
        # a slow radial pulsation, so that the flow compresses
        vel = -0.05 * pos
    else:
        ns = {"sod2d": (10 * size, size), "noh2d": (size, size),
              "sod3d": (4 * size, size, size), "sedov3d": (size,) * 3,
              "kh3d": (size,) * 3}[problem]
        dx = 1.0 / ns[0]
        pos = _lattice(ns, dx, gen, disc=problem == "noh2d")
        one = torch.ones(len(pos), dtype=F64, device=DEV)
        h = ETA[problem] * 2.0 * dx * one
        if problem.startswith("sod"):
            left = pos[:, 0] < 0.0
            rho, P = torch.where(left, 1.0, 0.125).to(F64), torch.where(left, 1.0, 0.1).to(F64)
            u = P / (0.4 * rho)
        elif problem == "noh2d":
            # cool gas (Mach 1.7): the adaptive viscosity starts from zero
            rho, P, u = one, 0.2 * one, 0.3 * one
            vel = -pos / pos.norm(dim=1, keepdim=True)
        elif problem == "sedov3d":
            q = pos.norm(dim=1) / (2.0 * h)
            w = torch.where(q < 1.0, (1 - q) ** 8 * (1 + q * (8 + q * (25 + q * 32))), 0.0)
            rho, u = one, 1e-5 + w / (dx ** 3 * w.sum())
            P = (2.0 / 3.0) * u
        else:  # kh3d
            band = pos[:, 1].abs() < 0.25
            rho, P = torch.where(band, 2.0, 1.0).to(F64), 2.5 * one
            u = P / ((2.0 / 3.0) * rho)
            vel = torch.zeros_like(pos)
            vel[:, 0] = torch.where(band, 0.5, -0.5).to(F64)
            vel[:, 1] = 0.01 * torch.sin(4.0 * math.pi * pos[:, 0])
        m = rho * dx ** D
    if vel is None:
        vel = torch.zeros_like(pos)
    s = {"m": m, "h": h, "rho": rho, "P": P, "u": u}
    for d in range(3):
        s["xyz"[d]] = pos[:, d].contiguous() if d < D else torch.zeros_like(h)
        s["v" + "xyz"[d]] = vel[:, d].contiguous() if d < D else torch.zeros_like(h)
    s["id"] = torch.arange(len(h), dtype=torch.int64, device=DEV)
    return s, _params(case, dx)


def _out_fields(p):
    D = p.dimension
    f = [a + "xyz"[d] for a in ("", "v", "vh", "a") for d in range(D)]
    f += ["rho", "P", "cs", "u", "vsig", "dt"]
    f += ["e", "dedt"] if p.thermokinetic_formulation else ["dudt"]
    if p.enable_fmm:
        f += ["gax", "gay", "gaz", "gpot"]
    if p.sph_viscosity == VISC_CULLEN:
        f += ["alpha", "divv"]
    return f + ["id", "key"]


def _member_cases(case):
    """Sizes of an ensemble's tubes: logarithmically spread up to `size`
    particles."""
    k = case["members"]
    out = []
    for i in range(k):
        n = 2000.0 * (case["size"] / 2000.0) ** (i / max(1, k - 1))
        out.append(dict(case, size=max(4, round(math.sqrt(n / 10.0)))))
    return out


def _particles(case):
    s = case["size"]
    if case["mode"] == "ensemble":
        return sum(10 * c["size"] ** 2 for c in _member_cases(case))
    return {"sod2d": 10 * s * s, "noh2d": int(0.785 * s * s), "sod3d": 4 * s ** 3,
            "polytrope3d": s}.get(case["problem"], s ** 3)


# ------------------------------------------------------- prepare and run --
# fields a host-side driver holds and hands to every step of a running system
IO_IN = ["x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az", "gax", "gay", "gaz", "m", "h",
         "cs", "u", "e", "dedt", "K"]


def prepare(case, seed):
    if case["mode"] == "ensemble":
        ens = Ensemble()
        for k, c in enumerate(_member_cases(case)):
            s, p = _state(c, seed * 1000 + k)
            ens.add(p, len(s["id"])).read_bodies_device(s)
        ens.set_lanes(8)
        ens.step(2)  # a running study: past the initial and one eager step
        ens.sync()
        return dict(case=case, ens=ens, fields=_out_fields(p))
    s, p = _state(case, seed)
    n = len(s["id"])
    capacity = n
    if case["problem"] == "kh3d":
        # the copies within 2.5 h of the faces, and a margin
        shell = 1.0 + 5.0 * float(s["h"][0])
        capacity = int(n * (1.0 + 1.25 * (shell ** 3 - 1.0))) + 1024
    bs = BodySystem(p, capacity)
    st = dict(case=case, bs=bs, batch=s, fields=_out_fields(p))
    if case["mode"] == "io":
        bs.read_bodies_device(s)
        bs.step()
        now = bs.download_device(sorted(set(IO_IN + st["fields"])), device=DEV)
        st["host_in"] = {f: now[f].cpu().pin_memory() for f in IO_IN + ["id"]}
        st["host_out"] = {f: now[f].cpu().pin_memory() for f in st["fields"]}
        st["vin"] = make_view_tensors(st["host_in"])
        st["vout"] = make_view_tensors(st["host_out"], n=n)
        del st["batch"]
    return st


def _driver_iteration(bs, first):
    """One iteration of the reference's hydro driver, call by call."""
    if first:
        bs.update_iteration()
        bs.eos_init()
        bs.set_total_energy()
        bs.density_pressure_soundspeed()
        bs.save_velocityhalf()
        bs.reset_ghosts()
        bs.acceleration()
        bs.compute_dt()
        bs.set_adaptive_timestep()
        bs.dedt()
        bs.recompute_pressure_soundspeed_thermokinetic()
    else:
        bs.leapfrog_kick_e()
        bs.leapfrog_kick_v()
        bs.save_velocityhalf()
        bs.leapfrog_drift()
        bs.update_iteration()
        bs.density_pressure_soundspeed()
        bs.reset_ghosts()
        bs.acceleration()
        bs.leapfrog_kick_v()
        bs.reset_ghosts()
        bs.dedt()
        bs.recompute_pressure_soundspeed_thermokinetic()
        bs.leapfrog_kick_e()
    bs.check_nans()
    bs.check_negativity()
    bs.compute_dt()
    bs.set_adaptive_timestep()
    bs.advance_time()


def run(state):
    case = state["case"]
    if case["mode"] == "ensemble":
        ens = state["ens"]
        ens.step(case["steps"])
        parts = [m.download_device(state["fields"], device=DEV) for m in ens.members]
        return {f: torch.cat([q[f] for q in parts]) for f in state["fields"]}
    bs = state["bs"]
    if case["mode"] == "io":
        bs.step_io(state["vin"], state["vout"])
        return state["host_out"]
    bs.read_bodies_device(state["batch"])
    for k in range(case["steps"] + 1):
        if case["mode"] == "calls":
            _driver_iteration(bs, k == 0)
        else:
            bs.step()
    return bs.download_device(state["fields"], device=DEV)


# ------------------------------------------------------------------ work --
def work(case):
    """Every input field read once, every output field written once; the pair
    terms of the method once per pair and iteration (operations as the
    reference writes them: density 31, signal speed 27, acceleration 82,
    energy 96, gravity 62 per accepted cell)."""
    n = _particles(case)
    D = 2 if case["problem"].endswith("2d") else 3
    eta = ETA[case["problem"]]
    nb = math.pi * (2 * eta) ** 2 if D == 2 else 4.0 / 3.0 * math.pi * (2 * eta) ** 3
    iterations = case["steps"] + (0 if case["mode"] in ("io", "ensemble") else 1)
    flops = n * iterations * nb * (31 + 27 + 82 + 96 + (20 if case["viscosity"] == "cullen" else 0))
    if case["problem"] == "polytrope3d":
        # cells and particles that a walk at this opening angle meets
        flops += n * iterations * 62 * 60 * math.log2(max(2.0, n / 32.0))
    fields_in = 5 + 2 * D + 1 if case["mode"] != "io" else len(IO_IN) + 1
    fields_out = 4 * D + 10 + (3 if case["problem"] == "polytrope3d" else 0)
    return {"bytes": 8.0 * n * (fields_in + fields_out), "flops": float(flops)}


# ------------------------------------------------- the same in 64 bits --
PAIR_LIMIT = 2.5e11  # pair distances of the direct neighbour search, all iterations


class _Reference:
    """The method in plain torch, FP64: direct neighbour search, pair sums by
    index_add, gravity by direct summation.  No periodic copies, no
    Cullen-Dehnen viscosity."""

    def __init__(self, s, p):
        self.p, self.D = p, p.dimension
        D = self.D
        self.x = torch.stack([s["xyz"[d]] for d in range(D)], 1)
        self.v = torch.stack([s["v" + "xyz"[d]] for d in range(D)], 1)
        zero = torch.zeros_like(s["h"])
        self.f = {k: s[k].clone() for k in ("m", "h", "rho", "P", "u")}
        for k in ("cs", "e", "dedt", "dudt", "K", "vsig", "dt"):
            self.f[k] = zero.clone()
        self.vh, self.a, self.g = self.v.clone(), torch.zeros_like(self.v), torch.zeros_like(self.v)
        self.gpot = zero.clone()
        self.dt, self.first = p.initial_dt, True

    # sort by Morton key; the keys quantise positions over the range of x +- h
    def update(self):
        D, md = self.D, 63 // self.D
        h = self.f["h"][:, None]
        lo, hi = (self.x - h).amin(0), (self.x + h).amax(0)
        c = ((self.x - lo) / (hi - lo) * 2.0 ** md).to(torch.int64).clamp(0, 2 ** md - 1)
        key = torch.zeros_like(c[:, 0])
        for b in range(md):
            for d in range(D):
                key |= ((c[:, d] >> b) & 1) << (D * b + d)
        o = torch.sort(key, stable=True).indices
        self.x, self.v, self.vh, self.a, self.g = (t[o] for t in (self.x, self.v, self.vh, self.a, self.g))
        self.f = {k: t[o] for k, t in self.f.items()}
        self.gpot = self.gpot[o]
        n = len(o)
        rows = max(1, int(1.5e8 // n))
        ii, jj = [], []
        h = self.f["h"]
        for r in range(0, n, rows):
            e = min(n, r + rows)
            d2 = torch.zeros((e - r, n), dtype=F64, device=DEV)
            for d in range(D):
                t = self.x[r:e, d, None] - self.x[None, :, d]
                d2 += t.mul_(t)
            near = d2 <= torch.maximum(h[r:e, None], h[None, :]) ** 2
            q = near.nonzero()
            ii.append(q[:, 0] + r)
            jj.append(q[:, 1])
        self.i, self.j = torch.cat(ii), torch.cat(jj)
        keep = self.i != self.j
        self.si = self.i[keep]
        self.sj = self.j[keep]
        self.pair_geometry()

    def pair_geometry(self):
        i, j, D = self.si, self.sj, self.D
        self.dx = self.x[i] - self.x[j]
        self.r = self.dx.norm(dim=1)
        self.hab = 0.5 * (self.f["h"][i] + self.f["h"][j])
        q = self.r / self.hab
        t = (1 - q).clamp(min=0.0)
        K = self.p.sph_kernel
        if K == KERNEL_CUBIC_SPLINE:
            s = 40.0 / (7.0 * math.pi) if D == 2 else 8.0 / math.pi
            q2 = 2.0 * q
            W = torch.where(q2 < 1, 1 - 1.5 * q2 ** 2 + 0.75 * q2 ** 3, 0.25 * (2 - q2).clamp(min=0) ** 3)
            dW = 2.0 * torch.where(q2 < 1, -3 * q2 + 2.25 * q2 ** 2, -0.75 * (2 - q2).clamp(min=0) ** 2)
        elif K == KERNEL_WENDLAND_C4:
            s = 9.0 / math.pi if D == 2 else 495.0 / (32.0 * math.pi)
            W = t ** 6 * (1 + q * (6 + q * (35.0 / 3.0)))
            dW = -56.0 / 3.0 * q * t ** 5 * (1 + 5 * q)
        else:
            s = 78.0 / (7.0 * math.pi) if D == 2 else 1365.0 / (64.0 * math.pi)
            W = t ** 8 * (1 + q * (8 + q * (25 + q * 32)))
            dW = -22.0 * q * t ** 7 * (1 + q * (7 + q * 16))
        self.W = s * W / self.hab ** D
        self.DW = self.dx * (s * dW / self.hab ** (D + 1) / self.r)[:, None]
        self.W0 = s / self.f["h"] ** D

    def sum(self, t):
        out = torch.zeros((len(self.x),) + t.shape[1:], dtype=F64, device=DEV)
        return out.index_add_(0, self.si, t)

    def eos(self, u):
        f, g = self.f, self.p.poly_gamma
        if self.p.eos_type == EOS_POLYTROPIC:
            f["P"] = f["K"] * f["rho"] ** g
            return torch.sqrt(g * f["P"] / f["rho"])
        f["P"] = (g - 1) * f["rho"] * u
        return torch.sqrt(g * (g - 1) * u)

    def density(self):
        f, i, j = self.f, self.si, self.sj
        f["rho"] = self.sum(f["m"][j] * self.W) + f["m"] * self.W0
        if self.p.thermokinetic_formulation:
            f["u"] = f["e"] - 0.5 * (self.v ** 2).sum(1)
        new = self.eos(f["u"])
        # particles are visited in descending key order, each setting its
        # sound speed just before its signal speed
        cb = torch.where(j > i, new[j], f["cs"][j])
        vn = ((self.v[i] - self.v[j]) * self.dx).sum(1) / self.r
        cand = torch.maximum(new[i], cb) - vn.clamp(max=0.0)
        f["vsig"] = torch.zeros_like(new).scatter_reduce_(0, i, cand, "amax")
        f["cs"] = new

    def viscosity(self):
        f, i, j, p = self.f, self.si, self.sj, self.p
        dot = ((self.vh[i] - self.vh[j]) * self.dx).sum(1)
        mu = self.hab * dot / (self.r ** 2 + p.sph_viscosity_epsilon * self.hab ** 2)
        mu = torch.where(dot < 0, mu, torch.zeros_like(mu))
        c, rho = 0.5 * (f["cs"][i] + f["cs"][j]), 0.5 * (f["rho"][i] + f["rho"][j])
        return (-p.sph_viscosity_alpha * c + p.sph_viscosity_beta * mu) * mu / rho

    def acceleration(self):
        f, i, j = self.f, self.si, self.sj
        A = f["P"] / f["rho"] ** 2
        s = -f["m"][j] * (A[i] + A[j] + self.viscosity())
        self.a = self.sum(self.DW * s[:, None])

    def gravity(self):
        n = len(self.x)
        G, m = self.p.gravitational_constant, self.f["m"]
        rows = max(1, int(1e8 // n))
        for r in range(0, n, rows):
            e = min(n, r + rows)
            d = [self.x[r:e, k, None] - self.x[None, :, k] for k in range(3)]
            r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
            inv = torch.where(r2 > 0, r2.rsqrt(), torch.zeros_like(r2))
            self.gpot[r:e] = -G * (inv @ m)
            inv = inv ** 3
            for k in range(3):
                self.g[r:e, k] = -G * ((inv * d[k]) @ m)

    def energy(self):
        """de/dt or du/dt, then pressure and sound speed at the half step
        ahead."""
        f, i, j = self.f, self.si, self.sj
        A, Pi, mj = f["P"] / f["rho"] ** 2, self.viscosity(), f["m"][j]
        if self.p.thermokinetic_formulation:
            va, vb = (self.v[i] * self.DW).sum(1), (self.v[j] * self.DW).sum(1)
            f["dedt"] = (self.g * self.v).sum(1) - self.sum(
                mj * (A[i] * vb + va * A[j] + 0.5 * Pi * (vb + va)))
            f["u"] = f["e"] - 0.5 * (self.v ** 2).sum(1)
            f["cs"] = self.eos(f["u"] + 0.5 * self.dt * (f["dedt"] - (self.v * self.a).sum(1)))
        else:
            w = mj * ((self.v[i] - self.v[j]) * self.DW).sum(1)
            f["dudt"] = A * self.sum(w) + 0.5 * self.sum(w * Pi)
            f["cs"] = self.eos(f["u"] + 0.5 * self.dt * f["dudt"])

    def timestep(self):
        f, p = self.f, self.p
        dx = f["h"] / (p.sph_eta * 2.0)
        tiny = 1e-24
        dtv = dx / (self.v.norm(dim=1) + tiny)
        dta = torch.sqrt(dx / ((self.a + self.g).norm(dim=1) + tiny))
        dtc = dx / (tiny + f["vsig"] * (1 + 0.6 * p.sph_viscosity_alpha))
        f["dt"] = p.timestep_cfl_factor * torch.minimum(torch.minimum(dtv, dta), dtc)
        least = float(f["dt"].min())
        if least < self.dt:
            self.dt = min(least, self.dt / 2)
        if least > 2 * self.dt:
            self.dt *= 2

    def iterate(self):
        f, p = self.f, self.p
        thermo = p.thermokinetic_formulation
        if self.first:
            self.update()
            f = self.f
            f["K"] = f["P"] / f["rho"] ** p.poly_gamma
            f["e"] = 0.5 * (self.v ** 2).sum(1) + f["u"]
            self.density()
            self.vh = self.v.clone()
            self.acceleration()
            if p.enable_fmm:
                self.gravity()
            self.timestep()
            self.energy()
            self.first = False
        else:
            rate = "dedt" if thermo else "dudt"
            f["e" if thermo else "u"] = f["e" if thermo else "u"] + 0.5 * self.dt * f[rate]
            self.v = self.v + (self.a + self.g) * (0.5 * self.dt)
            self.vh = self.v.clone()
            self.x = self.x + self.v * self.dt
            self.update()
            f = self.f
            self.density()
            self.acceleration()
            if p.enable_fmm:
                self.gravity()
            self.v = self.v + (self.a + self.g) * (0.5 * self.dt)
            self.energy()
            f["e" if thermo else "u"] = f["e" if thermo else "u"] + 0.5 * self.dt * f[rate]
        self.timestep()

    def outputs(self, fields):
        out = {}
        for k in fields:
            if k in ("id", "key"):
                out[k] = None
            elif k == "gpot":
                out[k] = self.gpot
            elif k in self.f:
                out[k] = self.f[k]
            else:
                src = {"": self.x, "v": self.v, "vh": self.vh, "a": self.a, "ga": self.g}
                out[k] = src[k[:-1]][:, "xyz".index(k[-1])].contiguous()
        return out


def exact(case, seed):
    n = _particles(case)
    if case["problem"] == "kh3d" or case["viscosity"] == "cullen":
        return None
    iterations = case["steps"] + {"io": 1, "ensemble": 2}.get(case["mode"], 1)
    sizes = ([10 * c["size"] ** 2 for c in _member_cases(case)]
             if case["mode"] == "ensemble" else [n])
    if sum(float(k) ** 2 for k in sizes) * iterations > PAIR_LIMIT:
        return None
    if case["mode"] == "ensemble":
        states = [_state(c, seed * 1000 + k) for k, c in enumerate(_member_cases(case))]
    else:
        states = [_state(case, seed)]
    parts = []
    for s, p in states:
        ref = _Reference(s, p)
        for _ in range(iterations):
            ref.iterate()
        parts.append(ref.outputs(_out_fields(p)))
    return {f: None if parts[0][f] is None else torch.cat([q[f] for q in parts])
            for f in parts[0]}
