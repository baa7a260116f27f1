"""Performance cases: the work a user of cudapic_b200 has it do.

Each case is one call (or the few calls that belong together) of a public
entry point: the drop-in kernels of ``cudapic_b200.kernels``, as a host that
owns its buffers calls them, and the drivers (``GpuSimState``, ``Batch``,
``VoltageSensitivity``).  Sizes follow the reference (N_G = 400, 120 000
particles per species, 13.56 MHz, N_T = 4000, N_SUB = 20), the benchmark
(4 194 304 + 4 194 304 particles; sweeps of discharges with 1e4 .. 1e6
particles, 5 .. 50 Pa, N_G 200 / 400 / 800) and the tests (N_G up to 16384).

Electrons of the single-kernel cases are Maxwellian at 3 eV with the tail cut
below the ionization threshold, between two sheaths that hold them (an argon
CCP's bulk): such a call gives every particle's result at its own slot, so
that results can be compared value by value.  Ionization, absorption and the
whole energy range are in the driver cases, whose particles interleave in an
unspecified order; these return the potential that the steps leave (the
particles' order and single nodes of the densities are noise), or the
measurement window's results.
"""
import math

import numpy as np
import torch

import cudapic_b200 as cp
from cudapic_b200.batch import Batch
from cudapic_b200.sensitivity import VoltageSensitivity
from cudapic_b200.sim import GpuSimState, ParticlesSoA
from cudapic_b200.workloads import DischargeSpec, c2_specs, initial_population

K = cp.kernels
E_CHARGE, E_MASS, AR_MASS, EPS0 = 1.60217662e-19, 9.10938356e-31, 6.63352090e-26, 8.85418781e-12
GAP, PRESSURE = 0.025, 10.0
ON_CHIP = 126e6     # bytes that stay on the chip between the steps of a run (L2)


def listed():
    return [
        # the field solve alone at the reference's grid: the smallest call, all latency
        {"name": "solve_400", "kind": "solve", "n_g": 400, "f32": False},
        # the charge deposit of a large population (after an upload, and every step of a drop-in host)
        {"name": "deposit_4m", "kind": "deposit", "particles": 4194304, "n_g": 400},
        # push, compaction and next deposit at the reference's own size (ragged), from a drop-in host
        {"name": "push_110k", "kind": "push", "particles": 110003, "n_g": 400, "species": "e", "deposit": True},
        # electron collisions of a drop-in host, an odd middle size
        {"name": "mcc_e_2m", "kind": "mcc_e", "particles": 2000001, "pressure": 10.0},
        # ion collisions of a drop-in host that knows its table's largest entry
        {"name": "mcc_i_4m", "kind": "mcc_i", "particles": 4194304, "pressure": 10.0, "bounded": True},
        # the electron half of a step in place (stream and scatter pass) on caller-owned planes
        {"name": "electron_step_4m", "kind": "electron_step", "particles": 4194304, "n_g": 400, "pressure": 10.0,
         "inplace": True},
        # seeding one stream per slot, once per run
        {"name": "seed_2m", "kind": "seed", "streams": 2097155},
        # one RF cycle of a small discharge (a sweep's smallest member on its own): launches and latency
        {"name": "discharge_10k", "kind": "discharge", "particles": 10000, "n_g": 400, "steps": 4000,
         "measure": False},
        # one measured RF cycle, as the precision study runs them: averages, EEPF, XT maps
        {"name": "measured_400k", "kind": "discharge", "particles": 400000, "n_g": 400, "steps": 4000,
         "measure": True},
        # the benchmark's one large discharge, a tenth of an RF cycle
        {"name": "discharge_4m", "kind": "discharge", "particles": 4194304, "n_g": 400, "steps": 400,
         "measure": False},
        # a parameter sweep stepped as one batch, a tenth of an RF cycle
        {"name": "sweep_24", "kind": "sweep", "discharges": 24, "sweep": 24301, "steps": 400},
        # observables and their voltage derivatives: forward and backward over 200 steps
        {"name": "sensitivity_200k", "kind": "sensitivity", "particles": 200000, "window": 200, "checkpoint": 100},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "deposit", "push", "mcc_e", "mcc_i", "electron_step", "seed", "discharge", "discharge",
                       "sweep", "sensitivity"])
    n_g = rng.choice([200, 400, 400, 800, _log(rng, 129, 4096)])
    pressure = math.exp(rng.uniform(math.log(5.0), math.log(50.0)))
    if kind == "solve":
        return {"kind": kind, "n_g": _log(rng, 100, 16384), "f32": rng.random() < 0.2}
    if kind == "deposit":
        return {"kind": kind, "particles": _log(rng, 1000, 4194304), "n_g": n_g}
    if kind == "push":
        return {"kind": kind, "particles": _log(rng, 1000, 4194304), "n_g": n_g, "species": rng.choice("ei"),
                "deposit": rng.random() < 0.6}
    if kind == "mcc_e":
        return {"kind": kind, "particles": _log(rng, 1000, 4194304), "pressure": pressure}
    if kind == "mcc_i":
        return {"kind": kind, "particles": _log(rng, 1000, 4194304), "pressure": pressure,
                "bounded": rng.random() < 0.6}
    if kind == "electron_step":
        return {"kind": kind, "particles": _log(rng, 1000, 4194304), "n_g": n_g, "pressure": pressure,
                "inplace": rng.random() < 0.7}
    if kind == "seed":
        return {"kind": kind, "streams": _log(rng, 1000, 4194304)}
    if kind == "discharge":
        measure = rng.random() < 0.3
        particles = _log(rng, 300000, 500000) if measure else _log(rng, 10000, 4000000)
        steps = 4000 if measure or particles < 400000 else 400
        return {"kind": kind, "particles": particles, "n_g": rng.choice([200, 400, 800]), "steps": steps,
                "measure": measure}
    if kind == "sweep":
        return {"kind": kind, "discharges": rng.randint(3, 24), "sweep": rng.randint(1, 1 << 20), "steps": 400}
    return {"kind": kind, "particles": _log(rng, 20000, 200000), "window": 200, "checkpoint": rng.choice([100, 200])}


# ------------------------------------------------------------------ inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _u32(v):
    return torch.tensor([v], dtype=torch.int32, device="cuda")


def _pad4(n):
    return (n + 3) // 4 * 4


def _plane(values, cap):
    out = torch.zeros(cap, dtype=values.dtype, device="cuda")
    out[:values.numel()] = values
    return out


def _bulk_x(n, gen, lo=0.0, hi=GAP):
    """Positions of a CCP's parabolic density profile over [lo, hi]."""
    r = torch.rand(3, n, generator=gen, device="cuda").sort(0).values[1]
    return (lo + (hi - lo) * r).clamp_(lo, hi)


def _maxwell(n, gen, mass, ev):
    return torch.randn(3, n, generator=gen, device="cuda") * math.sqrt(ev * E_CHARGE / mass)


def _electrons(n, gen):
    """3 eV electrons, those above 15 eV slowed down to it (a depleted tail)."""
    v = _maxwell(n, gen, E_MASS, 3.0)
    top = math.sqrt(2.0 * 15.0 * E_CHARGE / E_MASS)
    return v * (top / v.norm(dim=0)).clamp_(max=1.0)


def _sheath_field(n_g):
    """A field-free bulk between two sheaths of 0.12 L that turn electrons back."""
    x = np.linspace(0.0, 1.0, n_g)
    s, e_s = 0.12, 1.0e5
    return (-e_s * np.maximum(0.0, 1.0 - x / s) + e_s * np.maximum(0.0, 1.0 - (1.0 - x) / s)).astype(np.float32)


def _streams(n, seed):
    planes = [torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(4)]
    K.xoshiro128_seed_streams(_master(seed), n, *planes)
    return planes


def _master(seed):
    r = np.random.default_rng(seed)
    return [int(v) for v in r.integers(1, 1 << 32, 4)]


def _tables(grid):
    cs, se, si = K.init_cross_sections(grid.gas_density)
    return (torch.from_numpy(cs).cuda(), torch.from_numpy(se).cuda(), torch.from_numpy(si).cuda(), float(se.max()),
            float(si.max()))


def _weight(particles):
    """The reference's superparticle weight scaled to the particle count (the same plasma density)."""
    return 7.0e4 * 120000 / particles


class _DeviceView:
    """A library buffer as an array torch can read in place; its owner lives as long as the view."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (int(ptr), False), "version": 2}


def _pot_of(st, owner):
    return torch.as_tensor(_DeviceView(owner, st.buffers().pot, st.grid.n_g, "<f4"), device="cuda")


def _densities(case, seed):
    """Electron and ion densities of a CCP at a small and noisy charge imbalance (float32, host)."""
    r = np.random.default_rng(seed)
    n_g = case["n_g"]
    x = np.linspace(0.0, 1.0, n_g)
    ion = 5.0e15 * (0.15 + 0.85 * np.sin(math.pi * x)) * (1.0 + 0.01 * r.standard_normal(n_g))
    edge = np.clip(np.minimum(x, 1.0 - x) / 0.15, 0.0, 1.0)
    ele = ion * (0.02 + 0.98 * edge) * (1.0 + 0.01 * r.standard_normal(n_g))
    return ele.astype(np.float32), ion.astype(np.float32), float(np.float32(r.uniform(-250.0, 250.0)))


def _push_inputs(case, seed):
    """x, v of one species (float32, GPU), about one in a thousand leaving through an electrode this step."""
    gen = _gen(seed)
    n = case["particles"]
    ions = case["species"] == "i"
    g = cp.grid_from_params(n_g=case["n_g"], capacity=_pad4(n + n // 4), weight=_weight(n))
    x = _bulk_x(n, gen)
    v = _maxwell(n, gen, AR_MASS, 0.03) if ions else _maxwell(n, gen, E_MASS, 3.0)
    out = torch.rand(n, generator=gen, device="cuda") < 1e-3
    step = torch.rand(n, generator=gen, device="cuda") * v[0].abs() * (g.dt_i if ions else g.dt_e)
    x = torch.where(out, torch.where(v[0] < 0, step, GAP - step), x).clamp_(0.0, GAP)
    return g, x, v


def _step_inputs(case, seed):
    gen = _gen(seed)
    n = case["particles"]
    x = _bulk_x(n, gen, 0.15 * GAP, 0.85 * GAP)
    return x, _electrons(n, gen)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "solve":
        e, i, s["pot0"] = _densities(case, seed)
        s["grid"] = cp.grid_from_params(n_g=case["n_g"], flags=1 if case["f32"] else 0)
        s["e"], s["i"] = torch.from_numpy(e).cuda(), torch.from_numpy(i).cuda()
        s["pot"], s["efield"] = torch.zeros_like(s["e"]), torch.zeros_like(s["e"])
    elif kind == "deposit":
        n = case["particles"]
        s["grid"] = cp.grid_from_params(n_g=case["n_g"], capacity=_pad4(n + n // 4), weight=_weight(n))
        s["x"] = _bulk_x(n, _gen(seed))
        s["n"], s["density"] = _u32(n), torch.zeros(case["n_g"], device="cuda")
    elif kind == "push":
        g, x, v = _push_inputs(case, seed)
        n = case["particles"]
        s["grid"], s["src"] = g, [_plane(p, g.capacity) for p in (x, v[0], v[1], v[2])]
        s["dst"] = [torch.zeros(g.capacity, device="cuda") for _ in range(4)]
        s["efield"] = torch.from_numpy(_sheath_field(g.n_g)).cuda()
        s["factor"], s["dt"] = (g.factor_i, g.dt_i) if case["species"] == "i" else (g.factor_e, g.dt_e)
        s["n"], s["alive"], s["density"] = _u32(n), _u32(0), torch.zeros(g.n_g, device="cuda")
    elif kind in ("mcc_e", "mcc_i"):
        n = case["particles"]
        gen = _gen(seed)
        g = cp.grid_from_params(capacity=_pad4(n + n // 4), pressure=case["pressure"])
        if kind == "mcc_e":
            v = _electrons(n, gen)
            s["x"] = _plane(_bulk_x(n, gen), g.capacity)
            s["ions"] = [torch.zeros(g.capacity, device="cuda") for _ in range(4)]
            s["alive"], s["alive_i"] = _u32(n), _u32(0)
        else:  # thermal ions, one in twenty accelerated by a sheath (up to 30 eV)
            v = _maxwell(n, gen, AR_MASS, 0.03)
            fast = torch.rand(n, generator=gen, device="cuda") < 0.05
            ev = 30.0 * torch.rand(n, generator=gen, device="cuda")
            v[0] = torch.where(fast, (2.0 * ev * E_CHARGE / AR_MASS).sqrt(), v[0])
        s["grid"], s["v"], s["n"] = g, [_plane(p, g.capacity) for p in v], _u32(n)
        s["rng"] = _streams(g.capacity, seed)
        s["cs"], s["sigma_e"], s["sigma_i"], _, top = _tables(g)
        s["bound"] = top if case.get("bounded") else None
    elif kind == "electron_step":
        n = case["particles"]
        x, v = _step_inputs(case, seed)
        g = cp.grid_from_params(n_g=case["n_g"], capacity=_pad4(n + n // 4), weight=_weight(n),
                                pressure=case["pressure"])
        s["grid"], s["planes"] = g, [_plane(p, g.capacity) for p in (x, v[0], v[1], v[2])]
        s["rng"] = _streams(g.capacity, seed)
        s["ions"] = [torch.zeros(g.capacity, device="cuda") for _ in range(4)]
        s["other"] = [torch.zeros(g.capacity, device="cuda") for _ in range(4)]
        s["records"] = s["other"] + [torch.zeros(g.capacity, device="cuda") for _ in range(4)]
        s["efield"] = torch.from_numpy(_sheath_field(g.n_g)).cuda()
        s["cs"], s["sigma_e"], _, s["sigma_max"], _ = _tables(g)
        s["n_e"], s["n_i"], s["colliders"], s["ticket"], s["alive"] = (_u32(n), _u32(0), _u32(0), _u32(0), _u32(0))
        s["density"], s["density_i"] = torch.zeros(g.n_g, device="cuda"), torch.zeros(g.n_g, device="cuda")
    elif kind == "seed":
        s["n"], s["master"] = case["streams"], _master(seed)
        s["planes"] = [torch.empty(case["streams"], dtype=torch.int32, device="cuda") for _ in range(4)]
    elif kind in ("discharge", "sensitivity"):
        spec = DischargeSpec(voltage=250.0, pressure=PRESSURE, gap=GAP, n_g=case.get("n_g", 400),
                             particles=case["particles"], seed=seed)
        s["state"] = st = GpuSimState(spec.params(capacity_factor=1.5))
        e, i = initial_population(spec, st.grid.dt_e, st.grid.dt_i)
        st.upload_electrons(ParticlesSoA(*e))
        st.upload_ions(ParticlesSoA(*i))
        st.seed(e_master=_master(seed), i_master=_master(seed + 1))
        if kind == "discharge":
            s["pot"] = _pot_of(st, st)
        else:
            s["sens"] = VoltageSensitivity(st, window_steps=case["window"], checkpoint_every=case["checkpoint"])
    elif kind == "sweep":
        specs = c2_specs(case["discharges"], seed=case["sweep"])
        for k, spec in enumerate(specs):
            spec.seed = (seed * 1000 + k) % (1 << 31)
        s["batch"] = b = Batch(specs, capacity_factor=2.0)
        s["stream"] = torch.cuda.ExternalStream(b.batch.stream)
        s["pots"] = [_pot_of(st, b) for st in b.states]
    else:
        raise ValueError("unknown kind %r" % kind)
    return s


# --------------------------------------------------------------------- run

def run(s):
    return globals()["_run_" + s["kind"]](s)


def _run_solve(s):
    K.solve_poisson_scan_f32(s["e"], s["i"], s["pot"], s["efield"], s["pot0"], s["grid"])
    return {"pot": s["pot"], "efield": s["efield"]}


def _run_deposit(s):
    s["density"].zero_()
    K.get_density(s["x"], s["density"], s["n"], s["grid"])
    return {"density": s["density"]}


def _run_push(s):
    s["alive"].zero_()
    s["density"].zero_()
    args = (s["efield"], *s["src"], *s["dst"], s["alive"], s["n"], s["factor"], s["dt"])
    if s["case"]["deposit"]:
        K.move_and_compact_deposit(*args, s["density"], s["grid"])
    else:  # the reference's sequence: push, then the next step's deposit of the survivors
        K.move_and_compact(*args, s["grid"])
        K.get_density(s["dst"][0], s["density"], s["alive"], s["grid"])
    return {"alive": s["alive"], "density": s["density"]}


def _run_mcc_e(s):
    s["alive"].copy_(s["n"])
    K.check_collisions_e(s["sigma_e"], s["cs"], s["n"], s["x"], *s["v"], *s["rng"], *s["ions"], s["alive"],
                         s["alive_i"], s["grid"])
    return {"v": s["v"], "rng": s["rng"], "alive": s["alive"], "alive_i": s["alive_i"]}


def _run_mcc_i(s):
    K.check_collisions_i(s["sigma_i"], s["cs"], s["n"], *s["v"], *s["rng"], s["grid"], sigma_max_i=s["bound"])
    return {"v": s["v"], "rng": s["rng"]}


def _run_electron_step(s):
    s["density"].zero_()
    g = s["grid"]
    if s["case"]["inplace"]:
        K.step_electrons_inplace(s["efield"], *s["planes"], *s["rng"], s["sigma_e"], s["cs"], s["sigma_max"],
                                 s["n_e"], s["records"], s["colliders"], s["density"], g)
        K.scatter_colliders_e(*s["planes"], *s["rng"], s["cs"], s["records"], s["colliders"], s["ticket"], *s["ions"],
                              s["n_e"], s["n_i"], s["density"], s["density_i"], g)
        return {"planes": s["planes"], "rng": s["rng"], "n_e": s["n_e"], "density": s["density"]}
    s["alive"].zero_()   # the compacting step: survivors to the other side, in an unspecified order
    K.step_electrons(s["efield"], *s["planes"], *s["other"], *s["rng"], s["sigma_e"], s["cs"], s["sigma_max"],
                     *s["ions"], s["alive"], s["n_e"], s["n_i"], s["density"], s["density_i"], g)
    return {"rng": s["rng"], "alive": s["alive"], "density": s["density"]}


def _run_seed(s):
    K.xoshiro128_seed_streams(s["master"], s["n"], *s["planes"])
    return s["planes"]


def _run_discharge(s):
    st, case = s["state"], s["case"]
    if not case["measure"]:
        st.run_steps(case["steps"])
        return s["pot"]
    st.set_measure(True)
    st.run_steps(case["steps"])
    cumul_e, cumul_i, eepf = st.download_measurements()   # the window's averages, as a program saves them
    return {"n_e": cumul_e / case["steps"], "n_i": cumul_i / case["steps"],
            "eepf": eepf / max(1.0, float(eepf.sum())), "pot_xt": st.download_xt("pot"),
            "meanee": np.nanmean(st.download_xt("meanee"), axis=1)}


def _run_sweep(s):
    s["batch"].run_steps(s["case"]["steps"])
    with torch.cuda.stream(s["stream"]):   # every discharge's potential, gathered after the steps
        return torch.cat(s["pots"])


def _run_sensitivity(s):
    obs = s["sens"].forward(250.0)
    grad = s["sens"].backward()
    return {"obs": np.array([obs["power_e"], obs["ion_flux_gnd"]]),
            "grad": np.array([grad["power_e"], grad["ion_flux_gnd"]])}


# -------------------------------------------------------------------- work

def work(case):
    """Bytes each pass cannot do without: every input read once, every output written once."""
    kind, n, g = case["kind"], case.get("particles", 0), case.get("n_g", 400)
    if kind == "solve":
        return {"bytes": 16 * g, "flops": 20 * g}
    if kind == "deposit":
        return {"bytes": 4 * n + 4 * g, "flops": 8 * n}
    if kind == "push":
        return {"bytes": 32 * n + 8 * g, "flops": 20 * n}
    if kind in ("mcc_e", "mcc_i"):
        return {"bytes": 44 * n, "flops": 30 * n}
    if kind == "electron_step":
        return {"bytes": (56 if case["inplace"] else 64) * n + 8 * g, "flops": 60 * n}
    if kind == "seed":
        return {"bytes": 16 * case["streams"], "flops": 0}
    if kind == "sensitivity":   # forward, and per observable a recompute and a reverse sweep
        return _stepped(n, 5 * case["window"])
    if kind == "sweep":
        return _stepped(sum(sp.particles for sp in c2_specs(case["discharges"], seed=case["sweep"])), case["steps"])
    return _stepped(n, case["steps"])


def _stepped(n, steps):
    """Electrons (x, v, stream read; x, vx, stream written) every step, ions every 20th; a population that
    fits on the chip crosses HBM once."""
    if 2 * 32 * n <= ON_CHIP:
        return {"bytes": 2 * 56 * n, "flops": 63 * n * steps}
    return {"bytes": 56 * n * steps * 21 // 20, "flops": 63 * n * steps}


# ------------------------------------------------------------------- exact

def _deposit64(x, case):
    """CIC density in 64 bits (boundary nodes doubled)."""
    n_g = case["n_g"]
    dx = GAP / (n_g - 1)
    pos = x / dx
    p = np.clip(pos.astype(np.int64), 0, n_g - 2)
    rem = pos - p
    d = np.bincount(p, 1.0 - rem, n_g) + np.bincount(p + 1, rem, n_g)
    d *= _weight(case["particles"]) / (1e-4 * dx)
    d[[0, -1]] *= 2.0
    return d


def _push64(x, vx, field, factor, dt):
    n_g = len(field)
    pos = x * ((n_g - 1) / GAP)
    p = np.clip(pos.astype(np.int64), 0, n_g - 2)
    c = pos - p
    f = field.astype(np.float64)
    v = vx + factor * ((1.0 - c) * f[p] + c * f[p + 1])
    return x + v * dt, v


def _host64(t):
    return t.cpu().numpy().astype(np.float64)


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        e, i, pot0 = _densities(case, seed)
        n = case["n_g"]
        dx = GAP / (n - 1)
        rho = E_CHARGE * (i.astype(np.float64) - e.astype(np.float64))
        f = -dx * dx / EPS0 * rho[1:-1]
        f[0] -= pot0
        j = np.arange(1, n - 1, dtype=np.float64)
        r = -np.cumsum(j * f) / (j * (j + 1.0))
        pot = np.zeros(n)
        pot[0] = pot0
        pot[1:-1] = j * np.cumsum(r[::-1])[::-1]
        ef = np.zeros(n)
        ef[1:-1] = (pot[:-2] - pot[2:]) * (0.5 / dx)
        ef[0] = (pot[0] - pot[1]) / dx - rho[0] * dx / (2.0 * EPS0)
        ef[-1] = (pot[-2] - pot[-1]) / dx + rho[-1] * dx / (2.0 * EPS0)
        return {"pot": pot, "efield": ef}
    if kind == "deposit":
        return {"density": _deposit64(_host64(_bulk_x(case["particles"], _gen(seed))), case)}
    if kind == "push":
        g, x, v = _push_inputs(case, seed)
        factor, dt = (g.factor_i, g.dt_i) if case["species"] == "i" else (g.factor_e, g.dt_e)
        x1, _ = _push64(_host64(x), _host64(v[0]), _sheath_field(case["n_g"]), factor, dt)
        return {"alive": None, "density": _deposit64(x1[(x1 >= 0.0) & (x1 <= GAP)], case)}
    if kind == "electron_step":
        x, v = _step_inputs(case, seed)
        g = cp.grid_from_params(n_g=case["n_g"])
        x1, _ = _push64(_host64(x), _host64(v[0]), _sheath_field(case["n_g"]), g.factor_e, g.dt_e)
        density = _deposit64(x1, case)
        if not case["inplace"]:
            return {"rng": None, "alive": None, "density": density}
        plane = np.zeros(_pad4(len(x1) + len(x1) // 4))
        plane[:len(x1)] = x1
        return {"planes": [plane, None, None, None], "rng": None, "n_e": None, "density": density}
    return None
