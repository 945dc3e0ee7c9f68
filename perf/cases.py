"""Performance cases of the framework: what is timed, on which inputs, and how far outputs may move.

Every case is one call pattern of a user's program, through the public entry points (sphexa_b200.simulation,
.ensemble, .adjoint, and the C ABI of sphexa_b200.lib for the calls that take the caller's own arrays):

  step         a simulation restarted from a stored state, advanced by `steps` global time steps, state read back
  host_step    one step of a caller that keeps its particles in pinned host memory in the reference's default types
  stages       the force stages in place on a caller's device arrays (sphb_dataset_*), reference default types
  ensemble     independent members of uneven size uploaded from the device, advanced together (parameter sweep), and
               read to the host
  gradient     kinetic energy after `steps` steps and its gradient with respect to u0 and alphamax
  block_steps  a simulation uploaded from the device and advanced by substeps of the block time-step propagator
  order        SFC keys, key sort, gather and octree on caller-owned arrays

The particles are a Sedov blast in a periodic box, as the repository's initial conditions lay them out, at a time
when the shock has reached `radius`, or the Noh implosion in an open box.
"""
import ctypes as C
import math

import numpy as np
import torch

from sphexa_b200 import ic as icm
from sphexa_b200 import lib as L
from sphexa_b200.adjoint import AdjointRun
from sphexa_b200.ensemble import Ensemble
from sphexa_b200.ic import CONSERVED_FIELDS
from sphexa_b200.simulation import Simulation

#: fields that the reference's default types keep in double; the others are float
WIDE = ("x", "y", "z", "temp")
#: force outputs read beside the state
FORCES = ("ax", "ay", "az", "kx", "gradh", "divv")
DERIVED = ("xm", "kx", "gradh", "prho", "c", "rho", "p", "c11", "c12", "c13", "c22", "c23", "c33", "divv", "curlv",
           "ax", "ay", "az")
#: the exact results are computed up to this many particles
EXACT_MAX = 70_000
#: flops per neighbour pair of the five pair loops (XMass, VeDefGradh, IAD + divv/curlv, AV switches, momentum-energy)
PAIR_FLOPS = 18 + 31 + 88 + 55 + 140
NEIGHBOURS = 100


def listed():
    return [
        # the smallest simulation: a test or a notebook run, bound by launches and host reads
        {"name": "step16_mixed", "kind": "step", "problem": "blast", "side": 16, "precision": "mixed",
         "radius": 0.25, "av_clean": False, "steps": 10},
        # the reference's small regression size, in the all-double drop-in form
        {"name": "step30_fp64", "kind": "step", "problem": "blast", "side": 30, "precision": "fp64", "radius": 0.25,
         "av_clean": False, "steps": 10},
        # an ordinary run (the reference's regression tests use 50^3) with AV cleaning
        {"name": "step50_avclean", "kind": "step", "problem": "blast", "side": 50, "precision": "mixed",
         "radius": 0.3, "av_clean": True, "steps": 8},
        # the headline workload: production resolution, an early blast, mixed precision
        {"name": "step128_mixed", "kind": "step", "problem": "blast", "side": 128, "precision": "mixed",
         "radius": 0.12, "av_clean": False, "steps": 6},
        # a large all-double run of odd size, the blast well developed
        {"name": "step101_fp64", "kind": "step", "problem": "blast", "side": 101, "precision": "fp64",
         "radius": 0.3, "av_clean": False, "steps": 4},
        # every particle moves: the Noh implosion (open box, ragged size, a tree search every step)
        {"name": "noh81_mixed", "kind": "step", "problem": "noh", "side": 81, "precision": "mixed", "radius": 0.0,
         "av_clean": False, "steps": 8},
        # the drop-in step of a host code: copies to and from host memory every step
        {"name": "host100_mixed", "kind": "host_step", "side": 100, "precision": "mixed", "radius": 0.12},
        # the drop-in stages of the reference's propagator on its own device arrays
        {"name": "stages63_mixed", "kind": "stages", "side": 63, "precision": "mixed", "radius": 0.2},
        # a parameter sweep: uneven members, differing energies and gammas
        {"name": "ensemble16", "kind": "ensemble", "members": 16, "low": 20, "high": 48, "precision": "mixed",
         "radius": 0.2, "steps": 30},
        # gradients of a run (forward, checkpoints, recorded replay, adjoint)
        {"name": "gradient48_mixed", "kind": "gradient", "side": 48, "precision": "mixed", "steps": 20, "every": 5,
         "radius": 0.2},
        # block time steps: eight substeps, forces on the active rungs
        {"name": "block64_mixed", "kind": "block_steps", "side": 64, "precision": "mixed", "radius": 0.2,
         "steps": 8},
        # the domain primitives on caller-owned arrays of millions of particles
        {"name": "order4m", "kind": "order", "n": 4_000_037, "bucket": 64},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "host_step", "stages", "ensemble", "gradient", "block_steps",
                       "order"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    radius = round(rng.uniform(0.1, 0.4), 3)
    if kind == "step":
        problem = rng.choice(["blast", "blast", "blast", "noh"])
        side = _log_int(rng, 13, 110 if precision == "mixed" else 84)
        if problem == "noh":
            side = min(max(side, 17), 90)
        return {"kind": kind, "problem": problem, "side": side, "precision": precision,
                "radius": radius if problem == "blast" else 0.0, "av_clean": rng.random() < 0.25,
                "steps": rng.randint(3, 6) if side > 60 else rng.randint(5, 12)}
    if kind in ("host_step", "stages"):
        return {"kind": kind, "side": _log_int(rng, 13, 90), "precision": precision, "radius": radius}
    if kind == "ensemble":
        low = rng.randint(14, 24)
        return {"kind": kind, "members": rng.randint(3, 24), "low": low, "high": low + rng.randint(1, 16),
                "precision": precision, "radius": radius, "steps": rng.randint(10, 30)}
    if kind == "gradient":
        every = rng.randint(2, 5)
        return {"kind": kind, "side": rng.randint(14, 40), "precision": precision, "every": every,
                "steps": every * rng.randint(1, 3) + rng.randint(0, 1), "radius": radius}
    if kind == "block_steps":
        return {"kind": kind, "side": _log_int(rng, 18, 60), "precision": precision, "radius": radius,
                "steps": rng.randint(4, 12)}
    return {"kind": "order", "n": _log_int(rng, 3_000, 4_000_000), "bucket": rng.choice([16, 64, 64, 256])}


# -------------------------------------------------------------------------------------------------------------------
# inputs
# -------------------------------------------------------------------------------------------------------------------

def blast(side, seed, radius, energy=1.0, gamma=5.0 / 3.0, av_clean=False):
    """The Sedov lattice with the particles inside `radius` moved to a blast wave's profile: enclosed mass
    (r / radius)^5 (density 5/3 (r / radius)^2: an evacuated centre and a shell, as the smoothed profile of a run has
    them), velocity linear in r up to the post-shock speed, a pressure plateau inside, cold gas outside, and a slow
    smooth motion of all the gas."""
    f = icm.sedov(side, seed=seed, energy=energy, gamma=gamma)
    f["params"]["avClean"] = av_clean
    p = f["params"]
    x = np.stack([f["x"], f["y"], f["z"]])
    r0 = np.sqrt((x * x).sum(0))
    inside = r0 < radius
    q = np.where(inside, np.maximum(r0 / radius, 1e-6), 1.0)
    s = q ** 0.6  # new radius over `radius`, where it was q
    x = x * np.where(inside, s / q, 1.0)
    rho = np.where(inside, 5.0 / 3.0 * s * s, 1.0)
    shock = math.sqrt(energy)
    pressure = 2.0 / (gamma + 1.0) * shock ** 2 * (0.5 + 0.5 * s ** 8)
    u = np.where(inside, pressure / ((gamma - 1.0) * rho), 1e-4)
    rng = np.random.default_rng(seed)
    v = np.where(inside, 2.0 / (gamma + 1.0) * shock, 0.0) * x / radius
    for _ in range(4):
        k = rng.integers(1, 3, 3) * rng.choice([-1, 1], 3)
        v += 0.02 * shock * rng.normal(size=(3, 1)) * np.sin(2.0 * math.pi * (k @ x) + rng.uniform(0.0, 6.28))
    # the sphere of 2 h near the centre holds the denser gas around it: the mean density there, for 100 neighbours
    middle = (100.0 / (side ** 3 * 4.0 / 3.0 * math.pi * radius ** 3)) ** 0.4
    h = f["h"] * np.where(inside, rho + middle, 1.0) ** (-1.0 / 3.0)
    c = np.sqrt(gamma * (gamma - 1.0) * u)
    dt = float(0.1 * np.min(h / (c + np.sqrt((v * v).sum(0)))))
    f.update(x=x[0], y=x[1], z=x[2], vx=v[0], vy=v[1], vz=v[2], x_m1=v[0] * dt, y_m1=v[1] * dt, z_m1=v[2] * dt, h=h,
             temp=u / icm.ideal_gas_cv(p["mui"], gamma), alpha=np.where(inside, 0.05 + 0.6 * s ** 4, 0.05))
    p.update(minDt=dt, minDt_m1=dt)
    return f


def initial(case, seed):
    if case.get("problem") == "noh":
        f = icm.noh(case["side"], seed=seed)
        f["params"]["avClean"] = case["av_clean"]
        # the jitter moves particles across the cut: keep the innermost ones, the same number for every seed
        keep = np.argsort(f["x"] ** 2 + f["y"] ** 2 + f["z"] ** 2, kind="stable")[:int(0.98 * _size(case))]
        keep.sort()
        f.update({k: f[k][keep] for k in CONSERVED_FIELDS})
        f["id"] = np.arange(keep.size, dtype=np.uint64)
        return f
    return blast(case["side"], seed, case["radius"], av_clean=case.get("av_clean", False))


def members(case, seed):
    rng = np.random.default_rng(seed)
    sides = np.random.default_rng(case["members"]).integers(case["low"], case["high"] + 1, case["members"])
    sides[0], sides[-1] = case["low"], case["high"]
    return [blast(int(side), int(seed) * 97 + k, case["radius"], energy=float(rng.uniform(0.5, 2.0)),
                  gamma=float(rng.choice([1.4, 5.0 / 3.0]))) for k, side in enumerate(sides)]


def _state_buffers(n):
    return [torch.empty(n, dtype=torch.float64, device="cuda") for _ in CONSERVED_FIELDS], \
        torch.empty(n, dtype=torch.int64, device="cuda")


def _typed(sim, to):
    """The simulation's state in the reference's default types, in pinned host memory or on the device."""
    opts = {"pin_memory": True} if to == "cpu" else {"device": "cuda"}
    d = {f: torch.empty(sim.n, dtype=torch.float64 if f in WIDE else torch.float32, **opts) for f in CONSERVED_FIELDS}
    d["id"] = torch.empty(sim.n, dtype=torch.int64, **opts)
    tbl = L.make_fields(d)
    L.check(sim.lib.sphb_sim_store_fields(sim.h, tbl, len(tbl), int(to != "cpu")), "store_fields")
    return d


def prepare(case, seed):
    kind = case["kind"]
    if kind == "order":
        g = torch.Generator(device="cuda").manual_seed(seed)
        n = case["n"]
        uniform = torch.rand((3, n), generator=g, device="cuda", dtype=torch.float64) - 0.5
        centre = torch.rand((3, 16), generator=g, device="cuda", dtype=torch.float64) - 0.5
        which = torch.randint(16, (n,), generator=g, device="cuda")
        clump = 0.03 * torch.randn((3, n), generator=g, device="cuda", dtype=torch.float64) + centre[:, which]
        p = torch.where(torch.rand(n, generator=g, device="cuda") < 0.6, clump - torch.floor(clump + 0.5), uniform)
        p = p.clamp(-0.5, 0.5)
        h = 0.01 + 0.01 * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
        lib = L.load()
        cap = n // 2 + 4096
        scratch = int(lib.sphb_sort_by_key_scratch_bytes(n))
        src = [p[0].contiguous(), p[1].contiguous(), p[2].contiguous(), h]
        dst = [torch.empty_like(a) for a in src]
        return {"case": case, "lib": lib, "n": n, "cap": cap, "src": src, "dst": dst,
                "box": L.make_box((-0.5, 0.5) * 3, [1, 1, 1]),
                "keys": torch.empty(n, dtype=torch.int64, device="cuda"),
                "order": torch.empty(n, dtype=torch.int32, device="cuda"),
                "scratch": torch.empty(scratch, dtype=torch.uint8, device="cuda"),
                "leaves": torch.zeros(cap, dtype=torch.int64, device="cuda"),
                "counts": torch.zeros(cap, dtype=torch.int32, device="cuda")}
    if kind == "ensemble":
        ics = members(case, seed)
        start = [([torch.from_numpy(np.ascontiguousarray(ic[f])).cuda() for f in CONSERVED_FIELDS],
                  torch.from_numpy(ic["id"].astype(np.int64)).cuda()) for ic in ics]
        tables = [(C.c_void_p * len(fields))(*[a.data_ptr() for a in fields]) for fields, _ in start]
        return {"case": case, "ens": Ensemble(ics, case["precision"]), "start": start, "tables": tables}
    ic = initial(case, seed)
    if kind == "gradient":
        run = AdjointRun(ic, case["precision"], dt=ic["params"]["minDt"], steps=case["steps"], checkpoint_every=case["every"])
        u0 = ic["temp"] * icm.ideal_gas_cv(ic["params"]["mui"], ic["params"]["gamma"])
        return {"case": case, "run": run, "u0": u0}
    sim = Simulation(ic, case["precision"])
    state = {"case": case, "sim": sim, "dt": ic["params"]["minDt"]}
    fields, ids = _state_buffers(sim.n)
    if kind == "step":
        sim.store_state(fields, ids)
        out, out_ids = _state_buffers(sim.n)
        state.update(start=(fields, ids), out=(out, out_ids),
                     forces=[torch.empty(sim.n, dtype=torch.float64, device="cuda") for _ in FORCES])
    elif kind == "block_steps":
        sim.enable_block_timesteps()
        sim.store_state(fields, ids)
        state.update(start=dict(zip(CONSERVED_FIELDS, fields), id=ids), out=_state_buffers(sim.n))
    elif kind == "host_step":
        given = _typed(sim, "cpu")
        result = {f: torch.empty(a.shape, dtype=a.dtype, pin_memory=True) for f, a in given.items()}
        state.update(given=given, result=result, in_tbl=L.make_fields(given), out_tbl=L.make_fields(result))
    else:
        d = _typed(sim, "cuda")
        for f in DERIVED:
            d[f] = torch.zeros(sim.n, dtype=torch.float32, device="cuda")
        d["du"] = torch.zeros(sim.n, dtype=torch.float64, device="cuda")
        d["nc"] = torch.zeros(sim.n, dtype=torch.int32, device="cuda")
        d["keys"] = torch.zeros(sim.n, dtype=torch.int64, device="cuda")
        work = Simulation(ic, case["precision"], initial_sync=False)
        tbl = L.make_fields(d)
        torch.cuda.synchronize()
        L.check(work.lib.sphb_sim_bind_fields(work.h, tbl, len(tbl)), "bind_fields")
        eos = {f: d[f] for f in ("temp", "m", "kx", "xm", "gradh", "prho", "c", "rho", "p")}
        state.update(sim=work, d=d, box=L.make_box(ic["box"], [ic["periodic"]] * 3), eos=L.make_fields(eos),
                     mui=ic["params"]["mui"], gamma=ic["params"]["gamma"])
    return state


# -------------------------------------------------------------------------------------------------------------------
# one pass
# -------------------------------------------------------------------------------------------------------------------

def _restart(sim, dt):
    """the next step starts from the previous time step dt and chooses its own"""
    sim.set_fixed_dt(dt)
    sim.set_fixed_dt(0.0)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        sim = state["sim"]
        sim.load_state(*state["start"])
        _restart(sim, state["dt"])
        for _ in range(case["steps"]):
            sim.step()
        sim.store_state(*state["out"])
        for f, a in zip(FORCES, state["forces"]):
            sim.get_device(f, a)
        out = dict(zip(CONSERVED_FIELDS, state["out"][0]), id=state["out"][1])
        out.update(zip(FORCES, state["forces"]))
        return out
    if kind == "host_step":
        sim = state["sim"]
        _restart(sim, state["dt"])
        a, b = state["in_tbl"], state["out_tbl"]
        L.check(sim.lib.sphb_sim_step_fields(sim.h, a, len(a), b, len(b)), "step_fields")
        return state["result"]
    if kind == "stages":
        sim, box, d = state["sim"], state["box"], state["d"]
        lib, h, n = sim.lib, sim.h, sim.n
        L.check(lib.sphb_dataset_xmass(h, 0, n, C.byref(box)), "xmass")
        L.check(lib.sphb_dataset_ve_def_gradh(h, 0, n, C.byref(box)), "ve_def_gradh")
        L.check(lib.sphb_ideal_gas_eos(0, n, state["mui"], state["gamma"], state["eos"], len(state["eos"]),
                                       lib.sphb_sim_stream(h)), "eos")
        L.check(lib.sphb_dataset_iad_divv_curlv(h, 0, n, C.byref(box)), "iad")
        L.check(lib.sphb_dataset_av_switches(h, 0, n, C.byref(box), state["dt"]), "av")
        courant = C.c_float()
        L.check(lib.sphb_dataset_momentum_energy(h, 0, n, C.byref(box), C.byref(courant)), "momentum_energy")
        out = {f: d[f] for f in ("h", "nc", "xm", "alpha", "du") + DERIVED[1:]}
        out["courant"] = courant.value
        return out
    if kind == "ensemble":
        ens = state["ens"]
        for k, (table, (_, ids)) in enumerate(zip(state["tables"], state["start"])):
            L.check(ens.lib.sphb_ensemble_upload(ens.h, k, table, L.ptr(ids), 1), "ensemble_upload")
        L.check(ens.lib.sphb_ensemble_initial_sync(ens.h), "ensemble_initial_sync")
        ens.step(case["steps"])
        return {f: np.concatenate([ens.get(k, f) for k in range(ens.num)])
                for f in ("x", "y", "z", "vx", "vy", "vz", "temp", "h")}
    if kind == "gradient":
        r = state["run"]
        value = r.forward(state["u0"], 1.0)
        grad_u0, grad_alphamax = r.backward()
        return {"value": value, "grad_u0": grad_u0, "grad_alphamax": grad_alphamax}
    if kind == "block_steps":
        sim = state["sim"]
        sim.upload(state["start"], on_device=True)
        sim.initial_sync()
        for _ in range(case["steps"]):
            sim.bdt_step()
        sim.store_state(*state["out"])
        return dict(zip(CONSERVED_FIELDS, state["out"][0]), id=state["out"][1])
    s, lib, n = state, state["lib"], state["n"]
    stream = torch.cuda.current_stream().cuda_stream
    x, y, z, h = s["src"]
    L.check(lib.sphb_compute_sfc_keys(L.ptr(x), L.ptr(y), L.ptr(z), L.ptr(s["keys"]), n, C.byref(s["box"]), stream),
            "sfc_keys")
    L.check(lib.sphb_sort_by_key(L.ptr(s["keys"]), L.ptr(s["order"]), n, 1, L.ptr(s["scratch"]),
                                 s["scratch"].numel(), stream), "sort_by_key")
    src = (C.c_void_p * 4)(*[a.data_ptr() for a in s["src"]])
    dst = (C.c_void_p * 4)(*[a.data_ptr() for a in s["dst"]])
    L.check(lib.sphb_gather8(L.ptr(s["order"]), n, 4, src, dst, stream), "gather8")
    leaves = C.c_size_t()
    L.check(lib.sphb_compute_octree(L.ptr(s["keys"]), n, case["bucket"], L.ptr(s["leaves"]), L.ptr(s["counts"]),
                                    s["cap"], C.byref(leaves), stream), "octree")
    return {"keys": s["keys"], "order": s["order"], "fields": s["dst"], "leaves": s["leaves"], "counts": s["counts"],
            "num_leaves": leaves.value}


# -------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far its outputs may be off
# -------------------------------------------------------------------------------------------------------------------

def _size(case):
    if case["kind"] == "ensemble":
        mid = 0.5 * (case["low"] + case["high"])
        return case["members"] * mid ** 3
    return case["side"] ** 3 * (math.pi / 6 if case.get("problem") == "noh" else 1.0)


def work(case):
    if case["kind"] == "order":
        # coordinates read, keys and order written, four fields gathered, keys read and a leaf (key, count) per
        # bucket / 2 particles written
        n = case["n"]
        return {"bytes": n * (24 + 8 + 4 + 64 + 8) + 12 * n / (case["bucket"] / 2), "flops": 0}
    n = _size(case)
    steps = case.get("steps", 1)
    state = 15 * 8  # 14 conserved fields and the id, 8 bytes each
    pairs = n * NEIGHBOURS * PAIR_FLOPS
    if case["kind"] == "host_step":
        return {"bytes": n * 2 * 80, "flops": pairs}
    if case["kind"] == "stages":
        return {"bytes": n * (80 + 4 * 26), "flops": pairs}
    if case["kind"] == "gradient":
        # forward, replay, and an adjoint of twice a step's operations
        return {"bytes": 4 * steps * n * 2 * state, "flops": 4 * steps * pairs}
    if case["kind"] == "block_steps":
        # about half the particles are active in a substep
        return {"bytes": steps * n * 2 * state, "flops": 0.5 * steps * pairs}
    return {"bytes": steps * n * 2 * state, "flops": steps * pairs}


def tolerance(case):
    """About four times what the mixed and the all-double form of the same case differ by (1e-6 to 9e-6 for most
    outputs, 4e-5 with AV cleaning, whose limiter divides nearly cancelling sums, and after the ensemble's many steps;
    single particles more, where a neighbour count or a switch falls the other way)."""
    if case["kind"] == "order":
        return "exact"
    if case["precision"] == "fp64":
        return {"rel": 1e-9, "max": 1e-6}
    if case.get("av_clean") or case["kind"] == "ensemble":
        return {"rel": 1.5e-4, "max": 0.03}
    return {"rel": 4e-5, "max": 5e-3}


# -------------------------------------------------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# -------------------------------------------------------------------------------------------------------------------

TABLE = 20000
LEVELS = 21


def _kernel_tables(dev):
    """W = sinc(pi v / 2)^6 and its derivative at 20000 points of [0, 2], and the normalisation 1 / integral."""
    def sinc(v):
        a = 0.5 * math.pi * v
        return torch.where(v > 0, torch.sin(a) / torch.where(v > 0, a, 1.0), 1.0)

    v = torch.arange(TABLE, dtype=torch.float64, device=dev) * (2.0 / (TABLE - 1))
    s = sinc(v)
    a = 0.5 * math.pi * v
    safe = torch.where(v > 0, a, 1.0)
    ds = torch.where(v > 0, 0.5 * math.pi * (torch.cos(a) / safe - torch.sin(a) / (safe * safe)), 0.0)
    g = torch.linspace(0.0, 2.0, 2001, dtype=torch.float64, device=dev)
    f = 4.0 * math.pi * g * g * sinc(g) ** 6
    integral = (f[0] + f[-1] + 4.0 * f[1:-1:2].sum() + 2.0 * f[2:-1:2].sum()) * (2.0 / 2000) / 3.0
    return s ** 6, 6.0 * s ** 5 * ds, float(1.0 / integral)


def _lookup(table, v):
    inv = (TABLE - 1) / 2.0
    i = (v.detach() * inv).to(torch.int64).clamp(0, TABLE - 2)
    t0, t1 = table[i], table[i + 1]
    return torch.where(v * inv < TABLE - 1, t0 + (t1 - t0) * inv * (v - i.to(v.dtype) * (2.0 / (TABLE - 1))), 0.0)


def _hilbert(p, lo, hi):
    """Hilbert keys of the points p (3 tensors) on 2^21 cells an axis."""
    q = []
    for a, l, u in zip(p, lo, hi):
        m = 2.0 ** LEVELS * (1.0 / (u - l))
        q.append((torch.floor(a * m) - l * m).to(torch.int64).clamp(max=2 ** LEVELS - 1))
    x, y, z = q
    digit = torch.tensor([0, 1, 3, 2, 7, 6, 4, 5], device=x.device)
    key = torch.zeros_like(x)
    for level in range(LEVELS - 1, -1, -1):
        xi, yi, zi = (x >> level) & 1, (y >> level) & 1, (z >> level) & 1
        key = (key << 3) + digit[4 * xi + 2 * yi + zi]
        ny, nz = 1 - yi, 1 - zi
        x = x ^ -(xi & (ny | zi))
        y = y ^ -((xi & (yi | zi)) | (yi & nz))
        z = z ^ -((xi & ny & nz) | (yi & nz))
        cycle, swap = zi == 1, (zi == 0) & (yi == 0)
        x, y, z = torch.where(cycle, y, torch.where(swap, z, x)), torch.where(cycle, z, y), \
            torch.where(cycle, x, torch.where(swap, x, z))
    return key


class Exact:
    """One simulation in 64 bits on torch tensors: dense neighbour search, padded lists."""

    def __init__(self, ic, dev, typed=False):
        self.p = ic["params"]
        self.periodic = ic["periodic"]
        self.lo, self.hi = list(ic["box"][0::2]), list(ic["box"][1::2])
        self.f = {k: torch.from_numpy(np.ascontiguousarray(ic[k])).to(dev) for k in CONSERVED_FIELDS}
        self.id = torch.from_numpy(ic["id"].astype(np.int64)).to(dev)
        self.wh, self.whd, self.K = _kernel_tables(dev)
        self.cv = icm.ideal_gas_cv(self.p["mui"], self.p["gamma"])
        self.dt = self.dt_m1 = self.p["minDt"]
        self.first = True
        self.alphamax = self.p["alphamax"]
        self.sync()
        if typed:
            self.f = {k: a if k in WIDE else a.float().double() for k, a in self.f.items()}

    def sync(self):
        if not self.periodic:
            for k, a in enumerate("xyz"):
                lo, hi = float(self.f[a].min()), float(self.f[a].max())
                if not self.first:
                    size = self.hi[k] - self.lo[k]
                    lo, hi = min(lo, self.lo[k] + 0.05 * size), max(hi, self.hi[k] - 0.05 * size)
                self.lo[k], self.hi[k] = lo, hi
        self.first = False
        order = torch.sort(_hilbert([self.f[a].detach() for a in "xyz"], self.lo, self.hi), stable=True)[1]
        self.f = {k: a[order] for k, a in self.f.items()}
        self.id = self.id[order]

    def _near(self, rows, h):
        """(counts, particle of each pair's row, neighbour) of the particles `rows`, neighbours ascending"""
        P = [self.f[a].detach() for a in "xyz"]
        n = P[0].numel()
        size = max(1, int(1.5e8) // n)
        counts, where, who = [], [], []
        for b in range(0, rows.numel(), size):
            r = rows[b:b + size]
            d2 = 0.0
            for k in range(3):
                d = P[k][r][:, None] - P[k][None, :]
                if self.periodic:
                    span = self.hi[k] - self.lo[k]
                    d = d - span * torch.round(d * (1.0 / span))
                d2 = d2 + d * d
            hit = d2 < (4.0 * h[r] * h[r])[:, None]
            hit[torch.arange(r.numel(), device=r.device), r] = False
            counts.append(hit.sum(1))
            at = hit.nonzero()
            where.append(at[:, 0] + b)
            who.append(at[:, 1])
        return torch.cat(counts), torch.cat(where), torch.cat(who)

    def search(self):
        ng0, ngmax = self.p["ng0"], self.p["ngmax"]
        h = self.f["h"].detach().clone()
        n = h.numel()
        dev = h.device
        rows = torch.arange(n, device=dev)
        nc = torch.zeros(n, dtype=torch.int64, device=dev)
        self.nbr = torch.zeros((n, ngmax), dtype=torch.int64, device=dev)
        factor = torch.ones(n, dtype=torch.float64, device=dev)
        for it in range(11):
            count, where, who = self._near(rows, h)
            start = torch.cumsum(count, 0) - count
            slot = torch.arange(who.numel(), device=dev) - start[where]
            keep = slot < ngmax
            self.nbr[rows[where[keep]], slot[keep]] = who[keep]
            nc[rows] = count + 1
            bad = (ng0 // 4 > nc[rows]) | (nc[rows] - 1 > ngmax)
            rows = rows[bad]
            if it == 10 or rows.numel() == 0:
                break
            grow = 0.5 * (1.0 + 1023.0 * ng0 / nc[rows].double()) ** 0.1
            h[rows] = h[rows] * grow
            factor[rows] = factor[rows] * grow
        self.nc = nc
        self.f["h"] = self.f["h"] * factor
        kept = (nc - 1).clamp(max=ngmax)
        width = max(int(kept.max()), 1)
        self.nbr = self.nbr[:, :width]
        self.mask = torch.arange(width, device=dev)[None, :] < kept[:, None]

    def forces(self):
        f, p, j, mask, K = self.f, self.p, self.nbr, self.mask, self.K
        h, m = f["h"], f["m"]
        zero = torch.zeros((), dtype=torch.float64, device=h.device)

        def total(a):
            return torch.where(mask, a, zero).sum(1)

        r = []
        for k, a in enumerate("xyz"):
            d = f[a][:, None] - f[a][j]
            if self.periodic:
                d = d - (self.hi[k] - self.lo[k]) * torch.round(d.detach() * (1.0 / (self.hi[k] - self.lo[k])))
            r.append(torch.where(mask, d, 1e-3))
        dist = torch.sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2])
        hi = h[:, None]
        w = _lookup(self.wh, dist / hi)
        norm = K / h ** 3
        self.xm = xm = m / ((m + total(w * m[j])) * norm)
        dterh = -(3.0 * w + dist / hi * _lookup(self.whd, dist / hi))
        kx = (xm + total(w * xm[j])) * norm
        whomega = (-3.0 * xm + total(dterh * xm[j])) * norm / h
        wrho0 = (-3.0 * m + total(dterh * m[j])) * norm / h
        whomega = whomega * m / xm + (kx - norm * xm) * wrho0
        rho = kx * m / xm
        gradh = 1.0 + h / (3.0 * rho) * whomega
        tmp = self.cv * f["temp"] * (p["gamma"] - 1.0)
        c = torch.sqrt(p["gamma"] * tmp)
        prho = rho * tmp / (kx * m * m * gradh)
        vol = xm / kx
        t = [total(r[a] * r[b] * (vol[j] * w)) for a, b in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))]
        det = t[0] * t[3] * t[5] + 2.0 * t[1] * t[4] * t[2] - t[0] * t[4] ** 2 - t[3] * t[2] ** 2 - t[5] * t[1] ** 2
        fac = h ** 3 / (det * K)
        cij = [(t[3] * t[5] - t[4] ** 2) * fac, (t[2] * t[4] - t[5] * t[1]) * fac, (t[1] * t[4] - t[3] * t[2]) * fac,
               (t[0] * t[5] - t[2] ** 2) * fac, (t[2] * t[1] - t[0] * t[4]) * fac, (t[0] * t[3] - t[1] ** 2) * fac]
        pick = ((0, 1, 2), (1, 3, 4), (2, 4, 5))

        def gradient(of, weight):
            return [-sum(of(cij[q]) * r[b] for b, q in enumerate(pick[a])) * weight for a in range(3)]

        tA = gradient(lambda a: a[:, None], w)
        v = [f[a] for a in ("vx", "vy", "vz")]
        dv = [[total((v[a][j] - v[a][:, None]) * xm[j] * tA[b]) * norm / kx for b in range(3)] for a in range(3)]
        divv = dv[0][0] + dv[1][1] + dv[2][2]
        curl = ((dv[2][1] - dv[1][2]).detach() ** 2 + (dv[0][2] - dv[2][0]).detach() ** 2
                + (dv[1][0] - dv[0][1]).detach() ** 2)
        # artificial viscosity switches
        vij = [a[:, None] - a[j] for a in v]
        rv = r[0] * vij[0] + r[1] * vij[1] + r[2] * vij[2]
        vsig = torch.where(mask & (rv < 0), c[:, None] + c[j] - 3.0 * rv / dist, zero)
        vsig = torch.maximum(1e-40 * c, vsig.max(1)[0])
        gd = [total(vol[j] * (divv[:, None] - divv[j]) * a * norm[:, None]) for a in tA]
        g2 = gd[0] ** 2 + gd[1] ** 2 + gd[2] ** 2
        gd = torch.where(g2 > 0, torch.sqrt(torch.where(g2 > 0, g2, 1.0)), zero)
        const = h * h * gd
        alphaloc = torch.where(divv < 0, self.alphamax * const / (const + h * torch.abs(divv) + 0.05 * c), zero)
        alpha = f["alpha"]
        decay = h / (p["decay_constant"] * vsig)
        rate = (torch.where(alphaloc >= p["alphamin"], alphaloc, p["alphamin"] + zero) - alpha) / decay
        alpha = torch.where(alphaloc >= alpha, alphaloc, alpha + rate * self.dt)
        # momentum and energy
        wi, wj = w / hi ** 3, _lookup(self.wh, dist / h[j]) / h[j] ** 3
        tAi, tAj = gradient(lambda a: a[:, None], wi), gradient(lambda a: a[j], wj)
        if p.get("avClean"):
            g = [a.detach() for a in (dv[0][0], dv[0][1] + dv[1][0], dv[0][2] + dv[2][0], dv[1][1],
                                      dv[1][2] + dv[2][1], dv[2][2])]

            def quad(of):
                return (r[0] * (of(g[0]) * r[0] + of(g[1]) * r[1] + of(g[2]) * r[2])
                        + r[1] * (of(g[3]) * r[1] + of(g[4]) * r[2]) + r[2] * of(g[5]) * r[2])

            d1, d2 = quad(lambda a: a[:, None]), quad(lambda a: a[j])
            crit = (32.0 * math.pi / 3.0 / (mask.sum(1) + 1).double()) ** (1.0 / 3.0)
            eta = torch.minimum(dist / hi, dist / h[j]) - crit[:, None]
            d3 = torch.where(eta < 0, torch.exp(-(5.0 * eta) ** 2), 1.0 + zero)
            A = torch.where(d2 != 0, d1 / torch.where(d2 != 0, d2, 1.0), zero)
            q = (4.0 * A / ((1.0 + A) * (1.0 + A))).clamp(0.0, 1.0)
            rv = rv - 0.5 * d3 * q * (d1 + d2)
        wij = rv / dist
        cc = c[:, None] + c[j]
        visc = torch.where(wij < 0, -((alpha[:, None] + alpha[j]) * 0.25 * cc - 2.0 * wij) * wij, zero)
        self.vmax = torch.where(mask, 0.5 * cc - 2.0 * wij, zero).detach().max(1)[0].clamp(min=0.0)
        ri, rj = rho[:, None], rho[j]
        atwood = torch.abs(ri - rj) / (ri + rj)
        s = (10.0 * (atwood - 0.1)).clamp(0.0, 1.0)
        xi, xj = xm[:, None], xm[j]
        li, lj = torch.log(xi), torch.log(xj)
        ramp = (atwood >= 0.1) & (atwood <= 0.2)
        sr = torch.where(ramp, s, 0.5 + zero)
        am = torch.where(ramp, torch.exp((2.0 - sr) * li + sr * lj), torch.where(atwood < 0.1, xi * xi, xi * xj))
        bm = torch.where(ramp, torch.exp((2.0 - sr) * lj + sr * li), torch.where(atwood < 0.1, xj * xj, xi * xj))
        mj = m[j]
        av, bv = mj / ri * visc, mj / rj * visc
        acc, ev, ee = [], 0.0, 0.0
        for k in range(3):
            push = 0.5 * (av * tAi[k] + bv * tAj[k])
            ev = ev + push * vij[k]
            ee = ee + vij[k] * tAi[k]
            acc.append(-K * total(mj * prho[:, None] * am * tAi[k] + mj * prho[j] * bm * tAj[k] + push))
        self.a = acc
        self.du = K * (prho * total(mj * am * ee) + 0.5 * torch.relu(total(ev)))
        f["alpha"] = alpha
        self.c, self.divv, self.kx, self.gradh = c, divv, kx, gradh
        self.more = dict(prho=prho, c=c, rho=rho, p=rho * tmp, divv=divv, curlv=torch.sqrt(curl),
                         **dict(zip(("c11", "c12", "c13", "c22", "c23", "c33"), cij)))
        speed = torch.where(self.vmax > 0, self.vmax, c.detach())
        self.courant = float((float(np.float32(p["Kcour"])) * h.detach() / speed).min())
        top = abs(float(divv.max()))
        self.rho_dt = p["Krho"] / top if top else math.inf

    def integrate(self, fixed=None):
        f = self.f
        dt = fixed if fixed else min(self.courant, self.rho_dt, 1.1 * self.dt)
        self.dt_m1, self.dt = self.dt, dt
        m1 = self.dt_m1
        for k, (x, v, xm1) in enumerate((("x", "vx", "x_m1"), ("y", "vy", "y_m1"), ("z", "vz", "z_m1"))):
            vn = f[xm1] / m1 + 0.5 * m1 * self.a[k]
            f[v] = vn + self.a[k] * dt
            f[xm1] = (vn + 0.5 * self.a[k] * dt) * dt
            X = f[x] + f[xm1]
            if self.periodic:
                span = self.hi[k] - self.lo[k]
                X = torch.where(X > self.hi[k], X - span, torch.where(X < self.lo[k], X + span, X))
            f[x] = X
        u = self.cv * f["temp"]
        new = u + self.du * dt + 0.5 * (self.du - f["du_m1"]) / m1 * dt * dt
        low = new < 0
        f["temp"] = torch.where(low, u * torch.exp(torch.where(low, new * dt / u, 0.0)), new) / self.cv
        f["du_m1"] = self.du
        f["h"] = f["h"] * 0.5 * (1.0 + 1023.0 * self.p["ng0"] / self.nc.double()) ** 0.1

    def step(self, fixed=None):
        self.sync()
        self.search()
        self.forces()
        self.integrate(fixed)


def _exact_gradient(case, ic, dev):
    from torch.utils.checkpoint import checkpoint
    u0 = torch.from_numpy(ic["temp"]).to(dev) * icm.ideal_gas_cv(ic["params"]["mui"], ic["params"]["gamma"])
    u0.requires_grad_(True)
    am = torch.ones((), dtype=torch.float64, device=dev, requires_grad=True)
    dt = ic["params"]["minDt"]
    e = Exact(ic, dev)
    e.dt = e.dt_m1 = dt
    e.f["temp"] = (u0 / e.cv)[e.id]
    names = list(e.f)

    def one(ids, alphamax, *fields):
        s = object.__new__(Exact)
        s.__dict__.update(e.__dict__)
        s.f, s.id, s.alphamax, s.dt, s.dt_m1 = dict(zip(names, fields)), ids, alphamax, dt, dt
        s.step(fixed=dt)
        return (s.id,) + tuple(s.f[k] for k in names)

    ids, fields = e.id, tuple(e.f[k] for k in names)
    for _ in range(case["steps"]):
        ids, *fields = checkpoint(one, ids, am, *fields, use_reentrant=False)
    f = dict(zip(names, fields))
    value = 0.5 * (f["m"] * (f["vx"] ** 2 + f["vy"] ** 2 + f["vz"] ** 2)).sum()
    gu, ga = torch.autograd.grad(value, (u0, am))
    return {"value": float(value), "grad_u0": gu, "grad_alphamax": float(ga)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("order", "block_steps") or _size(case) * (case["steps"] if kind == "gradient" else 1) > \
            (EXACT_MAX * 6 if kind == "gradient" else EXACT_MAX):
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "gradient":
        return _exact_gradient(case, initial(case, seed), dev)
    with torch.no_grad():
        if kind == "ensemble":
            done = []
            for ic in members(case, seed):
                e = Exact(ic, dev)
                for _ in range(case["steps"]):
                    e.step()
                done.append(e.f)
            return {f: torch.cat([d[f] for d in done]) for f in ("x", "y", "z", "vx", "vy", "vz", "temp", "h")}
        ic = initial(case, seed)
        e = Exact(ic, dev, typed=kind in ("host_step", "stages"))
        if kind == "stages":
            e.sync()
            e.search()
            e.forces()
            out = {f: e.more.get(f) for f in DERIVED[1:]}
            out.update(h=e.f["h"], nc=e.nc, xm=e.xm, alpha=e.f["alpha"], du=e.du, kx=e.kx, gradh=e.gradh,
                       courant=e.courant)
            out.update(zip(("ax", "ay", "az"), e.a))
            return out
        for _ in range(case.get("steps", 1)):
            e.step()
        out = dict({f: e.f[f] for f in CONSERVED_FIELDS}, id=e.id)
        if kind == "step":
            out.update(zip(("ax", "ay", "az"), e.a), kx=e.kx, gradh=e.gradh, divv=e.divv)
        return out
