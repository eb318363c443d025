"""The work this framework is used for, as timed cases: what a program has in hand before a call, the call through the
public entry points, and what the call returns, with the same results from plain FP64 torch beside them.

A case names a kind of use and its sizes:

  state    Context.setPositions + Context.getState: energies and forces of snapshots held on the host
           (rescoring a trajectory, a force-matching data set, a geometry optimiser)
  engine   ix_compute_device_posq: the drop-in inside a GPU engine's step loop.  The engine's mixed-precision posq
           arrays in its own particle order, its int64 force buffer cleared every step, a few steps of a trajectory
  md       Context.runVelocityVerlet of rigid waters
  batch    BatchContext.compute: many small clusters at once
  windows  the context at many values of lambda_sterics at once (free energies), forces left on the device
  served   Server: a burst of MD requests of mixed sizes

The systems are 3-site waters at liquid density with the benchmark's kinds of parameters (two atom types unless
`variants` asks for more).  The library computes in FP32 and hands its results over in FP64 or fixed-point containers;
the programs here keep what they get in single precision, as trajectory files, training sets and single-precision
engines do.  Inputs (positions, velocities) are made from the seed alone; the force field is the same for every seed.
"""
import ctypes
import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "openmm-interax-plugin_b200"))

OH = 0.09572
HOH = math.radians(104.52)
HH = 2.0 * OH * math.sin(HOH / 2.0)
MASS = (15.99943, 1.007947, 1.007947)
WATERS_PER_NM3 = 33.4277
FORCE_FIELD_SEED = 1
DEVICE = "cuda"


def listed():
    return [
        # one small cluster, one call: what a geometry scan or an optimiser of a complex repeats; launches and copies
        dict(name="cluster_state", kind="state", waters=8, periodic=False, frames=1),
        # the smallest periodic box of the benchmark, one call per snapshot
        dict(name="box_648_state", kind="state", waters=216, periodic=True, cutoff=0.9, site_cutoff=0.6, frames=1),
        # two unrelated snapshots of the 24,000-atom box: every call builds the neighbor lists anew
        dict(name="box_24k_snapshots", kind="state", waters=8000, periodic=True, cutoff=1.0, site_cutoff=0.6, frames=2),
        # a force field of many atom types with the options in earnest use: order-2 overlap, switching function,
        # Tang-Toennies damping of the three-body term, an alchemical solute at an intermediate lambda; a ragged size
        dict(name="many_types_state", kind="state", waters=3917, periodic=True, cutoff=1.0, site_cutoff=0.6, frames=1,
             variants=32, overlap=2, switch=0.85, damped=True, solute=30, softcore=0.1, lam=0.4),
        # the benchmark's 24,000-atom box in an engine's step loop, and the 96,000-atom one
        dict(name="engine_24k", kind="engine", waters=8000, periodic=True, cutoff=1.0, site_cutoff=0.6, frames=16),
        dict(name="engine_96k", kind="engine", waters=32000, periodic=True, cutoff=1.0, site_cutoff=0.8, frames=8),
        # molecular dynamics: the benchmark's size, and a small box, whose steps are launches more than arithmetic
        dict(name="md_24k", kind="md", waters=8000, periodic=True, cutoff=1.0, site_cutoff=0.6, steps=100),
        dict(name="md_648", kind="md", waters=216, periodic=True, cutoff=0.9, site_cutoff=0.6, steps=100),
        # clusters of 2..32 waters without cutoffs, all in one evaluation
        dict(name="clusters_1024", kind="batch", clusters=1024, largest=32),
        # 16 lambda windows of a decoupled solute: the whole 96,000-atom box without a soft core (linear in lambda),
        # and a smaller one with a soft core
        dict(name="windows_96k", kind="windows", waters=32000, periodic=True, cutoff=1.0, site_cutoff=0.8, solute=30,
             windows=16),
        dict(name="windows_softcore", kind="windows", waters=4099, periodic=True, cutoff=1.0, site_cutoff=0.6,
             solute=20, softcore=0.1, windows=12),
        # a burst of requests of boxes and clusters, each a few MD steps
        dict(name="served_burst", kind="served", boxes=24, clusters=24, steps=20),
    ]


def _spread(rng, low, high):
    """A whole number between low and high, even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["state", "state", "engine", "md", "batch", "windows", "served"])
    c = dict(kind=kind)
    if kind == "batch":
        return dict(c, clusters=_spread(rng, 16, 1024), largest=rng.randint(4, 32))
    if kind == "served":
        return dict(c, boxes=rng.randint(2, 24), clusters=rng.randint(2, 24), steps=rng.randint(1, 20))
    if kind == "state" and rng.random() < 0.4:
        return dict(c, waters=_spread(rng, 2, 300), periodic=False, frames=rng.randint(1, 2))
    waters = _spread(rng, 216, {"state": 12000, "engine": 32000, "md": 8000, "windows": 16000}[kind])
    edge = (waters / WATERS_PER_NM3) ** (1.0 / 3.0)
    cutoff = round(min(rng.uniform(0.8, 1.1), 0.49 * edge), 3)
    c.update(waters=waters, periodic=True, cutoff=cutoff, site_cutoff=round(rng.uniform(0.5, 0.8), 3))
    if rng.random() < 0.35:
        c["variants"] = rng.choice([4, 9, 40])
    if kind == "state":
        c["frames"] = rng.randint(1, 2)
        if rng.random() < 0.5:
            c["switch"] = round(0.85 * cutoff, 3)
        if rng.random() < 0.35:
            c["overlap"] = 2
        if rng.random() < 0.35:
            c["damped"] = True
        if rng.random() < 0.4:
            c.update(solute=rng.randint(1, 20), lam=round(rng.uniform(0.0, 1.0), 3), softcore=rng.choice([0.0, 0.1]))
    elif kind == "engine":
        c["frames"] = rng.randint(2, 8)
    elif kind == "md":
        c["steps"] = rng.randint(10, 100)
    else:
        c.update(solute=rng.randint(1, 30), windows=rng.randint(2, 16), softcore=rng.choice([0.0, 0.1]))
    return c


# -- the force field and the systems ------------------------------------------------------------------------------

@functools.lru_cache(maxsize=64)
def _model_of(waters, periodic, cutoff, site_cutoff, variants, overlap, switch, damped, solute, softcore):
    """Per-particle and per-site parameters of a system of waters, as arrays."""
    from interaxplugin import workloads
    types = workloads.type_parameters(np.random.default_rng(FORCE_FIELD_SEED))
    rng = np.random.default_rng(777)
    keys = ("m1", "m2", "m3", "alpha", "disp_width", "amplitude", "width", "k", "l")
    rows = np.empty((2, variants, len(keys)))
    for t, name in enumerate("OH"):
        rows[t] = [types[name][k] for k in keys]
        if variants > 1:
            f = 1.0 + 0.01 * rng.uniform(-1.0, 1.0, size=(variants, 4))
            rows[t] *= f[:, [0, 0, 0, 0, 1, 3, 2, 3, 3]]
            rows[t][:, 3] = types[name]["alpha"]
    which = rng.integers(variants, size=waters)
    particles = np.stack([rows[0][which], rows[1][which], rows[1][which]], axis=1).reshape(-1, len(keys))
    omega = rng.uniform(700.0, 1300.0, waters)
    c9 = np.exp(rng.uniform(math.log(1e-7), math.log(1e-5), waters))
    sites = np.stack([(16.0 * c9 / (9.0 * omega)) ** (1.0 / 3.0), omega, rng.uniform(0.02, 0.04, waters)], axis=1)
    alch = np.arange(waters) < solute
    box = (waters / WATERS_PER_NM3) ** (1.0 / 3.0) if periodic else None
    return dict(waters=waters, box=box, particles=particles, sites=sites, alch=alch, cutoff=cutoff,
                site_cutoff=site_cutoff, overlap=overlap, switch=switch, damped=damped, softcore=softcore)


def _model(case):
    periodic = bool(case.get("periodic", False))
    return _model_of(case["waters"], periodic, case.get("cutoff", 1.0) if periodic else None,
                     case.get("site_cutoff", 0.6) if periodic else 100.0, case.get("variants", 1),
                     case.get("overlap", 0), case.get("switch", 0.0), case.get("damped", False), case.get("solute", 0),
                     case.get("softcore", 0.0))


_systems = {}


def _system(model, rigid=False):
    """The System of a model, through the Force API; kept, as a program keeps the System it simulates."""
    kept = _systems.get((id(model), rigid))
    if kept is not None and kept[0] is model:
        return kept[1]
    from interaxplugin import (System, InteraxDispersionForce, InteraxExchangeForce, InteraxShortRangeForce,
                               InteraxThreeBodyForce)
    system = System()
    waters, box = model["waters"], model["box"]
    if box:
        system.setDefaultPeriodicBoxVectors((box, 0, 0), (0, box, 0), (0, 0, box))
    dispersion, exchange, short = InteraxDispersionForce(), InteraxExchangeForce(), InteraxShortRangeForce()
    three = InteraxThreeBodyForce()
    for i, (m1, m2, m3, alpha, dw, amplitude, width, k, l) in enumerate(model["particles"].tolist()):
        alch = bool(model["alch"][i // 3])
        system.addParticle(MASS[i % 3])
        dispersion.addParticle(m1, m2, m3, alpha, dw, alch)
        exchange.addParticle(amplitude, width, alch)
        short.addParticle(k, l, width, alch)
    for group, f in enumerate((dispersion, exchange, short)):
        f.setForceGroup(group)
        f.setNonbondedMethod(f.CutoffPeriodic if box else f.NoCutoff)
        f.setCutoffDistance(model["cutoff"] or 1.0)
        f.setSoftcoreRadius(model["softcore"])
        if model["switch"]:
            f.setUseSwitchingFunction(True)
            f.setSwitchingDistance(model["switch"])
        for w in range(waters):
            for a, b in ((0, 1), (0, 2), (1, 2)):
                f.addExclusion(3 * w + a, 3 * w + b)
        system.addForce(f)
    dispersion.setDampingScale(1.0)
    dispersion.setUseLongRangeCorrection(bool(box))
    exchange.setOverlapMethod(model["overlap"])
    short.setOverlapMethod(model["overlap"])
    for w, (alpha, omega, width) in enumerate(model["sites"].tolist()):
        three.addSite([3 * w], alpha, omega, width, w, bool(model["alch"][w]))
    three.setCutoffDistance(model["site_cutoff"])
    three.setUsesPeriodicBoundaryConditions(bool(box))
    three.setForceGroup(3)
    if model["damped"]:
        three.setDampingMethod(three.TangToennies)
    system.addForce(three)
    if rigid:
        for w in range(waters):
            system.addConstraint(3 * w, 3 * w + 1, OH)
            system.addConstraint(3 * w, 3 * w + 2, OH)
            system.addConstraint(3 * w + 1, 3 * w + 2, HH)
    if len(_systems) >= 64:
        _systems.pop(next(iter(_systems)))
    _systems[(id(model), rigid)] = (model, system)
    return system


# -- configurations -----------------------------------------------------------------------------------------------

def _molecules(centres, rng):
    """Waters at the centres with uniformly random orientations: (3 waters, 3)."""
    frame = np.array([[0.0, 0.0, 0.0], [OH, 0.0, 0.0], [OH * math.cos(HOH), OH * math.sin(HOH), 0.0]])
    w, x, y, z = (lambda q: (q / np.linalg.norm(q, axis=1, keepdims=True)).T)(rng.normal(size=(len(centres), 4)))
    rot = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                    2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                    2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], axis=1).reshape(-1, 3, 3)
    return (centres[:, None, :] + np.einsum("wij,aj->wai", rot, frame)).reshape(-1, 3)


def _water_pairs(oxygen, reach, box, apart=None):
    """Pairs (a < b) of waters whose oxygens are within `reach`, in order; `apart`: waters of different groups are no
    pairs.  Torch tensors."""
    n = len(oxygen)
    first, second = [], []
    rows = max(1, 24_000_000 // n)
    index = torch.arange(n, device=oxygen.device)
    for lo in range(0, n, rows):
        hi = min(n, lo + rows)
        r2 = 0.0
        for k in range(3):
            d = oxygen[None, lo:, k] - oxygen[lo:hi, None, k]
            if box:
                d -= box * torch.round(d / box)
            r2 = r2 + d * d
        near = (r2 < reach * reach) & (index[None, lo:] > index[lo:hi, None])
        if apart is not None:
            near &= apart[None, lo:] == apart[lo:hi, None]
        i, j = torch.nonzero(near, as_tuple=True)
        first.append(i + lo)
        second.append(j + lo)
    return torch.cat(first), torch.cat(second)


def _atom_pairs(a, b):
    """The nine atom pairs of each pair of waters."""
    s = torch.arange(3, device=a.device)
    i = (3 * a[:, None, None] + s[None, :, None]).expand(-1, 3, 3).reshape(-1)
    j = (3 * b[:, None, None] + s[None, None, :]).expand(-1, 3, 3).reshape(-1)
    return i, j


def _relaxed(positions, box, iterations=40, apart=None):
    """The waters moved as wholes until none are in hot contact: capped steepest descent on a plain exponential
    repulsion between the atoms of different waters."""
    x = torch.as_tensor(positions, dtype=torch.float64, device=DEVICE)
    a, b = _water_pairs(x[::3], 0.55, box, apart)
    i, j = _atom_pairs(a, b)
    water = i // 3
    other = j // 3
    for _ in range(iterations):
        d = x[j] - x[i]
        if box:
            d = d - box * torch.round(d / box)
        r = d.norm(dim=1).clamp_min(0.02)
        push = d * (torch.exp((0.19 - r) / 0.03) / r)[:, None]
        force = torch.zeros(len(x) // 3, 3, dtype=torch.float64, device=DEVICE)
        force.index_add_(0, other, push)
        force.index_add_(0, water, -push)
        length = force.norm(dim=1, keepdim=True)
        step = 0.01 * force / length.clamp_min(1.0)
        x = x + step.repeat_interleave(3, dim=0)
    # a fixed grid of 2^-40 nm: the order of the sums above leaves no trace
    return torch.round(x * 2.0 ** 40).mul_(2.0 ** -40).cpu().numpy()


def _box_positions(waters, box, rng):
    side = int(math.ceil(waters ** (1.0 / 3.0) - 1e-9))
    chosen = np.sort(rng.permutation(side ** 3)[:waters])
    centres = np.stack([chosen // (side * side), chosen // side % side, chosen % side], axis=1) + 0.5
    centres = centres * (box / side) + rng.uniform(-0.05, 0.05, size=(waters, 3))
    return _relaxed(_molecules(centres, rng), box)


def _cluster_centres(waters, rng):
    """The sites of a randomly placed lattice at liquid density nearest the origin, jittered."""
    spacing = WATERS_PER_NM3 ** (-1.0 / 3.0)
    half = int(math.ceil((3.0 * waters / (4.0 * math.pi)) ** (1.0 / 3.0))) + 2
    grid = np.stack(np.meshgrid(*[np.arange(-half, half + 1)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    grid = (grid + rng.uniform(-0.5, 0.5, size=3)) * spacing
    keep = np.argsort((grid ** 2).sum(1), kind="stable")[:waters]
    return grid[keep] + rng.uniform(-0.04, 0.04, size=(waters, 3))


def _cluster_positions(sizes, rng):
    """One array per cluster of the given numbers of waters."""
    x = np.concatenate([_molecules(_cluster_centres(w, rng), rng) for w in sizes])
    apart = torch.as_tensor(np.repeat(np.arange(len(sizes)), sizes), device=DEVICE)
    x = _relaxed(x, None, apart=apart)
    return np.split(x, 3 * np.cumsum(sizes)[:-1])


def _velocities(waters, rng):
    """Every water's own thermal velocity at 300 K, its atoms together (nm/ps)."""
    v = rng.normal(size=(waters, 3)) * math.sqrt(0.00831446261815324 * 300.0 / sum(MASS))
    return np.repeat(v - v.mean(0), 3, axis=0)


def _frames(case, seed):
    """The snapshots of a state or engine case: unrelated ones, or steps of 2 fs along a trajectory."""
    model = _model(case)
    rng = np.random.default_rng([seed, 1])
    if case["kind"] == "state":
        if not model["box"]:
            return [_cluster_positions([model["waters"]], rng)[0] for _ in range(case["frames"])]
        return [_box_positions(model["waters"], model["box"], rng) for _ in range(case["frames"])]
    x, v = _box_positions(model["waters"], model["box"], rng), _velocities(model["waters"], rng)
    return [x + 0.002 * k * v for k in range(case["frames"])]


def _slots(case, seed):
    """An engine's particle order: the waters shuffled, each one's atoms together."""
    order = np.random.default_rng([seed, 2]).permutation(case["waters"])
    return (3 * order[:, None] + np.arange(3)).reshape(-1).astype(np.int32)


def _posq(frame, slots):
    """Mixed-precision posq and posqCorrection of a snapshot in the engine's order, and the positions they stand for."""
    x = frame[slots]
    high = np.zeros((len(x), 4), np.float32)
    low = np.zeros((len(x), 4), np.float32)
    high[:, :3] = x
    low[:, :3] = x - high[:, :3].astype(np.float64)
    held = np.empty_like(x)
    held[slots] = high[:, :3].astype(np.float64) + low[:, :3].astype(np.float64)
    return high, low, held


def _cluster_sizes(case):
    """The waters of each cluster of a batch: the same systems for every seed, in other configurations."""
    return np.random.default_rng(3).integers(2, case["largest"] + 1, size=case["clusters"])


BOX_WATERS = (340, 523, 1001, 1700, 2600)
CLUSTER_WATERS = (17, 31, 64, 120, 250)


def _requests(case, seed):
    """(model, positions, velocities, steps) of a burst's requests."""
    rng = np.random.default_rng([seed, 4])
    out = []
    for k in range(case["boxes"]):
        model = _model(dict(waters=BOX_WATERS[k % len(BOX_WATERS)], periodic=True, cutoff=1.0))
        out.append((model, _box_positions(model["waters"], model["box"], rng)))
    sizes = [CLUSTER_WATERS[k % len(CLUSTER_WATERS)] for k in range(case["clusters"])]
    for w, x in zip(sizes, _cluster_positions(sizes, rng)):
        out.append((_model(dict(waters=w)), x))
    order = rng.permutation(len(out))
    return [(out[k][0], out[k][1], _velocities(out[k][0]["waters"], rng), int(rng.integers(1, case["steps"] + 1)))
            for k in order]


# -- the calls ----------------------------------------------------------------------------------------------------

def _lambdas(case):
    return np.linspace(0.0, 1.0, case["windows"])


def prepare(case, seed):
    from interaxplugin import BatchContext, Context, Server, _capi
    kind = case["kind"]
    if kind == "batch":
        sizes = _cluster_sizes(case)
        positions = _cluster_positions(sizes, np.random.default_rng([seed, 1]))
        batch = BatchContext([_system(_model(dict(waters=int(w)))) for w in sizes])
        return dict(kind=kind, batch=batch, positions=np.concatenate(positions))
    if kind == "served":
        requests = [(_system(m, rigid=False), x, v, steps) for m, x, v, steps in _requests(case, seed)]
        return dict(kind=kind, requests=requests, server=Server(budget_bytes=4e9, max_running=64))
    model = _model(case)
    system = _system(model, rigid=kind == "md")
    context = Context(system)
    if case.get("solute"):
        context.setParameter("lambda_sterics", case.get("lam", 1.0))
    state = dict(kind=kind, context=context)
    if kind == "state":
        state["frames"] = _frames(case, seed)
    elif kind == "engine":
        L, handle = _capi.lib(), context._ctx
        n = 3 * case["waters"]
        slots = _slots(case, seed)
        frames = [_posq(f, slots)[:2] for f in _frames(case, seed)]
        state.update(lib=L, handle=handle, n=n, slots=torch.as_tensor(slots, device=DEVICE),
                     box=np.ascontiguousarray(np.eye(3) * model["box"]),
                     stream=torch.cuda.ExternalStream(L.ix_get_stream(handle)),
                     frames=[tuple(torch.as_tensor(a, device=DEVICE) for a in f) for f in frames],
                     posq=torch.zeros(n, 4, device=DEVICE), correction=torch.zeros(n, 4, device=DEVICE),
                     fixed=torch.zeros(3, n, dtype=torch.int64, device=DEVICE),
                     energy=torch.zeros(1, dtype=torch.float64, device=DEVICE),
                     status=torch.zeros(1, dtype=torch.int32, device=DEVICE))
    elif kind == "md":
        rng = np.random.default_rng([seed, 1])
        state.update(positions=_box_positions(model["waters"], model["box"], rng),
                     velocities=_velocities(model["waters"], rng), steps=case["steps"])
    else:
        n = 3 * case["waters"]
        context.setPositions(_box_positions(model["waters"], model["box"], np.random.default_rng([seed, 1])))
        state.update(lib=_capi.lib(), handle=context._ctx, values=_lambdas(case),
                     forces=torch.empty(case["windows"], n, 3, dtype=torch.float64, device=DEVICE))
    return state


def run(state):
    return globals()["_run_" + state["kind"]](state)


def _run_state(state):
    context, out = state["context"], []
    for x in state["frames"]:
        context.setPositions(x)
        s = context.getState()
        out.append((s.getTermEnergies().astype(np.float32), s.getForces().astype(np.float32)))
    return out


def _run_engine(state):
    L, handle, stream = state["lib"], state["handle"], state["stream"]
    posq, correction, fixed, energy = state["posq"], state["correction"], state["fixed"], state["energy"]
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    energies, forces = [], []
    with torch.cuda.stream(stream):
        for high, low in state["frames"]:
            posq.copy_(high)
            correction.copy_(low)
            fixed.zero_()
            energy.zero_()
            rc = L.ix_compute_device_posq(handle, -1, 1, p(posq), p(correction), p(state["slots"]),
                                          ctypes.c_void_p(state["box"].ctypes.data), p(fixed), state["n"], p(energy),
                                          p(state["status"]))
            if rc:
                raise RuntimeError(L.ix_last_error(handle).decode())
            forces.append(fixed.to(torch.float32) * (1.0 / 4294967296.0))
            energies.append(energy.to(torch.float32))
        return torch.cat(energies), torch.stack(forces)


def _run_md(state):
    context = state["context"]
    context.setPositions(state["positions"])
    x, v, energy = context.runVelocityVerlet(state["steps"], 0.001, state["velocities"])
    return x.astype(np.float32), v.astype(np.float32), np.float32(energy)


def _run_batch(state):
    energies, forces = state["batch"].compute(state["positions"])
    return energies.astype(np.float32), np.concatenate(forces).astype(np.float32)


def _run_windows(state):
    values, forces = state["values"], state["forces"]
    energies = np.zeros((len(values), 4))
    rc = state["lib"].ix_compute_windows_device(state["handle"], b"lambda_sterics", len(values),
                                                ctypes.c_void_p(values.ctypes.data),
                                                ctypes.c_void_p(energies.ctypes.data),
                                                ctypes.c_void_p(forces.data_ptr()))
    if rc:
        raise RuntimeError(state["lib"].ix_last_error(state["handle"]).decode())
    return energies.astype(np.float32), forces.to(torch.float32)


def _run_served(state):
    server = state["server"]
    ids = [server.submit(system, x, v, steps=steps, dt=0.001) for system, x, v, steps in state["requests"]]
    results = server.run_all()
    got = [results[k] for k in ids]
    return tuple(np.concatenate([getattr(r, name) for r in got]).astype(np.float32)
                 for name in ("term_energies", "forces", "positions", "velocities"))


# -- what a pass cannot do without --------------------------------------------------------------------------------

def _interactions(waters, cutoff, site_cutoff):
    """(pairs, triples) of a box at liquid density, or of a cluster without cutoffs (None)."""
    if cutoff is None:
        return 4.5 * waters * (waters - 1), waters * (waters - 1) * (waters - 2) / 6.0
    atoms = 4.0 / 3.0 * math.pi * cutoff ** 3 * 3.0 * WATERS_PER_NM3
    near = 4.0 / 3.0 * math.pi * site_cutoff ** 3 * WATERS_PER_NM3
    # of the pairs of sites within the cutoff of one, 15/32 are within it of each other; each triple has three apexes
    return 1.5 * waters * atoms, waters * near * near / 2.0 * (15.0 / 32.0) / 3.0


def work(case):
    """Positions read and forces written once, parameters read once; per evaluation about 150 operations a pair (three
    damped dispersion terms, the overlap, both uses of it and their derivatives) and 120 a triple."""
    kind = case["kind"]
    if kind == "batch":
        each = [_interactions(w, None, None) for w in range(2, case["largest"] + 1)]
        pairs, triples = (case["clusters"] * sum(e[k] for e in each) / len(each) for k in (0, 1))
        particles = case["clusters"] * 1.5 * (2 + case["largest"])
        return dict(bytes=particles * (24.0 + 24.0 + 72.0) + 32.0 * case["clusters"], flops=150 * pairs + 120 * triples)
    if kind == "served":
        evaluations = 1.0 + (1 + case["steps"]) / 2.0
        flops = size = 0.0
        for count, waters, periodic in ((case["boxes"], BOX_WATERS, True), (case["clusters"], CLUSTER_WATERS, False)):
            for k in range(count):
                w = waters[k % len(waters)]
                pairs, triples = _interactions(w, 1.0 if periodic else None, 0.6)
                flops += evaluations * (150 * pairs + 120 * triples)
                size += 3 * w * (5 * 24.0 + 72.0)
        return dict(bytes=size, flops=flops)
    waters = case["waters"]
    pairs, triples = _interactions(waters, case["cutoff"] if case.get("periodic") else None, case.get("site_cutoff"))
    evaluation, n = 150 * pairs + 120 * triples, 3 * waters
    if kind == "state":
        return dict(bytes=case["frames"] * n * 48.0 + n * 72.0, flops=case["frames"] * evaluation)
    if kind == "engine":
        return dict(bytes=case["frames"] * n * (32.0 + 24.0) + n * 72.0, flops=case["frames"] * evaluation)
    if kind == "md":
        return dict(bytes=n * (96.0 + 72.0), flops=case["steps"] * evaluation)
    # the terms are linear in lambda, but for the solute's own pairs with a soft core
    solute = 3.0 * case["solute"] * 2.0 * pairs / n
    soft = case["windows"] * 150 * solute if case.get("softcore") else 0.0
    return dict(bytes=n * (24.0 + 72.0) + case["windows"] * n * 24.0, flops=2 * evaluation + soft)


# -- the same results in 64 bits ----------------------------------------------------------------------------------

def _damping(n, x):
    """Tang and Toennies' f_n(x) = 1 - e^-x sum_{k <= n} x^k/k!, the regularised lower incomplete gamma function, with
    its derivative."""
    f = torch.special.gammainc(torch.full_like(x, n + 1.0), x)
    return f, torch.exp(n * torch.log(x) - x - math.lgamma(n + 1.0))


def _overlap(r, wi, wj, first, order2):
    """8 pi times the overlap of two normalised Slater functions exp(-r/w)/(8 pi w^3), and its r-derivative, without
    the cancellation of the textbook form for nearly equal widths; or its order-2 expansion about the width of the
    pair's first particle where the widths are within 0.01 bohr."""
    a, b = torch.minimum(wi, wj), torch.maximum(wi, wj)
    h, s = b - a, a + b
    ea, slope = torch.exp(-r / a), h / (a * b)
    d = r * slope
    term, p3, p4 = torch.ones_like(d), torch.zeros_like(d), torch.zeros_like(d)
    near = d.clamp(max=6.0)
    for n in range(48):                  # e^z = ... : sums of z^n/(n+3)! and z^n/(n+4)!
        p3 = p3 + term / float(math.factorial(n + 3))
        p4 = p4 + term / float(math.factorial(n + 4))
        term = term * near
    far = d.clamp(min=1.0)
    eb = torch.exp(-r / b)
    g3 = (eb - ea * (1.0 + far + 0.5 * far * far)) / far ** 3
    g4 = (g3 - ea / 6.0) / far
    e3, e4 = torch.where(d < 6.0, ea * p3, g3), torch.where(d < 6.0, ea * p4, g4)
    k1, k2 = h / (a ** 3 * b ** 2 * s ** 2), 4.0 / (a * b * s ** 3)
    c0, c1, c2 = 1.0 / s ** 3, 1.0 / (a * s ** 3), 0.5 / (a * a * b * s * s)
    br, dbr = r * r * (r * k1 - k2), r * (3.0 * r * k1 - 2.0 * k2)
    value = e3 * br + ea * (c0 + r * (c1 + r * c2))
    # d phi3/dz = phi3 - 3 phi4, so d(e_a phi3)/dr = -e3/a + slope (e3 - 3 e4)
    deriv = e3 * dbr + (e3 - 3.0 * e4) * slope * br + ea * (c1 + 2.0 * r * c2) - value / a
    if order2:
        l = torch.where(first, wi, wj)
        t, x = (torch.where(first, wj, wi) - l) / l, r / l
        poly, dpoly = 0.0, 0.0
        for n, c in enumerate(((1 / 64, 1 / 64, 1 / 192), (-3 / 128, -3 / 128, -1 / 192, 1 / 384),
                               (3 / 128, 3 / 128, 1 / 768, -5 / 768, 1 / 1280))):
            poly = poly + t ** n * sum(v * x ** k for k, v in enumerate(c))
            dpoly = dpoly + t ** n * sum(k * v * x ** (k - 1) for k, v in enumerate(c) if k)
        scale = 8.0 * torch.exp(-x) / l ** 3
        close = (wi - wj).abs() < 0.01 * 0.0529177210903
        value = torch.where(close, scale * poly, value)
        deriv = torch.where(close, scale / l * (dpoly - poly), deriv)
    return value, deriv


def _pair_coefficients(p, q):
    """C6, C8, C10 of rows (m1, m2, m3, alpha, ...) by the XDM combination rule."""
    pref = p[:, 3] * q[:, 3] / (p[:, 3] * q[:, 0] + q[:, 3] * p[:, 0])
    return (pref * p[:, 0] * q[:, 0], 1.5 * pref * (p[:, 0] * q[:, 1] + p[:, 1] * q[:, 0]),
            pref * (2.0 * (p[:, 0] * q[:, 2] + p[:, 2] * q[:, 0]) + 4.2 * p[:, 1] * q[:, 1]))


def _dispersion(r, coefficients, rate):
    energy = deriv = 0.0
    for n, c in zip((6, 8, 10), coefficients):
        f, df = _damping(n, rate * r)
        energy = energy - c * f / r ** n
        deriv = deriv - c * (rate * df - n * f / r) / r ** n
    return energy, deriv


def _switch(model, r):
    x = ((r - model["switch"]) / (model["cutoff"] - model["switch"])).clamp(min=0.0)
    s = 1.0 + x ** 3 * (-10.0 + x * (15.0 - 6.0 * x))
    return s, -30.0 * x * x * (1.0 - x) ** 2 / (model["cutoff"] - model["switch"])


def _pair_terms(model, x, groups, lam):
    """Energies per group (3 columns) and forces of the pair terms."""
    box, cutoff = model["box"], model["cutoff"]
    params, alch = (torch.as_tensor(model[k], device=x.device) for k in ("particles", "alch"))
    a, b = _water_pairs(x[::3], cutoff + 0.2 if cutoff else 1e9, box, groups)
    energies = torch.zeros(1 if groups is None else int(groups.max()) + 1, 3, dtype=torch.float64, device=x.device)
    forces = torch.zeros_like(x)
    for lo in range(0, len(a), 100_000):
        i, j = _atom_pairs(a[lo:lo + 100_000], b[lo:lo + 100_000])
        d = x[j] - x[i]
        if box:
            d = d - box * torch.round(d / box)
        r = d.norm(dim=1)
        if cutoff:
            keep = r < cutoff
            i, j, d, r = i[keep], j[keep], d[keep], r[keep]
        p, q = params[i], params[j]
        mixed = alch[i // 3] != alch[j // 3]
        scale = torch.where(mixed, lam, 1.0)
        re = r
        if model["softcore"]:
            re = torch.where(mixed, (r ** 6 + (1.0 - lam) * model["softcore"] ** 6) ** (1.0 / 6.0), r)
        e0, d0 = _dispersion(re, _pair_coefficients(p, q), 2.0 / (p[:, 4] + q[:, 4]))
        value, deriv = _overlap(re, p[:, 6], q[:, 6], i < j, model["overlap"] == 2)
        amplitude = p[:, 5] * q[:, 5] / (8.0 * math.pi)
        norm = (p[:, 6] + q[:, 6]) ** 3
        k, l = 0.5 * (p[:, 7] + q[:, 7]), 0.5 * (p[:, 8] + q[:, 8])
        st = norm * value
        energy = torch.stack([e0, amplitude * value, (k + l * st) * st], dim=1)
        slope = torch.stack([d0, amplitude * deriv, (k + 2.0 * l * st) * norm * deriv], dim=1)
        slope = slope * ((r / re) ** 5)[:, None]
        if model["switch"]:
            s, ds = _switch(model, r)
            slope = slope * s[:, None] + energy * ds[:, None]
            energy = energy * s[:, None]
        energy = energy * scale[:, None]
        f = d * (slope.sum(1) * scale / r)[:, None]
        forces.index_add_(0, i, f)
        forces.index_add_(0, j, -f)
        where = torch.zeros_like(i) if groups is None else groups[i // 3]
        energies.index_add_(0, where, energy)
    return energies, forces


def _tail(model, lam):
    """The long-range correction of the dispersion energy: the tail beyond the cutoff, and what the switching function
    removes inside it, averaged over the pairs of particles (each with itself among them)."""
    rows, inverse, counts = np.unique(np.concatenate(
        [model["particles"][:, :5], np.repeat(model["alch"], 3)[:, None]], axis=1), axis=0, return_inverse=True,
        return_counts=True)
    m = len(rows)
    i, j = np.triu_indices(m)
    weight = np.where(i == j, 0.5 * counts[i] * (counts[i] + 1.0), counts[i].astype(np.float64) * counts[j])
    weight = weight * np.where((rows[i, 5] + rows[j, 5]) > 0, lam, 1.0)
    p, q = torch.as_tensor(rows[i]), torch.as_tensor(rows[j])
    coefficients, rate = _pair_coefficients(p, q), 2.0 / (p[:, 4] + q[:, 4])
    nodes, weights = np.polynomial.legendre.leggauss(48)
    total = torch.zeros(len(i), dtype=torch.float64)
    for u, w in zip(0.5 * (nodes + 1.0), 0.5 * weights):      # r = cutoff / u
        r = torch.full_like(total, model["cutoff"] / u)
        total += w * _dispersion(r, coefficients, rate)[0] * r ** 4 / model["cutoff"]
    if model["switch"]:
        width = model["cutoff"] - model["switch"]
        for u, w in zip(0.5 * (nodes + 1.0), 0.5 * weights):
            r = torch.full_like(total, model["switch"] + u * width)
            total += w * width * _dispersion(r, coefficients, rate)[0] * r * r * (1.0 - _switch(model, r)[0])
    n = len(model["particles"])
    sum_ = float((total * torch.as_tensor(weight)).sum())
    return 2.0 * math.pi * n * n / (0.5 * n * (n + 1.0)) * sum_ / model["box"] ** 3


def _triple_terms(model, x, groups, lam):
    """Energies per group and forces on the waters of the three-body term."""
    box, cutoff = model["box"], model["site_cutoff"]
    sites, alch = (torch.as_tensor(model[k], device=x.device) for k in ("sites", "alch"))
    o = x[::3]
    n = len(o)
    a, b = _water_pairs(o, cutoff, box, groups)
    count = torch.bincount(a, minlength=n)
    start = torch.cumsum(count, 0) - count
    energies = torch.zeros(1 if groups is None else int(groups.max()) + 1, dtype=torch.float64, device=x.device)
    forces = torch.zeros_like(o)

    def away(p, q):
        d = o[q] - o[p]
        return d - box * torch.round(d / box) if box else d

    # the triples by their lowest site: all pairs of its later neighbors, a few million at a time
    pairs = count * (count - 1) // 2
    ends = torch.cumsum(pairs, 0).cpu().numpy()
    lo = 0
    while lo < n:
        done = ends[lo - 1] if lo else 0
        hi = max(lo + 1, int(np.searchsorted(ends, done + 3_000_000)))
        site = torch.repeat_interleave(torch.arange(lo, min(hi, n), device=x.device), pairs[lo:hi])
        k = torch.arange(len(site), device=x.device) + int(done) - (torch.cumsum(pairs, 0) - pairs)[site]
        c = ((1.0 + torch.sqrt(1.0 + 8.0 * k.double())) / 2.0).long()
        c = torch.where(c * (c - 1) // 2 > k, c - 1, c)
        c = torch.where((c + 1) * c // 2 <= k, c + 1, c)
        p, q = b[start[site] + k - c * (c - 1) // 2], b[start[site] + c]
        lo = hi
        u, v = away(site, p), away(site, q)
        w = v - u
        if box:
            w = w - box * torch.round(w / box)
        keep = w.norm(dim=1) < cutoff
        site, p, q, u, v, w = (t[keep] for t in (site, p, q, u, v, w))
        if not len(site):
            continue
        sa, sb, sc = sites[site], sites[p], sites[q]
        wa, wb, wc = sa[:, 1], sb[:, 1], sc[:, 1]
        c9 = 1.5 * sa[:, 0] * sb[:, 0] * sc[:, 0] * wa * wb * wc * (wa + wb + wc) / ((wa + wb) * (wb + wc) * (wc + wa))
        c9 = torch.where(alch[site] | alch[p] | alch[q], lam, 1.0) * c9
        vectors = [t.detach().requires_grad_(True) for t in (u, v, w)]
        u, v, w = vectors
        uu, vv, ww = ((t * t).sum(1) for t in vectors)
        cosines = (u * v).sum(1) * (u * w).sum(1) * (v * w).sum(1)
        product = uu * vv * ww
        energy = c9 * (product ** -1.5 - 3.0 * cosines * product ** -2.5)
        if model["damped"]:
            for t, g, f in ((uu, sa, sb), (vv, sa, sc), (ww, sb, sc)):
                y = 2.0 / (g[:, 2] + f[:, 2]) * torch.sqrt(t)
                energy = energy * (1.0 - torch.exp(-y) * (1.0 + y * (1.0 + y * (0.5 + y / 6.0))))
        du, dv, dw = torch.autograd.grad(energy.sum(), vectors)
        energies.index_add_(0, torch.zeros_like(site) if groups is None else groups[site], energy.detach())
        forces.index_add_(0, site, du + dv)
        forces.index_add_(0, p, dw - du)
        forces.index_add_(0, q, -dv - dw)
    return energies, forces


def _evaluate(model, positions, lam=1.0, groups=None):
    """Term energies (groups x 4) and forces of one configuration; `groups`: the cluster of each water (several systems
    evaluated side by side)."""
    device = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.as_tensor(positions, dtype=torch.float64, device=device)
    pair, forces = _pair_terms(model, x, groups, lam)
    three, site_forces = _triple_terms(model, x, groups, lam)
    forces[::3] += site_forces
    energies = torch.cat([pair, three[:, None]], dim=1)
    if model["box"]:
        energies[:, 0] += _tail(model, lam)
    return energies, forces


def exact(case, seed):
    kind = case["kind"]
    if kind in ("md", "served"):
        return None
    if kind == "batch":
        sizes = _cluster_sizes(case)
        positions = np.concatenate(_cluster_positions(sizes, np.random.default_rng([seed, 1])))
        models = [_model(dict(waters=int(w))) for w in sizes]
        whole = dict(models[0], **{k: np.concatenate([m[k] for m in models]) for k in ("particles", "sites", "alch")})
        groups = torch.as_tensor(np.repeat(np.arange(len(sizes)), sizes),
                                 device="cuda" if torch.cuda.is_available() else "cpu")
        return _evaluate(whole, positions, groups=groups)
    model = _model(case)
    if kind == "windows":
        x = _box_positions(model["waters"], model["box"], np.random.default_rng([seed, 1]))
        got = [_evaluate(model, x, float(v)) for v in (_lambdas(case) if model["softcore"] else (0.0, 1.0))]
        if not model["softcore"]:      # linear in lambda
            (e0, f0), (e1, f1) = got
            return (torch.cat([e0 + v * (e1 - e0) for v in _lambdas(case)]),
                    torch.stack([f0 + v * (f1 - f0) for v in _lambdas(case)]))
        return torch.cat([e for e, _ in got]), torch.stack([f for _, f in got])
    frames = _frames(case, seed)
    if kind == "state":
        return [(e[0], f) for e, f in (_evaluate(model, x, case.get("lam", 1.0)) for x in frames)]
    slots = _slots(case, seed)
    got = [_evaluate(model, _posq(x, slots)[2]) for x in frames]
    order = torch.as_tensor(slots.astype(np.int64), device=got[0][1].device)
    return torch.stack([e.sum() for e, _ in got]), torch.stack([f[order].T for _, f in got])
