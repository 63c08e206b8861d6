"""The calls whose speed this repository is measured by.

Each case is one use of the engine through its public Python entry points, over the range of
shapes and sizes that its configurations, tests and benchmark name: Monte Carlo runs of every
shape family (one system of a thousand bodies up to one of a million, and a batch of small
replicas), overlap relaxation, single moves, loading and checking a state, and pair
correlations.  Inputs are synthetic lattices whose bodies are displaced inside their lattice
cells (free of overlaps, as a run's state is), made from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from rampack_gb300 import _lib
from rampack_gb300 import correlation as corr
from rampack_gb300 import simulation as sim
from rampack_gb300 import workloads as W
from rampack_gb300.packing import BatchPacking, GpuPacking

PINNED = torch.cuda.is_available()


# ---- the cases ------------------------------------------------------------------------

def listed():
    return [
        # a small equation-of-state run: a thousand hard spheres at constant pressure, one
        # cycle per call as an averaging loop makes them
        dict(name="spheres_1000", family="run", shape="sphere", nx=10, ny=10, nz=10, phi=0.30, tstep=0.1, rstep=0.0,
             scaler="volume", box_step=0.01, pressure=10.0, calls=10, cycles=1, adjust=False, burn=300),
        # a liquid-crystal production run of long rods in a shape-changing box
        dict(name="rods5_64000", family="run", shape="spherocylinder", length=5.0, aspect=6.0, nx=40, ny=40, nz=40,
             phi=0.35, tstep=0.2, rstep=0.2, scaler="delta", box_step=0.005, pressure=1.5, calls=1, cycles=5,
             adjust=False, burn=20),
        # the largest system: a million short rods at high density
        dict(name="rods2_1000000", family="run", shape="spherocylinder", length=2.0, aspect=3.0, nx=100, ny=100, nz=100,
             phi=0.50, tstep=0.2, rstep=0.2, scaler="delta", box_step=0.005, pressure=1.5, calls=1, cycles=5,
             adjust=False, burn=10),
        # bent chains of five spheres while the step sizes adapt (thermalisation)
        dict(name="chains_100000", family="run", shape="chain", beads=5, nx=50, ny=80, nz=25, phi=0.45, tstep=0.2,
             rstep=0.2, scaler="delta", box_step=0.005, pressure=1.5, calls=1, cycles=5, adjust=True, burn=20),
        # bent rods of two spherocylinders, an odd number per side
        dict(name="bentrods_99975", family="run", shape="bentrod", nx=25, ny=43, nz=93, tstep=0.2, rstep=0.2,
             scaler="delta", box_step=0.005, pressure=1.5, calls=1, cycles=5, adjust=False, burn=20),
        # generic convex bodies (rounded boxes)
        dict(name="convex_262144", family="run", shape="convex", nx=64, ny=64, nz=64, tstep=0.2, rstep=0.2,
             scaler="delta", box_step=0.005, pressure=1.5, calls=1, cycles=1, adjust=False, burn=2),
        # a soft (WCA) fluid, translations only, with its total energy at the end
        dict(name="wca_97336", family="run", shape="wca", nx=46, ny=46, nz=46, phi=0.40, tstep=0.2, rstep=0.0,
             scaler="delta", box_step=0.005, pressure=1.5, calls=1, cycles=3, adjust=False, burn=10),
        # overlap relaxation: rods thrown in at random, overlaps counted and driven down
        dict(name="relax_27000", family="relax", shape="spherocylinder", length=2.0, aspect=3.0, nx=30, ny=30, nz=30,
             phi=0.30, tstep=0.2, rstep=0.2, scaler="volume", box_step=0.001, pressure=1.5, calls=1, cycles=2,
             adjust=False, burn=5),
        # many independent state points at once: 32 sphere and 32 rod systems of 500 to 20,000
        dict(name="replicas_64", family="batch", spheres=32, rods=32, lo=500, hi=20000, length=3.0, phi=0.30, tstep=0.2,
             rstep=0.2, box_step=0.005, burn=5, cycles=1),
        # single moves tried and accepted one by one from host code (the serial path)
        dict(name="moves_8000", family="serial", shape="spherocylinder", length=2.0, aspect=3.0, nx=20, ny=20, nz=20,
             phi=0.40, tstep=0.2, rstep=0.2, moves=64),
        # a stored state loaded, checked for overlaps and its nematic order measured
        dict(name="load_1000000", family="load", shape="spherocylinder", length=2.0, aspect=3.0, nx=100, ny=100, nz=100,
             phi=0.50),
        # g(r) of the million-rod state out to eight diameters
        dict(name="gr_1000000", family="corr", shape="spherocylinder", length=2.0, aspect=3.0, nx=100, ny=100, nz=100,
             phi=0.50, max_r=8.0, bins=200, function="density"),
    ]


def _sides(rng, lo, hi, least=7):
    """Three lattice counts, unequal, whose product is about a size spread over [lo, hi] by its
    logarithm; `least` per side keeps the box at least two interaction ranges wide."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    side = n ** (1.0 / 3.0)
    nx = max(least, round(side * rng.uniform(0.8, 1.25)))
    ny = max(least, round(side * rng.uniform(0.8, 1.25)))
    return dict(nx=nx, ny=ny, nz=max(least, int(n / (nx * ny))))


def _cycles(n, budget):
    return max(1, min(10, int(budget / n)))


def draw(rng):
    pick = rng.choice(["sphere", "rod", "rod", "chain", "bentrod", "convex", "wca", "relax", "batch", "serial", "load",
                       "corr"])
    move = dict(tstep=round(rng.uniform(0.05, 0.25), 3), rstep=round(rng.uniform(0.05, 0.25), 3), calls=1,
                adjust=rng.random() < 0.3, pressure=round(rng.uniform(1.0, 10.0), 2))
    move.update(rng.choice([dict(scaler="delta", box_step=0.005), dict(scaler="volume", box_step=0.002),
                            dict(scaler="none", box_step=0.0)]))
    length = round(rng.uniform(1.5, 5.0), 2)
    rod = dict(shape="spherocylinder", length=length, aspect=length + 1.0)
    wide = math.ceil(2 * (length + 1.0)) + 1
    if pick == "sphere":
        s = _sides(rng, 500, 500000)
        n = s["nx"] * s["ny"] * s["nz"]
        c = dict(family="run", shape="sphere", phi=round(rng.uniform(0.15, 0.45), 3), **s, **move, cycles=_cycles(n, 5e6),
                 burn=10)
        c["rstep"] = 0.0
        return c
    if pick == "rod":
        s = _sides(rng, 1000, 800000 if length < 3.0 else 60000, wide)
        n = s["nx"] * s["ny"] * s["nz"]
        return dict(family="run", phi=round(rng.uniform(0.15, 0.45), 3), **rod, **s, **move,
                    cycles=_cycles(n, 4e6 if length < 3.0 else 3e5), burn=10)
    if pick == "chain":
        s = _sides(rng, 1000, 100000, 9)
        n = s["nx"] * s["ny"] * s["nz"]
        return dict(family="run", shape="chain", beads=rng.randint(3, 6), phi=round(rng.uniform(0.2, 0.42), 3), **s, **move,
                    cycles=_cycles(n, 5e5), burn=10)
    if pick == "bentrod":
        s = _sides(rng, 1000, 100000, 9)
        n = s["nx"] * s["ny"] * s["nz"]
        return dict(family="run", shape="bentrod", **s, **move, cycles=_cycles(n, 2.5e5), burn=10)
    if pick == "convex":
        return dict(family="run", shape="convex", **_sides(rng, 1000, 100000), **move, cycles=1, burn=2)
    if pick == "wca":
        s = _sides(rng, 1000, 200000)
        n = s["nx"] * s["ny"] * s["nz"]
        c = dict(family="run", shape="wca", phi=round(rng.uniform(0.2, 0.45), 3), **s, **move, cycles=_cycles(n, 4e5), burn=10)
        c["rstep"] = 0.0
        return c
    if pick == "relax":
        return dict(family="relax", phi=round(rng.uniform(0.15, 0.35), 3), shape="spherocylinder", length=2.0, aspect=3.0,
                    **_sides(rng, 1500, 30000), **move, cycles=2, burn=3)
    if pick == "batch":
        return dict(family="batch", spheres=rng.randint(4, 32), rods=rng.randint(4, 32), lo=500, hi=rng.randint(2000, 20000),
                    length=round(rng.uniform(2.0, 3.5), 2), phi=0.30, tstep=move["tstep"], rstep=move["rstep"],
                    box_step=0.005, burn=3, cycles=1)
    if pick == "serial":
        return dict(family="serial", phi=round(rng.uniform(0.2, 0.45), 3), **rod, **_sides(rng, 1500, 50000, wide),
                    tstep=move["tstep"], rstep=move["rstep"], moves=rng.randint(16, 64))
    if pick == "load":
        return dict(family="load", phi=round(rng.uniform(0.2, 0.5), 3), **rod, **_sides(rng, 1500, 800000, wide))
    return dict(family="corr", phi=round(rng.uniform(0.2, 0.5), 3), **rod, **_sides(rng, 1500, 200000, wide),
                max_r=round(rng.uniform(3.0, 6.0), 2), bins=rng.randint(50, 400), function=rng.choice(["density", "S220"]))


# ---- inputs -----------------------------------------------------------------------------

CONVEX_EXTENT = (1.2, 1.2, 2.2)     # of workloads.ROUNDED_BOX, whose cells are 1.5 x 1.5 x 2.5
BENTROD_CELL, BENTROD_EXTENT = (2.0, 0.62, 0.95), (1.8, 0.5, 0.8)
CHAIN_RADIUS, CHAIN_ANGLE = 0.6 / (2 * math.sin(math.radians(15))), math.radians(30)


def _system(case, rng):
    """(kind, params, positions, orientations, box): the lattice of the case's bodies, each
    displaced at random inside its own lattice cell."""
    counts = (case["nx"], case["ny"], case["nz"])
    shape = case["shape"]
    if shape in ("sphere", "wca"):
        a = (W.sphere_volume(0.5) / case["phi"]) ** (1.0 / 3.0)
        kind, prm, cell, ext, mid = W.SPHERE, np.array([0.5]), np.full(3, a), np.ones(3), np.zeros(3)
    elif shape == "spherocylinder":
        ratio = np.array([1.0, 1.0, case["aspect"]])
        a = (W.spherocylinder_volume(case["length"], 0.5) / case["phi"] / ratio.prod()) ** (1.0 / 3.0)
        kind, prm, cell = W.SPHEROCYLINDER, np.array([case["length"], 0.5]), a * ratio
        ext, mid = np.array([1.0, 1.0, case["length"] + 1.0]), np.zeros(3)
    elif shape == "chain":
        k = case["beads"]
        centres = W.banana_centres(CHAIN_RADIUS, CHAIN_ANGLE * (k - 1), k)
        lo, hi = centres.min(0) - 0.5, centres.max(0) + 0.5
        ext, mid = hi - lo, (lo + hi) / 2
        s = (W.banana_volume(centres, 0.5, CHAIN_ANGLE * (k - 1)) / (case["phi"] * ext.prod())) ** (1.0 / 3.0)
        kind, prm, cell = W.POLYSPHERE, W.polysphere_params(centres, 0.5), ext * s
    elif shape == "bentrod":
        kind, prm = W.POLYSPHEROCYLINDER, W.polyspherocylinder_params(W.BENT_ROD)
        cell, ext, mid = np.array(BENTROD_CELL), np.array(BENTROD_EXTENT), np.zeros(3)
    else:
        kind, prm = W.CONVEX, W.ROUNDED_BOX
        cell, ext, mid = np.array([1.5, 1.5, 2.5]), np.array(CONVEX_EXTENT), np.zeros(3)
    pos = W.lattice(counts, cell)
    side = cell * np.array(counts)
    pos += rng.uniform(-0.45, 0.45, pos.shape) * np.maximum(cell - ext, 0.0) - mid
    pos = np.mod(pos, side)
    pos[pos >= side] = 0.0
    return kind, prm, np.ascontiguousarray(pos), W.aligned_rotations(len(pos)), W.diag_box(*side)


def _random_rotations(n, rng):
    """Uniformly distributed rotation matrices (from unit quaternions), row-major."""
    q = rng.normal(size=(n, 4))
    q /= np.linalg.norm(q, axis=1)[:, None]
    w, x, y, z = q.T
    m = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                  2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                  2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], axis=1)
    return np.ascontiguousarray(m)


def _tilted_rotations(n, angle, rng):
    """Rotations by up to `angle` about random axes."""
    ax = rng.normal(size=(n, 3))
    ax /= np.linalg.norm(ax, axis=1)[:, None]
    th = rng.uniform(-angle, angle, n)
    c, s = np.cos(th), np.sin(th)
    x, y, z = ax.T
    k = 1 - c
    m = np.stack([c + x * x * k, x * y * k - z * s, x * z * k + y * s,
                  y * x * k + z * s, c + y * y * k, y * z * k - x * s,
                  z * x * k - y * s, z * y * k + x * s, c + z * z * k], axis=1)
    return np.ascontiguousarray(m)


def _pinned(*shape):
    return torch.zeros(shape, dtype=torch.float64, pin_memory=PINNED).numpy()


def _copied(a):
    b = _pinned(*a.shape)
    b[...] = a
    return b


def _scaler(case):
    if case["scaler"] == "delta":
        return sim.delta_triclinic(case["box_step"])
    return sim.log_volume(case["box_step"] / 3) if case["scaler"] == "volume" else None


def _loaded(case, rng):
    """A state at rest: displaced bodies, slightly tilted within their cells."""
    kind, prm, pos, _, box = _system(case, rng)
    gap = (box[0] / case["nx"] - 1.0) * 0.1
    return kind, prm, pos, _tilted_rotations(len(pos), max(gap, 0.0) / (case["length"] + 1.0), rng), box


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    family = case["family"]
    if family in ("run", "relax"):
        kind, prm, pos, rot, box = _system(case, rng)
        if family == "relax":
            pos = np.ascontiguousarray(rng.uniform(0.0, 1.0, pos.shape) * box[[0, 4, 8]])
            rot = _random_rotations(len(pos), rng)
        g = GpuPacking(kind, prm, pos, rot, box)
        if case["shape"] == "wca":
            g.set_soft(_lib.SOFT_REPULSIVE_LJ, 1.0, 1.0, False)
        if family == "relax":
            g.set_counting(True)
        s = sim.Simulation(g, case["tstep"], case["rstep"], seed, _scaler(case))
        s.set_conditions(1.0, case["pressure"])
        s.run(case["burn"])
        return dict(case=case, packing=g, sim=s, out=(_pinned(g.n, 3), _pinned(g.n, 9), np.zeros(9)))
    if family == "batch":
        groups = []
        for kind, count, tag in ((W.SPHERE, case["spheres"], 0), (W.SPHEROCYLINDER, case["rods"], 1)):
            # sizes and pressures are the case's, the displacements the seed's
            sizes = np.round(np.exp(np.random.default_rng(1234 + tag).uniform(
                math.log(case["lo"]), math.log(case["hi"]), count))).astype(int)
            systems = []
            for n in sizes:
                k, prm, pos, rot, box = W.replica_lattice(kind, int(n), case["phi"], case["length"])
                pos = pos + rng.uniform(-0.02, 0.02, pos.shape)
                systems.append((np.mod(pos, box[[0, 4, 8]]), rot, box))
            b = BatchPacking(kind, prm, systems)
            total = int(sizes.sum())
            groups.append(dict(batch=b, kind=kind, sizes=sizes.astype(np.float64),
                               pressure=np.exp(np.linspace(0.0, math.log(20.0), count)),
                               boxes=np.array([s[2] for s in systems]),
                               out=(_pinned(total, 3), _pinned(total, 9), np.zeros((count, 9)))))
        state = dict(case=case, groups=groups, rng=np.random.default_rng(seed + 1), seed=seed, k=0)
        for _ in range(case["burn"]):
            _batch_cycle(state)
        return state
    if family == "serial":
        kind, prm, pos, rot, box = _system(case, rng)
        g = GpuPacking(kind, prm, pos, rot, box)
        m = case["moves"]
        return dict(case=case, packing=g, particle=rng.integers(0, g.n, m).tolist(), turn=(rng.random(m) < 0.5).tolist(),
                    shift=rng.uniform(-case["tstep"], case["tstep"], (m, 3)),
                    rotation=_tilted_rotations(m, case["rstep"], rng),
                    out=(_pinned(g.n, 3), _pinned(g.n, 9), np.zeros(9)))
    kind, prm, pos, rot, box = _loaded(case, rng)
    g = GpuPacking(kind, prm, pos, rot, box)
    if family == "load":
        return dict(case=case, packing=g, inputs=(_copied(pos), _copied(rot), box))
    if case["function"] == "density":
        obs = corr.PairDensityCorrelation(corr.RadialEnumerator(), case["max_r"], case["bins"])
    else:
        obs = corr.PairAveragedCorrelation(corr.RadialEnumerator(), corr.S220Correlation(), case["max_r"], case["bins"])
    return dict(case=case, packing=g, observable=obs)


# ---- one pass ---------------------------------------------------------------------------

def _batch_cycle(state):
    """One cycle of every replica: a sweep of particle moves, then a box move each whose
    volume term is tested on the host first."""
    case, rng, k = state["case"], state["rng"], state["k"]
    for g in state["groups"]:
        g["batch"].sweep(case["tstep"], case["rstep"] if g["kind"] == W.SPHEROCYLINDER else 0.0,
                         seed=state["seed"] + g["kind"], counter=k, stats=False)
    for g in state["groups"]:
        b, old = g["batch"], g["boxes"]
        new = old + rng.uniform(-case["box_step"], case["box_step"], size=old.shape)
        v0 = np.abs(np.linalg.det(old.reshape(-1, 3, 3)))
        v1 = np.abs(np.linalg.det(new.reshape(-1, 3, 3)))
        expo = g["sizes"] * np.log(v1 / v0) - g["pressure"] * (v1 - v0)
        propose = (rng.uniform(size=b.R) <= np.exp(np.minimum(expo, 700.0))).astype(np.uint8)
        energy = b.try_scaling(np.where(propose[:, None] == 1, new, old), propose)
        bad = (propose == 1) & (energy > 0)
        b.revert_scaling(bad.astype(np.uint8))
        keep = (propose == 1) & ~bad
        old[keep] = new[keep]
    state["k"] = k + 1


def run(state):
    case = state["case"]
    family = case["family"]
    if family in ("run", "relax"):
        for _ in range(case["calls"]):
            st = state["sim"].run(case["cycles"], adjust_steps=case["adjust"])
        g = state["packing"]
        out = list(g.state(state["out"]))
        out += [int(st[k]) for k in ("cycles", "translations", "accepted_translations", "rotations", "accepted_rotations",
                                     "box_moves", "accepted_box_moves")]
        out += [float(st[k]) for k in ("translation_step", "rotation_step", "box_step")]
        if case["shape"] == "wca":
            out.append(g.total_energy())
        if family == "relax":
            out.append(g.cached_overlaps())
        return out
    if family == "batch":
        for _ in range(case["cycles"]):
            _batch_cycle(state)
        return [list(g["batch"].states(g["out"])) for g in state["groups"]]
    if family == "serial":
        g = state["packing"]
        energies = np.zeros(case["moves"])
        for i, (p, turn) in enumerate(zip(state["particle"], state["turn"])):
            if turn:
                energies[i] = g.try_move(p, _lib.MOVE_ROTATION, rotation=state["rotation"][i])
            else:
                energies[i] = g.try_move(p, _lib.MOVE_TRANSLATION, translation=state["shift"][i])
            if energies[i] <= 0.0:
                g.accept_move()
        return list(g.state(state["out"])) + [energies > 0.0]
    g = state["packing"]
    if family == "load":
        g.upload(*state["inputs"])
        overlaps = g.count_total_overlaps()
        q, p2 = g.nematic_order()
        return dict(overlaps=overlaps, q=q, p2=p2)
    obs = state["observable"]
    obs.clear()
    obs.add_snapshot(g)
    x, y, count = obs.values()
    return dict(x=x, y=y, count=count.astype(np.int64))


# ---- what a pass cannot do without --------------------------------------------------------

def _bodies(case):
    return case["nx"] * case["ny"] * case["nz"]


def _move_flops(case):
    """Arithmetic of one move: the neighbours within the interaction range at the mean density,
    each a distance (8 operations) and, beyond the core, the shape's own test."""
    shape = case["shape"]
    if shape in ("sphere", "wca"):
        near = 8.0 * case["phi"]                       # pairs within one diameter
        return near * (8 if shape == "sphere" else 2 * 20)
    if shape == "spherocylinder":
        length = case["length"]
        near = 4.0 / 3.0 * math.pi * (length + 1.0) ** 3 * case["phi"] / W.spherocylinder_volume(length, 0.5)
        return near * (8 + 60)
    if shape == "chain":
        return 20 * (8 + 8 * case["beads"] ** 2)
    if shape == "bentrod":
        return 20 * (8 + 4 * 60)
    return 20 * (8 + 400)


def work(case):
    family = case["family"]
    if family in ("run", "relax"):
        n, cycles = _bodies(case), case["calls"] * case["cycles"]
        turns = case["rstep"] > 0
        state = 24 + (72 if turns else 0)
        moves = (2 if turns else 1) * n * (2 if family == "relax" else 1)
        # every cycle reads and writes each body's state once; the result is copied out once
        return {"bytes": cycles * 2.0 * n * state + 2.0 * n * 96, "flops": cycles * moves * _move_flops(case)}
    if family == "batch":
        total, flops = 0.0, 0.0
        for shape, count, tag in (("sphere", case["spheres"], 0), ("spherocylinder", case["rods"], 1)):
            sizes = np.exp(np.random.default_rng(1234 + tag).uniform(math.log(case["lo"]), math.log(case["hi"]), count))
            total += float(sizes.sum()) * (2 * (24 + 72 * tag) * case["cycles"] + 2 * 96)
            flops += float(sizes.sum()) * (1 + tag) * case["cycles"] * _move_flops(dict(case, shape=shape))
        return {"bytes": total, "flops": flops}
    if family == "serial":
        near = _move_flops(case)
        return {"bytes": 2.0 * _bodies(case) * 96 + case["moves"] * 200.0 * near / 68, "flops": case["moves"] * near}
    n = _bodies(case)
    if family == "load":
        return {"bytes": 3.0 * n * 96, "flops": n * (_move_flops(case) / 2 + 60)}
    pairs = 0.5 * n * 4.0 / 3.0 * math.pi * case["max_r"] ** 3 * case["phi"] / W.spherocylinder_volume(case["length"], 0.5)
    return {"bytes": n * (24.0 if case["function"] == "density" else 96.0), "flops": pairs * (12 if case["function"] == "density" else 24)}


# ---- the same in 64 bits with plain torch ---------------------------------------------------

def _exact_corr(case, pos, rot, box):
    """Radial pair histogram: slabs along the longest side, every pair of a slab with itself and
    the next ones within reach."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    side = torch.tensor(box[[0, 4, 8]], dtype=torch.float64, device=dev)
    p = torch.tensor(pos, dtype=torch.float64, device=dev)
    ax = torch.tensor(rot.reshape(-1, 3, 3)[:, :, 2].copy(), dtype=torch.float64, device=dev)
    d = int(torch.argmax(side))
    nb, max_r, n = case["bins"], case["max_r"], len(pos)
    slabs = int(float(side[d]) / max_r)
    counts = torch.zeros(nb, dtype=torch.float64, device=dev)
    sums = torch.zeros(nb, dtype=torch.float64, device=dev)
    density = case["function"] == "density"

    def add(a, b, same):
        step = max(1, int(4e7 // max(1, len(b))))
        for i in range(0, len(a), step):
            ia = a[i:i + step]
            d2 = torch.zeros(len(ia), len(b), dtype=torch.float64, device=dev)
            for k in range(3):
                t = p[ia, k][:, None] - p[b, k][None, :]
                t -= side[k] * torch.round(t / side[k])
                d2 += t * t
            keep = d2 < max_r * max_r
            if same:
                keep &= ia[:, None] < b[None, :]
            at = keep.nonzero()
            r = torch.sqrt(d2[at[:, 0], at[:, 1]])
            m = torch.clamp((r / (max_r / nb)).to(torch.int64), max=nb - 1)
            counts.add_(torch.bincount(m, minlength=nb).to(torch.float64))
            if not density:
                c = (ax[ia[at[:, 0]]] * ax[b[at[:, 1]]]).sum(1)
                sums.add_(torch.bincount(m, weights=1.5 * (c * c - 1.0 / 3.0), minlength=nb))

    everything = torch.arange(n, device=dev)
    if slabs < 4:
        add(everything, everything, True)
    else:
        which = torch.clamp((p[:, d] / side[d] * slabs).to(torch.int64), max=slabs - 1)
        members = [everything[which == s] for s in range(slabs)]
        for s in range(slabs):
            add(members[s], members[s], True)
            add(members[s], members[(s + 1) % slabs], False)
    c, s = counts.cpu().numpy(), sums.cpu().numpy()
    x = (np.arange(nb) + 0.5) * (max_r / nb)
    if density:
        edges = np.linspace(0.0, max_r, nb + 1)
        rho = n / float(np.prod(box[[0, 4, 8]]))
        shell = np.diff(4.0 / 3.0 * math.pi * edges ** 3 * rho)
        y = c * (2.0 / shell / n)
    else:
        with np.errstate(invalid="ignore", divide="ignore"):
            y = s / c
    return dict(x=x, y=y, count=None)


def exact(case, seed):
    family = case["family"]
    if family not in ("load", "corr"):
        return None     # a Markov chain's state follows the engine's own random stream
    rng = np.random.default_rng(seed)
    _, _, pos, rot, box = _loaded(case, rng)
    if family == "corr":
        return _exact_corr(case, pos, rot, box)
    a = rot.reshape(-1, 3, 3)[:, :, 2]
    q = 1.5 * (a.T @ a) / len(a) - 0.5 * np.eye(3)
    ev = np.linalg.eigvalsh(q)
    return dict(overlaps=None, q=q, p2=float(ev[np.argmax(np.abs(ev))]))
