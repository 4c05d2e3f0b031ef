"""What the mechanics framework is timed on: the work its users have it do, over the sizes of
its own benchmark, tests and growth runs, each through the package's public entry points.

Kinds of case
  biofilm   a biofilm without growth (the benchmark's state: 300 um disk at 100k cells, z up to
            10 um), advanced between two frames: iterate(steps), then the frame's cells.  It runs
            on from where the last pass ended, as a simulation between two writes does.
  colony    a growing 3-D colony somewhere on its way from a founder to 40,000 cells (the array
            sizes are those of the whole run): the restart of a saved state, `steps` iterations
            with growth and division, the frame's cells and the lineage.
  colony2d  the same for the 2-D model (Bogacki-Shampine, the 2-D driver's growth).
  replicates  independent 2-D colonies of uneven size, advanced together.
  verlet    velocity Verlet, frame to frame.
  functions the driver's free functions one by one: getCellNeighbors, then the pair forces.
  device    the pair forces on device buffers that the caller owns (no allocation).

A state that grows is restarted from the same cells in every pass, so a pass costs the same
however often it runs.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "biofilm-abms_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import abm_b200                                             # noqa: E402
from abm_b200 import replicates, stepsize, workloads        # noqa: E402

R, RCELL, E0, ECELL, GAMMA = 0.8, 0.5, 3900.0, 3.9e6, 100.0
METHODS = {"he21": abm_b200.HEUN_EULER, "bs32": abm_b200.BOGACKI_SHAMPINE,
           "rkf45": abm_b200.RUNGE_KUTTA_FEHLBERG, "dp54": abm_b200.DORMAND_PRINCE}
STAGES = {"he21": 2, "bs32": 4, "rkf45": 6, "dp54": 7}
CONTROLLERS = {"reference": abm_b200.CONTROLLER_REFERENCE, "learned": abm_b200.CONTROLLER_LEARNED,
               "pi": abm_b200.CONTROLLER_PI}
LDIV, LDIV_2D = 5.6, replicates.CONFIG0["Ldiv"]
COLONY_CAP = 40000          # cells that a growth run reserves


def listed():
    return [
        # a young colony, a few divisions after the founder: launches and latency are all there is
        dict(name="colony_64", kind="colony", n=64, steps=200, precision="fp64", controller="reference"),
        # the growing colony of everyday size, in the configuration chosen for speed
        dict(name="colony_2k_learned", kind="colony", n=2000, steps=100, precision="mixed", controller="learned"),
        # late in a growth run: most of its wall time is spent at sizes like this one
        dict(name="colony_20k", kind="colony", n=20011, steps=100, precision="fp64", controller="reference"),
        # the headline benchmark in the chosen configuration
        dict(name="biofilm_100k_learned", kind="biofilm", n=100000, steps=200, method="he21", precision="mixed",
             controller="learned", noise=False, friction=False),
        # the largest: the growth run's target size in the reference's own configuration
        dict(name="biofilm_200k", kind="biofilm", n=200000, steps=200, method="he21", precision="fp64",
             controller="reference", noise=False, friction=False),
        # the high-order method with noise, an odd size
        dict(name="biofilm_30k_dp54_noise", kind="biofilm", n=30031, steps=100, method="dp54", precision="fp64",
             controller="reference", noise=True, friction=False),
        # cell-cell friction
        dict(name="biofilm_10k_friction", kind="biofilm", n=10007, steps=100, method="he21", precision="fp64",
             controller="reference", noise=False, friction=True),
        # velocity Verlet
        dict(name="verlet_5k", kind="verlet", n=5003, steps=100),
        # the 2-D model, growing, with adhesion
        dict(name="colony2d_5k", kind="colony2d", n=5000, steps=100, adhesion=True),
        # replicate colonies advanced together
        dict(name="replicates_24", kind="replicates", colonies=24, lo=200, hi=4000, steps=40),
        # a driver that keeps its own loop and calls the functions one by one
        dict(name="functions_50k", kind="functions", n=50021, precision="fp64"),
        # the pair forces inside somebody else's device program
        dict(name="device_forces_20k", kind="device", n=20000, precision="fp64", lanes=8),
    ]


def _size(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n | 1 if rng.random() < 0.5 else n


def draw(rng):
    kind = rng.choice(["colony", "colony", "biofilm", "biofilm", "biofilm", "verlet", "colony2d", "replicates",
                       "functions", "device"])
    if kind == "colony":
        return dict(kind=kind, n=_size(rng, 32, 20000), steps=rng.choice([50, 100]),
                    precision=rng.choice(["fp64", "mixed"]), controller=rng.choice(["reference", "learned", "pi"]))
    if kind == "biofilm":
        friction = rng.random() < 0.2
        return dict(kind=kind, n=_size(rng, 1000, 30000 if friction else 150000), steps=rng.choice([50, 100]),
                    method=rng.choice(["he21", "he21", "bs32", "rkf45", "dp54"]),
                    precision="fp64" if friction else rng.choice(["fp64", "mixed"]),
                    controller="reference" if friction else rng.choice(["reference", "learned", "pi"]),
                    noise=rng.random() < 0.25, friction=friction)
    if kind == "verlet":
        return dict(kind=kind, n=_size(rng, 500, 20000), steps=rng.choice([50, 100]))
    if kind == "colony2d":
        return dict(kind=kind, n=_size(rng, 32, 20000), steps=rng.choice([50, 100]), adhesion=rng.random() < 0.5)
    if kind == "replicates":
        return dict(kind=kind, colonies=rng.randint(4, 24), lo=rng.choice([50, 200, 500]),
                    hi=_size(rng, 1000, 4000), steps=rng.choice([20, 40]))
    if kind == "functions":
        return dict(kind=kind, n=_size(rng, 500, 100000), precision=rng.choice(["fp64", "mixed"]))
    return dict(kind=kind, n=_size(rng, 500, 30000), precision=rng.choice(["fp64", "mixed"]),
                lanes=rng.choice([4, 8, 16]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _cells_3d(n, seed, lmax=5.0, growing=False, friction=False, moving=False):
    """The benchmark's biofilm at n cells: its areal density, most cells touching a neighbour."""
    cells, _ = workloads.biofilm_3d(n=n, seed=seed, disk_radius=300.0 * math.sqrt(n / 1e5) + 4.0, lmax=lmax,
                                    p_contact=0.9)
    rng = np.random.default_rng(seed + 104729)
    if growing:
        cells[:, 16] = rng.normal(1.5, 0.1, n)
    if moving or friction:
        cells[:, 7:10] = rng.normal(0.0, 0.4, (n, 3))
        dn = rng.normal(0.0, 0.4, (n, 3))
        nn = cells[:, 4:7]
        cells[:, 10:13] = dn - (dn * nn).sum(1, keepdims=True) * nn
    if friction:
        cells = np.asfortranarray(np.hstack([cells, rng.uniform(1.0, 8.0, (n, 1))]))
    return cells


def _simulation(cells, seed, controller="reference", **params):
    sim = abm_b200.Simulation(rng_seed=seed & 0x7FFFFFFF, controller=CONTROLLERS[controller], **params)
    if controller == "learned":
        sim.set_stepsize_weights(stepsize.load())
    sim.upload_cells(cells)
    return sim


def _precision(case):
    return abm_b200.PRECISION_MIXED if case.get("precision") == "mixed" else abm_b200.PRECISION_FP64


class Restart:
    """A growing colony: its simulation, the saved state that a pass starts from, and the buffers
    that the frame and the lineage at the end of a pass go to, with room for the divisions."""

    def __init__(self, sim, cells, dt):
        self.sim, self.cells, self.dt = sim, cells, dt
        self.parents = -np.ones(len(cells), dtype=np.int32)
        room = len(cells) + len(cells) // 8 + 64
        self.frame = np.zeros((room, cells.shape[1]), dtype=np.float64, order="F")
        self.lineage = np.zeros(2 * room, dtype=np.int32)

    def load(self):
        self.sim.upload_cells(self.cells)
        self.sim.set_parents(self.parents)
        self.sim.set_clock(0.0, self.dt, 0)
        self.sim.get_cell_neighbors()

    def write(self):
        n = self.sim.num_cells()
        self.sim.download_cells_raw(self.frame.ctypes.data, len(self.frame))
        parents = self.sim.parents()
        self.lineage[:len(parents)] = parents
        return dict(n=n, cells=self.frame, lineage=self.lineage)


def _colony(case, seed):
    cells = _cells_3d(case["n"], seed, lmax=LDIV, growing=True)
    sim = _simulation(cells, seed, case["controller"], precision=_precision(case), cap_cells=COLONY_CAP,
                      Ldiv=LDIV, max_stepsize=1e-4, growth_mean=1.5, growth_std=0.1, daughter_length_std=0.01,
                      daughter_angle_xy_bound=0.05, daughter_angle_z_bound=0.05)
    return dict(sim=sim, restart=Restart(sim, cells, 1e-6), steps=case["steps"])


def _cells_2d(n, seed):
    """A 2-D colony whose lengths reach up to the division length."""
    cells = workloads.biofilm_2d(n, seed=seed, lmin=1.4, lmax=LDIV_2D)
    cells[:, 12] = np.random.default_rng(seed + 7919).normal(1.5, 0.1, n)
    return cells


def _colony2d(case, seed):
    cells = _cells_2d(case["n"], seed)
    params = dict(replicates.CONFIG0)
    if case["adhesion"]:
        params.update(adhesion_mode=1, adhesion_strength=20.0, adhesion_mindist=1.2)
    sim = _simulation(cells, seed, cap_cells=2 * case["n"] + 64, **params)
    return dict(sim=sim, restart=Restart(sim, cells, 1e-6), steps=case["steps"])


def _biofilm(case, seed):
    cells = _cells_3d(case["n"], seed, friction=case["friction"])
    params = dict(cap_cells=case["n"], integration_mode=METHODS[case["method"]], precision=_precision(case),
                  max_stepsize=1e-6)
    if case["noise"]:
        params.update(max_rxy_noise=5.0, max_rz_noise=5.0, max_nxy_noise=2.0, max_nz_noise=2.0)
    if case["friction"]:
        params.update(friction_mode=1, cell_cell_coulomb_coeff=1.0)
    sim = _simulation(cells, seed, case["controller"], **params)
    sim.get_cell_neighbors()
    return dict(sim=sim, steps=case["steps"])


def _verlet(case, seed):
    cells = _cells_3d(case["n"], seed, moving=True)
    sim = _simulation(cells, seed, integration_mode=abm_b200.VELOCITY_VERLET, M0=30.0, L0=2.0, max_stepsize=1e-6,
                      cap_cells=case["n"])
    sim.get_cell_neighbors()
    return dict(sim=sim, steps=case["steps"])


def _replicates(case, seed):
    restarts = []
    for r, n in enumerate(np.geomspace(case["lo"], case["hi"], case["colonies"])):
        cells = _cells_2d(int(n), seed + r)
        sim = _simulation(cells, seed + r, cap_cells=2 * int(n) + 64, **replicates.CONFIG0)
        restarts.append(Restart(sim, cells, 1e-6))
        restarts[-1].load()
    return dict(batch=abm_b200.Batch([r.sim for r in restarts]), restarts=restarts, steps=case["steps"])


def _functions(case, seed):
    cells = _cells_3d(case["n"], seed)
    return dict(sim=_simulation(cells, seed, cap_cells=case["n"], precision=_precision(case)))


def _close_pairs(cells, threshold):
    """Unordered pairs (i > j) whose centrelines come closer than `threshold`, with the plain
    closest-point record of each, in 64 bits on the torch device."""
    dev = torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")
    c = torch.from_numpy(np.ascontiguousarray(cells[:, :22])).to(dev)
    reach = threshold + 2.0 * float(c[:, 14].max())
    order = torch.argsort(c[:, 1])                       # slabs along x bound the candidates
    x = c[order, 1].contiguous()
    end = torch.searchsorted(x, x + reach, right=True)
    pi, pj, step = [], [], 2048
    for a in range(0, len(x), step):
        b = min(a + step, len(x))
        e = int(end[b - 1])
        d = torch.cdist(c[order[a:b], 1:4], c[order[a:e], 1:4], compute_mode="donot_use_mm_for_euclid_dist")
        p, q = torch.nonzero(d < reach, as_tuple=True)
        keep = q > p
        pi.append(order[a + p[keep]])
        pj.append(order[a + q[keep]])
    i, j = torch.cat(pi), torch.cat(pj)
    i, j = torch.maximum(i, j), torch.minimum(i, j)
    d, s, t = _segments(c, i, j)
    near = d.norm(dim=1) < threshold
    return c, i[near], j[near], d[near], s[near], t[near]


def _device(case, seed):
    cells = _cells_3d(case["n"], seed)
    params, _ = abm_b200.make_params(cap_cells=case["n"], precision=_precision(case), pair_lanes=case["lanes"])
    _, i, j, _, _, _ = _close_pairs(cells, params.neighbor_threshold)
    n = case["n"]
    src, dst = torch.cat([i, j]), torch.cat([j, i])
    key = torch.sort(src * n + dst).values
    row_ptr = torch.searchsorted(key, torch.arange(n + 1, device=key.device) * n).to(torch.int32)
    delta, radius = abm_b200.jkr_radius_table(R, RCELL, E0, GAMMA)
    return dict(params=params, n=n, cells=torch.from_numpy(np.ascontiguousarray(cells.T)).cuda(),
                row_ptr=row_ptr.cuda(), col=(key % n).to(torch.int32).cuda(), delta=delta, radius=radius,
                out=torch.zeros(6, n, dtype=torch.float64, device="cuda"))


_PREPARE = dict(colony=_colony, colony2d=_colony2d, biofilm=_biofilm, verlet=_verlet, replicates=_replicates,
                functions=_functions, device=_device)


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    state["kind"] = case["kind"]
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _counts(stats):
    return {k: stats[k] for k in ("iterations", "attempts", "retries", "rebuilds", "divisions", "n_cells", "n_pairs",
                                  "rejected", "cell_steps")}


def run(state):
    kind = state["kind"]
    if kind in ("biofilm", "verlet"):
        stats = state["sim"].iterate(state["steps"])
        return dict(cells=state["sim"].download_cells(), t=stats["t"], dt=stats["dt"], counts=_counts(stats))
    if kind in ("colony", "colony2d"):
        state["restart"].load()
        stats = state["sim"].iterate(state["steps"])
        return dict(state["restart"].write(), t=stats["t"], dt=stats["dt"], counts=_counts(stats))
    if kind == "replicates":
        for r in state["restarts"]:
            r.load()
        state["batch"].iterate(state["steps"])
        state["batch"].synchronize()
        return [dict(frame=r.write()["cells"], n=r.sim.num_cells()) for r in state["restarts"]]
    if kind == "functions":
        m = state["sim"].get_cell_neighbors()
        return dict(pairs=m, forces=state["sim"].cell_cell_forces())
    dp = ctypes.POINTER(ctypes.c_double)
    rc = abm_b200.LIB.abm_cell_cell_forces_noalloc(
        ctypes.byref(state["params"]), state["cells"].data_ptr(), state["n"], state["cells"].shape[0], state["n"],
        state["row_ptr"].data_ptr(), state["col"].data_ptr(), state["col"].numel(),
        state["delta"].ctypes.data_as(dp), state["radius"].ctypes.data_as(dp), len(state["delta"]),
        state["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    if rc:
        raise RuntimeError(abm_b200.LIB.abm_noalloc_last_error().decode())
    return state["out"]


# ---------------------------------------------------------------------------
# the work that a pass cannot do without
# ---------------------------------------------------------------------------
# cells move by far less than a cell per pass, so the pairs are those of the start: measured
# 7.5 pairs within the neighbor threshold and 1.45 touching pairs per cell (2-D: 3 and 1)
def work(case):
    kind = case["kind"]
    if kind == "replicates":
        mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        return _loop_work(case["colonies"] * mean, case["steps"], 4, 3.0, 1.0, 3, 17, 2)
    if kind == "colony2d":
        return _loop_work(case["n"], case["steps"], 4, 3.0, 1.0, 3, 17, 2)
    if kind == "verlet":
        return _loop_work(case["n"], case["steps"], 2, 7.5, 1.45, 2, 22, 1)
    if kind in ("biofilm", "colony"):
        evals = 1 if case["controller"] in ("learned", "pi") else 2
        return _loop_work(case["n"], case["steps"], STAGES[case.get("method", "he21")], 7.5, 1.45, evals, 22,
                          2 if kind == "colony" else 1)
    n = case["n"]
    pairs = 7.5 * n
    if kind == "functions":
        return {"bytes": n * (64 + 48.0), "flops": pairs * 150.0}
    return {"bytes": n * (64 + 48 + 4.0) + 2 * pairs * 4, "flops": pairs * 150.0}


def _loop_work(n, steps, stages, pairs, touching, evals, ncols, copies):
    """Per step each cell's records read and written once (geometry 64, velocities 48, length 8,
    the rest 56 read only) and the neighbor entries read once; a distance per pair (about 100
    operations), a force per touching pair (about 60) and stages x evaluations of the cell's
    velocity (about 150).  The frame goes out once, a restart's cells come in once."""
    per_step = n * (2 * 120 + 56 + 4 * 2 * pairs)
    flops = n * (pairs * 100.0 + touching * 60.0 + stages * evals * 150.0)
    return {"bytes": steps * per_step + copies * 8.0 * ncols * n, "flops": steps * flops}


# ---------------------------------------------------------------------------
# the pair forces in 64 bits
# ---------------------------------------------------------------------------
def _clamp(s, h):
    return torch.minimum(torch.maximum(s, -h), h)


def _segments(c, i, j):
    """Closest points of the centrelines of cells i and j: d from i's point to j's, and the body
    coordinates s on i and t on j."""
    ri, ni, hi = c[i, 1:4], c[i, 4:7], c[i, 14]
    rj, nj, hj = c[j, 1:4], c[j, 4:7], c[j, 14]
    w = rj - ri
    b = (ni * nj).sum(1)
    p, q = (ni * w).sum(1), (nj * w).sum(1)
    s = _clamp((p - b * q) / (1.0 - b * b).clamp_min(1e-12), hi)
    t = _clamp(b * s - q, hj)
    s = _clamp(b * t + p, hi)
    par = torch.nonzero(b.abs() >= 0.9999)[:, 0]
    if len(par):
        s[par], t[par] = _near_parallel(ri[par], ni[par], hi[par], rj[par], nj[par], hj[par])
    return w + t[:, None] * nj - s[:, None] * ni, s, t


def _near_parallel(r1, n1, h1, r2, n2, h2):
    """The model's contact of two nearly parallel cells: where they overlap sideways it lies
    midway, from the two smallest of the four end-to-body distances (distances.hpp:227-337)."""
    def nearest(r, n, h, q):
        return _clamp(((q - r) * n).sum(1), h)

    def at(r, n, x):
        return r + x[:, None] * n

    def gap(a, b):
        return (a - b).norm(dim=1)

    p1, q1, p2, q2 = at(r1, n1, -h1), at(r1, n1, h1), at(r2, n2, -h2), at(r2, n2, h2)
    sp1, sq1 = nearest(r2, n2, h2, p1), nearest(r2, n2, h2, q1)
    sp2, sq2 = nearest(r1, n1, h1, p2), nearest(r1, n1, h1, q2)
    g = torch.stack([gap(at(r2, n2, sp1), p1), gap(at(r2, n2, sq1), q1),
                     gap(at(r1, n1, sp2), p2), gap(at(r1, n1, sq2), q2)], 1)
    rank = torch.argsort(torch.argsort(g, dim=1, stable=True), dim=1)
    low = rank < 2
    end1 = torch.where(low[:, 0], -h1, h1)
    s = (end1 + torch.where(low[:, 2], sp2, sq2)) / 2
    t = nearest(r2, n2, h2, at(r1, n1, s))
    zero = torch.zeros_like(s)
    both, none = low[:, 0] & low[:, 1], ~low[:, 0] & ~low[:, 1]
    s, t = torch.where(both, zero, s), torch.where(both, nearest(r2, n2, h2, r1), t)
    s, t = torch.where(none, nearest(r1, n1, h1, r2), s), torch.where(none, zero, t)
    first = g[:, 0] < g[:, 1]
    clear = sp1 == sq1                                   # no sideways overlap: an end of cell 1
    s = torch.where(clear, torch.where(first, -h1, h1), s)
    t = torch.where(clear, sp1, t)
    return s, t


def _pair_forces(cells):
    """dE/dq of the isotropic JKR adhesion with the fixed radius table and the hard core."""
    c, i, j, d, s, t = _close_pairs(cells, 2 * R)
    dev = c.device
    delta, radius = (torch.from_numpy(x).to(dev) for x in abm_b200.jkr_radius_table(R, RCELL, E0, GAMMA))
    dist = d.norm(dim=1)
    overlap = 2 * R - dist
    top = 2 * (R - RCELL)
    capped = overlap.clamp_max(top)
    k = (torch.searchsorted(delta, capped, right=True) - 1).clamp(0, len(delta) - 2)
    a = (radius[k] * (delta[k + 1] - capped) + radius[k + 1] * (capped - delta[k])) / (delta[k + 1] - delta[k])
    m = 4 * E0 * a ** 3 / (3 * (R / 2)) - 4 * torch.sqrt(math.pi * a ** 3 * GAMMA * E0)
    m = m + (4.0 / 3.0) * ECELL * math.sqrt(RCELL / 2) * (overlap - top).clamp_min(0.0) ** 1.5
    v = (m / dist)[:, None] * d
    out = torch.zeros(len(cells), 6, dtype=torch.float64, device=dev)
    out.index_add_(0, i, torch.cat([v, s[:, None] * v], 1))
    out.index_add_(0, j, -torch.cat([v, t[:, None] * v], 1))
    return out


def exact(case, seed):
    """The pair forces of the two force calls.  A loop has no such value here: its steps are as
    long as its own error estimates make them."""
    if case["kind"] not in ("functions", "device"):
        return None
    f = _pair_forces(_cells_3d(case["n"], seed))
    if case["kind"] == "device":
        return f.T.contiguous()
    return dict(pairs=None, forces=np.asfortranarray(f.cpu().numpy()))
