"""Performance cases of the droplet step: what a user's program has the package do, at its sizes.

Every case goes through the drop-in classes of ``particle-simulator_b200/dem``
with the physics of the measured configurations (water droplets in oil,
lognormal radii of median 5 um, 2 % volume fraction, E = 3e5 V/m, dt = 1e-4 s).
``listed()`` holds fixed sizes, ``draw(rng)`` others of the same ranges;
``prepare`` makes the inputs and the calculator, ``run`` is one pass,
``work`` the bytes and operations that a pass cannot do without and ``exact``
the same outputs from plain torch in FP64.
"""

from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "particle-simulator_b200"))

EPS0 = 8.85418781762039e-12
EPS_OIL, ETA_OIL, ETA_WATER, FIELD, DT = 2.85, 0.06, 0.001, 3e5, 1e-4
M_CONST = 12 * np.pi * EPS0 * EPS_OIL * FIELD**2
ETA_CONST = 1 / (8 * np.pi * ETA_OIL)
STOKES = 2 * np.pi * ETA_OIL * (2 * ETA_OIL + 3 * ETA_WATER) / (ETA_OIL + ETA_WATER)
VOLUME_FRACTION = 0.02
CORR_L, CORR_FZ, CORR_ETA = 1e-3, 1.1126e-11, 0.065  # a COMSOL-like run of one droplet in a periodic cell


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest calls: a unit-test sized open box, where launches and latency count
        dict(name="direct fp64 500 open", path="direct", n=500, precision="fp64", periodic=False),
        # the reference's plain run (main.py): 2,000 droplets, default precision
        dict(name="direct fp64 2000", path="direct", n=2000, precision="fp64", periodic=True),
        # the drop-in at an odd, larger size
        dict(name="direct fp64 20011", path="direct", n=20011, precision="fp64", periodic=True),
        # mixed precision at the plain run's size
        dict(name="direct mixed 2000", path="direct", n=2000, precision="mixed", periodic=True),
        # mixed precision at the benchmark's size
        dict(name="direct mixed 65536", path="direct", n=65536, precision="mixed", periodic=True),
        # a gradient study: forward and backward through a few steps
        dict(name="adjoint 16384", path="adjoint", n=16384, precision="mixed", periodic=True, steps=4),
        # convection with the periodic-image correction (48^3 grid)
        dict(name="corrected mixed 8192", path="corrected", n=8192, precision="mixed", periodic=True, grid=48),
        # collision detection of the large tree runs
        dict(name="hash 1048576", path="hash", n=1 << 20, periodic=True),
        # main_tree.py: the reference's octree, open box, one droplet per leaf
        dict(name="parity tree 100003 open", path="parity_tree", n=100003, leaf=1, periodic=False, theta=0.5),
        # the large Barnes-Hut step on Morton keys
        dict(name="morton tree 1048576", path="morton_tree", n=1 << 20, leaf=16, periodic=True, theta=0.5),
        # main_multi.py: many uneven boxes stepped together
        dict(name="ensemble 32 boxes", path="ensemble", boxes=32, n_min=1024, n_max=16384, periodic=True),
        # a whole run: detection, forces, convection, update and frames of every step
        dict(name="solver fp64 2000", path="solver", n=2000, precision="fp64", periodic=True, steps=40),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["direct", "direct", "direct", "direct", "adjoint", "corrected", "hash", "parity_tree",
                       "morton_tree", "ensemble", "solver"])
    periodic = rng.random() < 0.7
    c = dict(path=path, periodic=periodic)
    if path == "direct":
        c["precision"] = rng.choice(["fp64", "mixed"])
        c["n"] = _log_int(rng, 200, 24000 if c["precision"] == "fp64" else 65536)
    elif path == "adjoint":
        c.update(n=_log_int(rng, 300, 16384), precision=rng.choice(["fp64", "mixed"]), steps=rng.randint(1, 4))
        if c["n"] > 8192:
            c["precision"] = "mixed"
    elif path == "corrected":
        c.update(n=_log_int(rng, 500, 8192), precision=rng.choice(["fp64", "mixed"]), grid=rng.choice([24, 48]))
    elif path == "hash":
        c["n"] = _log_int(rng, 1000, 1 << 20)
    elif path == "parity_tree":
        c.update(n=_log_int(rng, 2000, 150000), leaf=rng.choice([1, 2, 4, 8, 16]), theta=0.5)
    elif path == "morton_tree":
        c.update(n=_log_int(rng, 5000, 1 << 20), leaf=rng.choice([8, 16, 32]), theta=rng.choice([0.5, 0.7]))
    elif path == "ensemble":
        c.update(boxes=rng.randint(3, 24), n_min=_log_int(rng, 200, 2000), n_max=_log_int(rng, 4000, 16384))
    else:
        c.update(n=_log_int(rng, 300, 4000), precision=rng.choice(["fp64", "mixed"]), steps=rng.randint(10, 40))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _touching(pos, r, L, gap, periodic, rows):
    """Which droplets of ``rows`` (indices) lie within r_i + r_j + gap of a droplet that is not
    in ``rows`` or has a smaller index."""
    n = len(r)
    fresh = torch.zeros(n, dtype=torch.bool, device=pos.device)
    fresh[rows] = True

    def hit(i, j, valid):
        d = pos[j] - pos[i][:, None, :]
        if periodic:
            d = d - L * torch.round(d / L)
        near = (d * d).sum(-1) < (r[i][:, None] + r[j] + gap) ** 2
        return (near & valid & (j != i[:, None]) & (~fresh[j] | (j < i[:, None]))).any(1)

    if n <= 1024:
        return hit(rows, torch.arange(n, device=pos.device).expand(len(rows), n), torch.ones((), dtype=torch.bool,
                                                                                              device=pos.device))
    m = max(1, int(L / (2 * float(r.max()) + max(gap, 0.0))))
    cell = (pos / L * m).long().clamp_(0, m - 1)
    key = (cell[:, 0] * m + cell[:, 1]) * m + cell[:, 2]
    order = torch.argsort(key, stable=True)
    count = torch.bincount(key, minlength=m**3)
    start = torch.cumsum(count, 0) - count
    slots = torch.arange(int(count.max()), device=pos.device)
    bad = torch.zeros(len(rows), dtype=torch.bool, device=pos.device)
    reach = (-1, 0, 1) if m >= 3 else range(m)
    for a in reach:
        for b in reach:
            for c in reach:
                nb = cell[rows] + torch.tensor([a, b, c], device=pos.device)
                inside = torch.ones(len(rows), dtype=torch.bool, device=pos.device)
                if periodic or m < 3:
                    nb = nb % m
                else:
                    inside = ((nb >= 0) & (nb < m)).all(1)
                    nb = nb.clamp(0, m - 1)
                k = (nb[:, 0] * m + nb[:, 1]) * m + nb[:, 2]
                for lo in range(0, len(rows), 1 << 18):
                    s = slice(lo, lo + (1 << 18))
                    valid = (slots[None, :] < count[k[s], None]) & inside[s, None]
                    j = order[(start[k[s], None] + slots).clamp_(max=n - 1)]
                    bad[s] |= hit(rows[s], j, valid)
    return bad


def _droplets(n, seed, periodic, gap=1e-6, uniform=False):
    """Positions (n, 3), radii (n,) and box side: positions uniform in the box, droplets closer
    than ``gap`` to another drawn again."""
    g = torch.Generator("cuda").manual_seed(seed)
    kw = dict(device="cuda", dtype=torch.float64, generator=g)
    if uniform:  # the tree benchmark's radii
        r = 2.5e-6 + 5e-6 * torch.rand(n, **kw)
    else:
        r = (math.log(5e-6) + 0.35 * torch.randn(n, **kw)).exp_().clamp_(1e-6, 30e-6)
    L = float((4.0 / 3.0 * math.pi * (r**3).sum() / VOLUME_FRACTION) ** (1.0 / 3.0))
    pos = L * torch.rand((n, 3), **kw)
    rows = torch.arange(n, device="cuda")
    for _ in range(200):
        rows = rows[_touching(pos, r, L, gap, periodic, rows)]
        if len(rows) == 0:
            break
        pos[rows] = L * torch.rand((len(rows), 3), **kw)
    return pos, r, L


def _moved(n, seed, periodic):
    """Droplets that have moved since they were last found apart: a few in a thousand touch."""
    pos, r, L = _droplets(n, seed, periodic, gap=0.0)
    g = torch.Generator("cuda").manual_seed(seed + 1)
    pos = pos + 3e-7 * (2 * torch.rand(pos.shape, device="cuda", dtype=torch.float64, generator=g) - 1)
    return (pos % L if periodic else pos.clamp(0.0, L)), r, L


def _corr_grids(m):
    """A smooth correction field on an m^3 grid with a z-Stokeslet's parities."""
    c = np.linspace(-CORR_L / 2, CORR_L / 2, m)
    x, y, z = np.meshgrid(c, c, c, indexing="ij")
    k = 2 * np.pi / CORR_L
    u = 1e-9 * np.sin(k * x) * np.sin(k * z) * (1 + 0.3 * np.cos(k * y))
    v = 1e-9 * np.sin(k * y) * np.sin(k * z) * (1 + 0.3 * np.cos(k * x))
    w = 1e-9 * (0.8 + 0.5 * np.cos(k * z) + 0.25 * np.cos(k * x) * np.cos(k * y))
    return u, v, w


def _ensemble_sizes(case, seed):
    rng = np.random.default_rng(1)  # the boxes' sizes belong to the case, their droplets to the seed
    return [int(v) for v in rng.integers(case["n_min"], case["n_max"] + 1, case["boxes"])]


def _boundary(case):
    return "periodic" if case["periodic"] else "open"


def _direct(case, L, **kw):
    from dem.force_calculator import DirectDropletForceCalculator

    return DirectDropletForceCalculator(num_particles=case["n"], eps_oil=EPS_OIL, eta_oil=ETA_OIL,
                                        eta_water=ETA_WATER, E=FIELD, L=L, boundary_mode=_boundary(case),
                                        precision=case["precision"], **kw)


class _NoDisplay:
    stop_simulation = False

    def update_solution(self, solution):
        pass


def prepare(case, seed):
    path, periodic = case["path"], case["periodic"]
    s = dict(case=case)
    if path == "ensemble":
        from dem.ensemble import DropletEnsemble

        boxes = [_droplets(n, 1000 * seed + b, periodic) for b, n in enumerate(_ensemble_sizes(case, seed))]
        s["ens"] = DropletEnsemble([(p.cpu().numpy(), r.cpu().numpy()) for p, r, _ in boxes], [L for *_, L in boxes],
                                   eps_oil=EPS_OIL, eta_oil=ETA_OIL, eta_water=ETA_WATER, E=FIELD,
                                   boundary_mode=_boundary(case))
        return s
    n = case["n"]
    if path == "hash":
        from dem.collision_detector import SpatialHashCollisionDetector

        s["pos"], s["r"], L = _moved(n, seed, periodic)
        s["det"] = SpatialHashCollisionDetector(n, L=L, boundary_mode=_boundary(case))
        s["list"] = torch.empty((n // 8 + 64, 2), dtype=torch.int32, device="cuda")
        return s
    pos, r, L = _droplets(n, seed, periodic, uniform=path == "parity_tree")
    s.update(pos=pos, r=r, L=L)
    if path == "direct":
        s["calc"] = _direct(case, L)
    elif path == "corrected":
        from dem.periodic_correction import COMSOLLatticeCorrection

        s["calc"] = _direct(case, L, correction_grid_resolution=case["grid"])
        s["calc"].load_periodic_correction(
            COMSOLLatticeCorrection.from_grid(*_corr_grids(case["grid"]), L_comsol=CORR_L, Fz_comsol=CORR_FZ,
                                              eta_comsol=CORR_ETA), L_sim=L)
    elif path == "adjoint":
        from dem.adjoint import DirectTrajectory

        s["traj"] = DirectTrajectory(L, case["steps"], DT, precision=case["precision"], eps_oil=EPS_OIL,
                                     eta_oil=ETA_OIL, eta_water=ETA_WATER, boundary_mode=_boundary(case))
        s["E"] = torch.tensor(FIELD, dtype=torch.float64, device="cuda")
    elif path == "parity_tree":
        from dem.octree import TreeDropletForceCalculator

        s["calc"] = TreeDropletForceCalculator(num_particles=n, theta=case["theta"], mpl=case["leaf"],
                                               eps_oil=EPS_OIL, eta_oil=ETA_OIL, eta_water=ETA_WATER, E=FIELD, L=L,
                                               periodic=periodic)
    elif path == "morton_tree":
        from dem.octree import MortonTreeForceCalculator

        s["calc"] = MortonTreeForceCalculator(num_particles=n, theta=case["theta"], mpl=case["leaf"],
                                              eps_oil=EPS_OIL, eta_oil=ETA_OIL, eta_water=ETA_WATER, E=FIELD, L=L,
                                              periodic=periodic)
    elif path == "solver":
        from dem.collision_detector import SpatialHashCollisionDetector

        s["calc"] = _direct(case, L)
        s["det"] = SpatialHashCollisionDetector(n, L=L, boundary_mode=_boundary(case))
        s["host"] = pos.cpu().numpy(), r.cpu().numpy()
    return s


def run(s):
    case = s["case"]
    path = case["path"]
    if path in ("direct", "corrected"):
        return s["calc"].calculate_forces_and_convection(s["pos"], s["r"])
    if path == "adjoint":
        from dem.adjoint.direct_adjoint import mean_squared_z_displacement

        x0, r, E = (t.detach().requires_grad_(True) for t in (s["pos"], s["r"], s["E"]))
        x, D = s["traj"](x0, r, E)
        return (x.detach(), D.detach()) + torch.autograd.grad(mean_squared_z_displacement(D), (x0, r, E))
    if path == "hash":
        found, pairs = s["det"].detect(s["pos"], s["r"])
        s["list"].fill_(-1)[: len(pairs)] = pairs  # the program's own list of this step's pairs
        return found, s["list"]
    if path in ("parity_tree", "morton_tree"):
        return s["calc"].calculate_forces_and_total_velocity(s["pos"], s["r"], STOKES)
    if path == "ensemble":
        s["ens"].step(DT, 1, graph=True)
        return s["ens"].pos, s["ens"].F, s["ens"].V
    from dem.particle_state import DropletState
    from dem.solution import DropletSolution
    from dem.solver import EulerDropletSolver

    pos, r = s["host"]
    solver = EulerDropletSolver(s["calc"], DropletSolution(DropletState(pos.copy(), r.copy(), 0.0)), _NoDisplay(),
                                s["det"], verbose=False)
    solver.solve(DT, (case["steps"] - 0.5) * DT)
    return solver.solution.get_current_positions(), solver.solution.get_trajectories()


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    path = case["path"]
    pair = 33 + 34  # operations of a force and an Oseen term
    if path == "ensemble":
        sizes = _ensemble_sizes(case, 0)
        return {"bytes": 128.0 * sum(sizes), "flops": pair * float(sum(n * (n - 1) for n in sizes))}
    n = case["n"]
    pairs = float(n) * (n - 1)
    if path == "direct":
        return {"bytes": 80.0 * n, "flops": pair * pairs}
    if path == "corrected":
        return {"bytes": 80.0 * n + 24.0 * case["grid"] ** 3, "flops": (pair + 9 * 15 + 18) * pairs}
    if path == "adjoint":  # each step forward, and its VJP (an Oseen pass and 186 operations per pair)
        return {"bytes": 168.0 * n * case["steps"], "flops": case["steps"] * (pair + 36 + 186) * pairs}
    if path == "hash":  # a droplet's own and half the 26 neighbour cells, about 7.5 droplets each
        return {"bytes": 32.0 * n, "flops": 10.0 * 14 * 7.5 * n}
    if path in ("parity_tree", "morton_tree"):  # 27 leaves and 189 nodes per level for each droplet
        levels = max(1.0, math.log(max(2.0, n / case["leaf"]), 8))
        return {"bytes": 80.0 * n, "flops": n * (pair * 27.0 * case["leaf"] + (103 + 90) * 189.0 * levels)}
    return {"bytes": 56.0 * n * case["steps"], "flops": pair * pairs * case["steps"]}


# ---------------------------------------------------------------------------
# the same in plain FP64
# ---------------------------------------------------------------------------
def _rows(n):
    step = max(1, (1 << 23) // n)
    return [(i, min(n, i + step)) for i in range(0, n, step)]


def _separation(a, b, L, periodic):
    d = a[None, :, :] - b[:, None, :]
    if periodic:
        d = torch.where(d.abs() > 0.5 * L, d - torch.sign(d) * L, d)
    return d[..., 0], d[..., 1], d[..., 2]


def _force_rows(x, r, i0, i1, L, periodic, m):
    dx, dy, dz = _separation(x, x[i0:i1], L, periodic)
    r2 = dx * dx + dy * dy + dz * dz
    own = torch.arange(len(r), device=x.device)[None, :] == torch.arange(i0, i1, device=x.device)[:, None]
    keep = (r2.detach().sqrt() > r[None, :] + r[i0:i1, None]) & ~own
    r2 = torch.where(keep, r2, torch.ones_like(r2))
    M = torch.where(keep, m * (r[i0:i1, None] * r[None, :]) ** 3 / (r2.sqrt() * r2**3), torch.zeros_like(r2))
    fxy = M * (4 * dz * dz - dx * dx - dy * dy)
    fz = M * (2 * dz * dz - 3 * dx * dx - 3 * dy * dy)
    return torch.stack([(fxy * dx).sum(1), (fxy * dy).sum(1), (fz * dz).sum(1)], 1)


def _oseen_rows(x, F, i0, i1, L, periodic):
    dx, dy, dz = _separation(x, x[i0:i1], L, periodic)
    r2 = dx * dx + dy * dy + dz * dz
    own = torch.arange(len(x), device=x.device)[None, :] == torch.arange(i0, i1, device=x.device)[:, None]
    inv = torch.where(own, torch.zeros_like(r2), torch.where(own, torch.ones_like(r2), r2).rsqrt())
    s = (dx * F[None, :, 0] + dy * F[None, :, 1] + dz * F[None, :, 2]) * inv**3
    return ETA_CONST * torch.stack([(inv * F[None, :, c] + s * d).sum(1) for c, d in enumerate((dx, dy, dz))], 1)


def _forces(x, r, L, periodic, m=M_CONST):
    return torch.cat([_force_rows(x, r, i0, i1, L, periodic, m) for i0, i1 in _rows(len(r))])


def _convection(x, F, L, periodic):
    return torch.cat([_oseen_rows(x, F, i0, i1, L, periodic) for i0, i1 in _rows(len(x))])


def _correction(x, F, L, periodic, m):
    """The periodic-image correction: three permuted trilinear lookups per pair and the self term."""
    grids = [torch.from_numpy(g).to(x).reshape(-1) for g in _corr_grids(m)]
    inv_dx = (m - 1) / CORR_L
    cL = CORR_L / L
    common = cL * (CORR_ETA / ETA_OIL) / CORR_FZ

    def lookup(cells, a, b, c):
        (ia, ta), (ib, tb), (ic, tc) = cells[a], cells[b], cells[c]
        out = [0.0, 0.0, 0.0]
        for p in (0, 1):
            for q in (0, 1):
                for s in (0, 1):
                    at = ((ia + p) * m + ib + q) * m + ic + s
                    wt = (ta if p else 1 - ta) * (tb if q else 1 - tb) * (tc if s else 1 - tc)
                    out = [o + wt * g[at] for o, g in zip(out, grids)]
        return out

    parts = []
    for i0, i1 in _rows(len(x)):
        d = _separation(-x, -x[i0:i1], L, periodic)  # x_i - x_j
        cells = []
        for comp in d:
            f = ((comp * cL + CORR_L / 2) * inv_dx).clamp(0, m - 1)
            k = f.floor().clamp(max=m - 2)
            cells.append((k.long(), f - k))
        zu, zv, zw = lookup(cells, 0, 1, 2)
        xu, xv, xw = lookup(cells, 2, 1, 0)
        yu, yv, yw = lookup(cells, 0, 2, 1)
        own = torch.arange(len(x), device=x.device)[None, :] == torch.arange(i0, i1, device=x.device)[:, None]
        f = torch.where(own[..., None], torch.zeros((), dtype=x.dtype, device=x.device), common * F[None, :, :])
        parts.append(torch.stack([(gx * f[..., 0] + gy * f[..., 1] + gz * f[..., 2]).sum(1)
                                  for gx, gy, gz in ((xw, yu, zu), (xv, yw, zv), (xu, yv, zw))], 1))
    zero = [(torch.full((), math.floor((m - 1) / 2), device=x.device).long(),
             torch.full((), (m - 1) / 2 - math.floor((m - 1) / 2), device=x.device, dtype=x.dtype))] * 3
    return torch.cat(parts) + common * lookup(zero, 0, 1, 2)[2] * F


def _exact_step(x, r, L, periodic):
    F = _forces(x, r, L, periodic)
    V = _convection(x, F, L, periodic)
    y = x + (F / (STOKES * r[:, None]) + V) * DT
    return (torch.remainder(y, L) if periodic else y), F, V


def _exact_adjoint(case, seed):
    from torch.utils.checkpoint import checkpoint

    n, periodic = case["n"], case["periodic"]
    pos, r, L = _droplets(n, seed, periodic)
    E = torch.tensor(FIELD, dtype=torch.float64, device="cuda")
    x0, r, E = (t.requires_grad_(True) for t in (pos, r, E))
    x, D = x0, torch.zeros_like(x0)
    m = 12 * np.pi * EPS0 * EPS_OIL * E**2

    def rows(f, *a):
        return torch.cat([checkpoint(f, *a[:2], i0, i1, *a[2:], use_reentrant=False) for i0, i1 in _rows(n)])

    for _ in range(case["steps"]):
        F = rows(_force_rows, x, r, L, periodic, m)
        V = rows(_oseen_rows, x, F, L, periodic)
        u = DT * (F / (STOKES * r[:, None]) + V)
        x, D = x + u, D + u
    return (x.detach(), D.detach()) + torch.autograd.grad((D[:, 2] ** 2).mean(), (x0, r, E))


def exact(case, seed):
    path, periodic = case["path"], case["periodic"]
    if path == "adjoint":
        return _exact_adjoint(case, seed)
    if path == "ensemble":
        out = [_exact_step(*_droplets(n, 1000 * seed + b, periodic), periodic)
               for b, n in enumerate(_ensemble_sizes(case, seed))]
        return tuple(torch.cat([o[k] for o in out]).T.contiguous() for k in range(3))
    if path not in ("direct", "corrected", "solver"):
        return None  # whole numbers, or the value that a walk's acceptance rule defines
    x, r, L = _droplets(case["n"], seed, periodic)
    if path == "solver":
        frames = [x]
        for _ in range(case["steps"]):
            x = _exact_step(x, r, L, periodic)[0]
            frames.append(x)
        return x, torch.stack(frames)
    F = _forces(x, r, L, periodic)
    V = _convection(x, F, L, periodic)
    if path == "corrected":
        V = V + _correction(x, F, L, periodic, case["grid"])
    return F, V
