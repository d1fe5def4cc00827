"""The work that users of gpucpm have it do, as cases that can be timed.

Every case goes through the public Python API (`gpucpm.Cpm`, `gpucpm.Batch`,
`gpucpm.create_box`, `gpucpm.grad`) with the engine's defaults, as a program
written for the reference's `gpucpm.Cpm` does.  Lattices are the workloads'
own kinds: cells painted as squares (sorting) or a periodic Voronoi tissue.

kinds
  frames    run some Monte Carlo steps (MCS), synchronize, pull the lattice:
            one frame of the reference's example loop
  restart   write the host lattice, push, run, pull: a whole short run from
            the user's arrays and back
  run       a stretch of MCS of one lattice that stays on the device (read
            there, so the program waits for it)
  tables    the same, then the area / perimeter / centroid tables
  batch     a stretch of MCS of many replicas in one launch, then the order
            parameter of each
  gradient  likelihood-ratio forward and backward of an ensemble
  measure   seed a Voronoi tissue, recount, measure the order parameter and
            the boundary lengths
"""
import math
import pathlib
import sys

import numpy as np
import torch

sys.path.insert(0, str(pathlib.Path(__file__).resolve().parent.parent / "gpu-cpm_gb300"))
import gpucpm  # noqa: E402
from gpucpm import grad as G  # noqa: E402
from gpucpm import workloads as W  # noqa: E402


def listed():
    return [
        # the smallest call: a frame of an interactive run of the 200^2
        # two-type sorting recipe (400 cells of 5 x 5), a few MCS and the
        # lattice back on the host; launch and phase latency count
        dict(name="frame_sorting_200", kind="frames", nx=200, ny=200, nz=1, cells=400, mcs=10),
        # the sorting recipe at 256^2 (655 cells) run to completion, 1000 MCS
        dict(name="sorting_256", kind="run", start="squares", nx=256, ny=256, nz=1, cells=655,
             types=2, perim=False, term="none", mcs=1000),
        # a tissue of ordinary size from the user's arrays and back: push,
        # a short run, pull
        dict(name="restart_tissue_1024", kind="restart", nx=1024, ny=1024, nz=1, area=100,
             types=3, fill=1.0, perim=True, term="none", mcs=20),
        # a 2D box of odd sides (no multiple of 4), then its cell tables
        dict(name="tables_2d_1001x777", kind="tables", start="voronoi", nx=1001, ny=777, nz=1,
             area=100, types=3, fill=0.8, perim=True, term="none", mcs=20),
        # the headline 2D tissue: 4096^2, 100 sites a cell, area + perimeter
        dict(name="tissue_4096", kind="run", start="voronoi", nx=4096, ny=4096, nz=1, area=100,
             types=3, fill=1.0, perim=True, term="none", mcs=50),
        # motile cells (the act model) in a 512^2 dish
        dict(name="act_512", kind="run", start="voronoi", nx=512, ny=512, nz=1, area=100,
             types=2, fill=0.7, perim=True, term="act", mcs=50),
        # the headline 3D tissue: 256^3, 500 sites a cell, 26 neighbours
        dict(name="tissue3d_256", kind="run", start="voronoi", nx=256, ny=256, nz=256, area=500,
             types=2, fill=0.8, perim=True, term="none", mcs=20),
        # a 3D box of odd sides with a chemotactic field, then its tables
        dict(name="tables_3d_101x75x61", kind="tables", start="voronoi", nx=101, ny=75, nz=61,
             area=300, types=2, fill=0.6, perim=True, term="chemo", mcs=20),
        # persistent migration in 3D: directions updated every 5 MCS
        dict(name="persist3d_96", kind="run", start="voronoi", nx=96, ny=96, nz=96, area=300,
             types=2, fill=0.6, perim=True, term="persist", mcs=20),
        # a parameter study: 256 ragged replicas, sides log-uniform in
        # [64, 1024], own parameters each, one launch
        dict(name="ensemble_256", kind="batch", replicas=256, lo=64, hi=1024, area=50, mcs=20),
        # a gradient step: 128 replicas of the 256^2 sorting grid
        dict(name="gradient_128x256", kind="gradient", replicas=128, n=256, cells=2600, mcs=100),
        # seeding and analysis of a 2048^2 tissue
        dict(name="measure_2048", kind="measure", nx=2048, ny=2048, nz=1, area=100, types=3,
             fill=0.9),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frames", "restart", "run2", "run2", "run3", "run3", "tables2", "tables3",
                       "batch", "gradient", "measure"])
    term2 = rng.choice(["none", "none", "act", "chemo"])
    term3 = rng.choice(["none", "none", "chemo", "persist"])
    perim = rng.random() < 0.7
    types = rng.randint(1, 4)
    fill = rng.choice([0.6, 0.8, 1.0])
    if kind == "frames":
        n = _log(rng, 64, 512)
        return dict(kind=kind, nx=n, ny=n, nz=1, cells=max(4, n * n // 100),
                    mcs=rng.randint(1, 20))
    if kind in ("restart", "run2", "tables2"):
        nx, ny = _log(rng, 48, 3000), _log(rng, 48, 3000)
        if rng.random() < 0.5:  # square, as the reference's lattices are
            nx = ny = (nx + 3) // 4 * 4
        c = dict(kind={"run2": "run", "tables2": "tables"}.get(kind, kind), nx=nx, ny=ny, nz=1,
                 area=rng.choice([25, 50, 100, 200]), types=types, fill=fill, perim=perim,
                 term=term2, mcs=rng.randint(5, 40))
        if kind != "restart":
            c["start"] = "voronoi"
        return c
    if kind in ("run3", "tables3"):
        n = [_log(rng, 20, 200) for _ in range(3)]
        if rng.random() < 0.5:
            n = [(n[0] + 3) // 4 * 4] * 3
        return dict(kind=kind[:-1], start="voronoi", nx=n[0], ny=n[1], nz=n[2],
                    area=rng.choice([100, 300, 500]), types=types, fill=fill, perim=perim,
                    term=term3, mcs=rng.randint(4, 12))
    if kind == "batch":
        lo = _log(rng, 32, 200)
        return dict(kind=kind, replicas=_log(rng, 8, 150), lo=lo,
                    hi=min(1024, lo * rng.randint(1, 6)), area=rng.choice([25, 50, 100]),
                    mcs=rng.randint(5, 20))
    if kind == "gradient":
        n = _log(rng, 60, 256)
        return dict(kind=kind, replicas=_log(rng, 16, 128), n=n, cells=(n // 5) ** 2 - 1,
                    mcs=rng.randint(20, 100))
    if rng.random() < 0.6:
        nx, ny, nz = _log(rng, 100, 2500), _log(rng, 100, 1600), 1
        area = rng.choice([50, 100, 200])
    else:
        nx, ny, nz = (_log(rng, 24, 120) for _ in range(3))
        area = rng.choice([300, 500])
    return dict(kind="measure", nx=nx, ny=ny, nz=nz, area=area, types=types, fill=fill)


# ---- inputs --------------------------------------------------------------------

def _rng(seed):
    return np.random.Generator(np.random.Philox(int(seed)))


def _ndim(case):
    return 3 if case.get("nz", 1) > 1 else 2


def _shape(case):
    s = (case["nx"], case["ny"], case["nz"])
    return s[:_ndim(case)]


def _engine(case, ncells, temperature, has_act=False, history=1):
    """A Cpm where the lattice is square or cubic, else a box."""
    s = _shape(case)
    if len(set(s)) == 1:
        return gpucpm.Cpm(s[0], len(s), ncells, temperature, False, history, has_act)
    e = gpucpm.create_box(case["nx"], case["ny"], case["nz"], len(s), ncells, temperature)
    if history != 1:
        e.set_history(history)
    return e


def _tissue(case, rng):
    """Points and values (id | type << 24) of a Voronoi tissue: `area` sites a
    region, a fraction `fill` of the regions cells, the others medium."""
    s = _shape(case)
    nreg = max(2, math.prod(s) // case["area"])
    pts = rng.random((nreg, len(s))) * np.array(s, np.float64)
    ncells = max(1, round(nreg * case["fill"]))
    is_cell = rng.permutation(nreg) < ncells
    ids = np.zeros(nreg, np.int64)
    ids[is_cell] = np.arange(1, ncells + 1)
    types = np.where(is_cell, rng.integers(1, case["types"] + 1, nreg), 0)
    return pts, (ids | (types << 24)).astype(np.uint32), ncells


def _params(case, rng):
    """A StaticParams record in the ranges of the tissue workloads."""
    nt, three = case["types"] + 1, _ndim(case) == 3
    J = rng.uniform(*((4.0, 16.0) if three else (2.0, 20.0)), (nt, nt)).astype(np.float32)
    J = np.triu(J) + np.triu(J, 1).T
    p = gpucpm.StaticParams()
    p.temperature = 20.0
    surface = 5.5 * case["area"] ** (2.0 / 3.0) if three else 4.0 * math.sqrt(case["area"])
    for a in range(nt):
        for b in range(nt):
            p.J[a * gpucpm.MAX_TYPES + b] = float(J[a, b])
        if a == 0:
            continue
        p.lambda_area[a], p.target_area[a] = 1.0, case["area"]
        if case["perim"]:
            p.lambda_perimeter[a] = 0.2 if three else 0.5
            p.target_perimeter[a] = int(surface)
    term = case["term"]
    if term == "act":
        p.act_lambda[1], p.act_max[1] = 40.0, 20
    elif term == "chemo":
        p.chemotaxis[1] = 30.0
    elif term == "persist":
        p.persistence_lambda[1], p.persistence_diffusion[1] = 20.0, 0.8
        p.persistence_time[1] = 5
    return p


def _squares(n, cells, rng):
    """Two-type 5 x 5 squares on an n x n lattice: non-overlapping random
    places, or the slots of a grid where they would not fit at random."""
    if cells * 25 <= 0.3 * n * n:
        corners = W.place_squares(n, n, cells, 5, rng)
    else:
        per = n // 5
        cells = min(cells, per * per)
        corners = [(int(k % per) * 5, int(k // per) * 5) for k in rng.permutation(per * per)[:cells]]
    lat = np.zeros((n, n), np.uint32)
    types = rng.permutation(np.repeat([1, 2], [cells // 2, cells - cells // 2]))
    for i, (x, y) in enumerate(corners):
        ys, xs = np.arange(y, y + 5) % n, np.arange(x, x + 5) % n
        lat[ys[:, None], xs[None, :]] = np.uint32((i + 1) | (int(types[i]) << 24))
    return lat, cells


def _sorting(case, seed):
    rng = _rng(seed)
    n = case["nx"]
    lat, cells = _squares(n, case["cells"], rng)
    sim = gpucpm.Cpm(n, 2, cells, 10, False, 1, 0)
    J = W.sorting_J()
    for a in range(3):
        if a:
            sim.set_constraints(cell_type=a, lambda_area=1, target_area=25)
        for b in range(a, 3):
            sim.set_constraints(cell_type=a, other_cell_type=b, adhesion=float(J[a, b]))
    sim.get_state()[...] = lat.view(np.int32)
    sim.set_seed(int(seed) & 0xFFFFFFFF)
    sim.push_to_gpu()
    return sim


def _run_mcs(sim, mcs, inner=None):
    """run() with the reference's argument list where the object has it."""
    inner = inner or mcs
    if isinstance(sim, gpucpm.Cpm):
        sim.run(cell_sync=0, block_sync=0, global_sync=1, threads_per_block=4,
                positions_per_thread=8, positions_per_checkerboard=4,
                updates_per_checkerboard_switch=1, updates_per_barrier=1, iterations=mcs,
                inner_iterations=inner)
    else:
        for _ in range(mcs // inner):
            sim.run_mcs(inner)


RELAX_MCS = 10  # of a seeded tissue, so that a pass meets grown cells


def prepare(case, seed):
    kind, rng = case["kind"], _rng(seed)
    if kind == "frames" or case.get("start") == "squares":
        return dict(case=case, sim=_sorting(case, seed))
    if kind in ("run", "tables", "restart"):
        pts, vals, ncells = _tissue(case, rng)
        term = case["term"]
        sim = _engine(case, ncells, 20, term == "act", 5 if term == "persist" else 1)
        if term == "chemo":
            view = sim.field(0)
            for k in range(_ndim(case)):
                view[k] = rng.uniform(-0.3, 0.3, view.shape[1:]) + (1.0 if k == 0 else 0.0)
            sim.push_to_gpu()  # the field goes along (the lattice follows)
        if isinstance(sim, gpucpm.Cpm) and term == "persist":
            sim.set_constraints(cell_type=1, lambda_persistence=20, persistence_diffusion=0.8,
                                persistence_time=5)
        sim.set_params(None, _params(case, rng))
        sim.set_seed(int(seed) & 0xFFFFFFFF)
        sim.seed_voronoi(0, pts, vals)
        sim.recount()
        _run_mcs(sim, RELAX_MCS, 5)
        sim.synchronize()
        state = dict(case=case, sim=sim)
        if kind == "restart":
            sim.pull_from_gpu()
            state["lattice"] = sim.host_lattice(0).copy()
        return state
    if kind == "batch":
        sides = np.exp(_rng(3).uniform(math.log(case["lo"]), math.log(case["hi"]),
                                       case["replicas"])).round().astype(int)
        cells = [max(1, int(s) * int(s) // case["area"]) for s in sides]
        b = gpucpm.Batch(2, [(int(s), int(s)) for s in sides], cells)
        for r, s in enumerate(sides):
            c = dict(nx=int(s), ny=int(s), nz=1, area=case["area"], types=2, fill=1.0,
                     perim=False, term="none")
            p = _params(c, rng)
            lam = float(rng.uniform(0.5, 2.0))
            p.lambda_area[1] = p.lambda_area[2] = lam
            p.temperature = float(rng.uniform(5.0, 30.0))
            b.set_params(r, p)
            pts = rng.random((cells[r], 2)) * float(s)
            types = rng.integers(1, 3, cells[r])
            b.seed_voronoi(r, pts, ((np.arange(cells[r]) + 1) | (types << 24)).astype(np.uint32))
        b.set_seed(int(seed) & 0xFFFFFFFF)
        b.recount()
        b.run_mcs(RELAX_MCS)
        b.synchronize()
        views = [b.device_lattice(r).reshape(-1) for r in range(len(sides))]
        return dict(case=case, sim=b, views=views)
    if kind == "gradient":
        w = W.sorting_grid(n=case["n"], ncells=case["cells"], seed=int(seed) & 0xFFFFFFFF)
        ens = G.Ensemble([w] * case["replicas"], seed=int(seed) & 0xFFFFFFFF)
        views = [ens.batch.device_lattice(r).reshape(-1) for r in range(case["replicas"])]
        return dict(case=case, ens=ens, theta=ens.theta0(), views=views)
    if kind == "measure":
        pts, vals, ncells = _tissue(case, rng)
        return dict(case=case, sim=_engine(case, ncells, 20), points=pts, values=vals)
    raise ValueError(kind)


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "gradient":
        theta = state["theta"].clone().requires_grad_(True)
        mcs = case["mcs"]
        O = G.LikelihoodRatio.apply(theta, state["ens"], mcs, [mcs // 2, mcs])
        O.mean().backward()
        return dict(order=O.detach(), gradient=theta.grad, lattices=torch.cat(state["views"]))
    sim = state["sim"]
    if kind == "frames":
        _run_mcs(sim, case["mcs"])
        sim.synchronize()
        sim.pull_from_gpu()
        return sim.get_state()
    if kind == "restart":
        sim.host_lattice(0)[...] = state["lattice"]
        sim.tick = 0
        if case["term"] == "act":
            sim.act_lattice(0)[...] = 0
        sim.push_to_gpu()
        _run_mcs(sim, case["mcs"])
        sim.synchronize()
        sim.pull_from_gpu()
        return sim.host_lattice(0)
    if kind == "run":
        _run_mcs(sim, case["mcs"], 5 if case["term"] == "persist" and case["mcs"] % 5 == 0 else None)
        sim.synchronize()  # before the device lattice is read
        out = dict(lattice=sim.device_lattice(0))
        if case["term"] == "persist":
            out["directions"] = sim.persistence_state(0)[0]
        return out
    if kind == "tables":
        _run_mcs(sim, case["mcs"])
        sim.synchronize()
        area, perim, sums = sim.tables(0)
        return dict(lattice=sim.device_lattice(0), area=area, perimeter=perim, sums=sums)
    if kind == "batch":
        sim.run_mcs(case["mcs"])
        order = sim.observe_heterotypic()  # waits for the run
        return dict(lattices=torch.cat(state["views"]), order=order)
    # measure
    sim.seed_voronoi(0, state["points"], state["values"])
    sim.recount()
    out = dict(lattice=sim.device_lattice(0), boundaries=sim.boundary_counts(case["types"] + 1).view(np.int64))
    if _ndim(case) == 2:
        out["order"] = sim.observe_heterotypic()
    return out


# ---- what a pass cannot do without ------------------------------------------------

def work(case):
    """Bytes: the lattice in and out once (4 B a site each way) and what else
    is returned.  Operations per copy attempt: the neighbour comparisons of
    the boundary test (8 or 26) and, for the evaluated ones, a draw and two
    adhesion sums: about 64 in 2D and 128 in 3D."""
    kind = case["kind"]
    if kind == "batch":  # sides log-uniform: mean square side
        lo, hi = case["lo"], case["hi"]
        mean = lo * lo if hi <= lo else (hi * hi - lo * lo) / (2.0 * math.log(hi / lo))
        sites = case["replicas"] * mean
    elif kind == "gradient":
        sites = case["replicas"] * case["n"] ** 2
    else:
        sites = math.prod(_shape(case))
    if kind == "measure":
        return dict(bytes=4.0 * sites, flops=sites * (8 + 20.0))
    per = 128.0 if _ndim(case) == 3 else 64.0
    extra = 32.0 * case["replicas"] * case["mcs"] if kind == "gradient" else 0.0
    return dict(bytes=8.0 * sites + extra, flops=per * sites * case["mcs"])


# ---- the same in 64 bits ------------------------------------------------------------

def exact(case, seed):
    """The order parameter of a seeded 2D tissue from a brute-force Voronoi
    tiling in double.  The other cases' outputs are whole numbers, or (the
    gradient, the directions) the end of a Monte Carlo run."""
    if case["kind"] != "measure" or _ndim(case) == 3:
        return None
    nx, ny = case["nx"], case["ny"]
    pts, vals, _ = _tissue(case, _rng(seed))
    if nx * ny * float(len(pts)) > 3e11:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    P = torch.from_numpy(pts).to(dev)
    V = torch.from_numpy(vals.astype(np.int64)).to(dev)

    def dist2(coords, axis, n):
        d = (coords[:, None] - P[None, :, axis]).abs()
        return torch.minimum(d, n - d) ** 2

    dx = dist2(torch.arange(nx, dtype=torch.float64, device=dev), 0, nx)  # [nx, points]
    lat = torch.empty((ny, nx), dtype=torch.int64, device=dev)
    for y in range(ny):
        dy = dist2(torch.tensor([float(y)], dtype=torch.float64, device=dev), 1, ny)[0]
        near = (dy <= dy.min() + 36.0 * case["area"]).nonzero()[:, 0]  # rows that can hold it
        d = dx[:, near] + dy[near][None, :]
        best = d.min(dim=1)
        far = best.values > 36.0 * case["area"]  # nearest point outside the strip: look at all
        row = V[near[best.indices]]
        if bool(far.any()):
            row[far] = V[(dx[far] + dy[None, :]).argmin(dim=1)]
        lat[y] = row
    pairs = hetero = 0
    for sy, sx in ((0, 1), (1, -1), (1, 0), (1, 1)):
        w = torch.roll(lat, (-sy, -sx), (0, 1))
        both = ((lat & 0xFFFFFF) > 0) & ((w & 0xFFFFFF) > 0) & (lat != w)
        pairs += int(both.sum())
        hetero += int((both & ((lat >> 24) != (w >> 24))).sum())
    order = np.array([hetero / pairs if pairs else 0.0], np.float64)
    return dict(lattice=None, boundaries=None, order=order)
