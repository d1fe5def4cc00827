"""Seeding and order-parameter kernels at the sizes where their tiles and
shortcuts end: replica sides around the order parameter's 32-column by 16-row
tasks, many replicas under one block, and point sets whose two nearest points
are closer to each other than FP32 tells apart (the seeding kernel decides
those in double)."""
import numpy as np
import pytest

import oracle
import refmodel

pytestmark = pytest.mark.gpu


def test_order_parameter_tile_edges(engine_lib):
    import gpucpm
    sides = [(3, 3), (31, 16), (32, 17), (33, 15), (65, 3), (3, 49), (64, 32), (100, 200)] * 9
    rng = np.random.default_rng(5)
    b = gpucpm.Batch(2, sides, [9] * len(sides))
    lats = []
    for r, (nx, ny) in enumerate(sides):
        ids = rng.integers(0, 10, (ny, nx))
        lat = (ids | np.where(ids > 0, 1 + ids % 3, 0) << 24).astype(np.uint32)
        lats.append(lat)
        b.lattice(r)[...] = lat.view(np.int32)
    b.push_to_gpu()
    got = b.observe_heterotypic()
    for r, lat in enumerate(lats):
        # the kernel's counts are exact; the ratio is rounded once to FP32
        want = refmodel.heterotypic_fraction(lat)
        assert abs(float(got[r]) - want) <= want * 2.0 ** -24, (r, sides[r])


@pytest.mark.parametrize("shape", [(40, 700), (257, 64), (24, 30, 90)])
@pytest.mark.parametrize("gap", [0.0, 1e-9, 1e-4, 1e-2])
def test_voronoi_near_ties(engine_lib, shape, gap):
    """Points mirrored about lattice columns, one of each pair moved by `gap`."""
    import gpucpm
    nd, nx = len(shape), shape[-1]
    rng = np.random.default_rng(int(gap * 1e9) + nx)
    dims = np.array(shape[::-1], np.float64)
    half = rng.random((80, nd)) * dims
    other = half.copy()
    other[:, 0] = (2.0 * np.floor(rng.random(80) * nx) - half[:, 0] + gap) % nx
    pts = np.concatenate([half, other])
    vals = ((np.arange(160) + 1) | (1 << 24)).astype(np.uint32)
    if nd == 2:
        e = gpucpm.create_box(shape[1], shape[0], 1, 2, 160, 10.0)
    else:
        e = gpucpm.create_box(shape[2], shape[1], shape[0], 3, 160, 10.0)
    e.seed_voronoi(0, pts, vals)
    e.pull_from_gpu()
    np.testing.assert_array_equal(e.lattice(0).view(np.uint32), oracle.voronoi(shape, pts, vals))


@pytest.mark.parametrize("shape", [(3, (1 << 24) + 5), (40, 64), (7, 33), (5, 6, 67)])
@pytest.mark.parametrize("width", [1, 5, 400])
def test_recount_sums_runs_of_sites(engine_lib, shape, width):
    """Tables of cells that are runs of `width` sites in raster order (across
    rows, warps and blocks, medium between them), also where a side is too
    long for 32-bit sums: those of the oracle."""
    import gpucpm
    sites = int(np.prod(shape))
    run = np.arange(sites) // (width if sites < 10**6 else sites // 50 * width // 400 + 1)
    ids = run % 7 * (1 + run // 7 % 40)
    ncells = int(ids.max())
    lat = (ids | np.where(ids > 0, 1 + ids % 3, 0) << 24).astype(np.uint32).reshape(shape)
    dims = shape[::-1] + ((1,) if len(shape) == 2 else ())
    e = gpucpm.create_box(*dims, len(shape), ncells, 5.0)
    e.lattice(0)[...] = lat.view(np.int32)
    e.push_to_gpu()
    e.synchronize()
    sim = oracle.OracleSim(lat, ncells, np.zeros((4, 4), np.float32), [0] * 4, [0] * 4)
    for got, want in zip(e.tables(0), (sim.area, sim.perim, sim.csum)):
        np.testing.assert_array_equal(got, want)
