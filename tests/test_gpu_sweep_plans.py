"""The sweep at the sizes where its plan changes, against the oracle bit for
bit: one, three and four rows of targets drawn side by side, several tasks per
warp, one target per task, lattices one task wide or a few rows high, odd
sides, every tile variant; and targets so large that a constraint's integers
no longer fit FP32."""
import numpy as np
import pytest

import oracle
from gpucpm import workloads as W
from test_gpu_batch import _batch, _batch_state
from test_gpu_parity import assert_same, finish, make_engine
from test_gpu_rowtiles import _terms

pytestmark = pytest.mark.gpu


def _check(w, mcs, variant=0, seed=5):
    e = make_engine(w, seed=seed)
    e.set_variant(variant)
    e.run_mcs(mcs)
    finish(e)
    sim = oracle.OracleSim(w.lattice, w.ncells, **w.oracle_kwargs(), seed=seed).run(mcs)
    assert_same(e, sim)
    assert int(sim.counters[2]) > 0


@pytest.mark.parametrize("variant", [0, 1, 2, 3])
@pytest.mark.parametrize("shape,ncells,mcs", [
    ((3, 5), 2, 40), ((2001, 5), 60, 4), ((5, 2003), 60, 4), ((67, 65), 25, 8),
    ((4, 6, 3), 3, 30), ((3, 7, 70), 20, 8), ((35, 3, 33), 30, 8),
])
def test_narrow_and_odd_shapes(engine_lib, shape, ncells, mcs, variant):
    _check(W.random_small(shape, ncells, seed=40 + ncells, temperature=12.0), mcs, variant)


@pytest.mark.parametrize("shape,mcs", [
    ((570, 1024), 3),        # three rows side by side
    ((1301, 1025), 2),       # four rows, one task per warp, odd sides
    ((4000, 2000), 1),       # 8-row tasks, several per warp
    ((135, 136, 64), 2),     # 3D, three rows
    ((200, 201, 63), 1),     # 3D, four rows, odd
    ((312, 314, 128), 1),    # 3D, 8-row tasks
])
def test_plans_by_size(engine_lib, shape, mcs):
    ncells = int(np.prod(shape)) // (200 if len(shape) == 2 else 800)
    _check(W.random_small(shape, ncells, ntypes=3, seed=len(shape), temperature=10.0), mcs)


@pytest.mark.parametrize("shape", [(40, 50), (16, 14, 18)])
@pytest.mark.parametrize("target", [2**21 - 1, 2**21, -2**21, 2**24 + 1])
def test_targets_beyond_fp32_integers(engine_lib, shape, target):
    w = W.random_small(shape, 20, seed=9, temperature=15.0)
    w.tgt_area = w.tgt_area.copy()
    w.tgt_perim = w.tgt_perim.copy()
    w.lam_area = w.lam_area * np.float32(1e-7)
    w.lam_perim = w.lam_perim * np.float32(1e-7)
    w.tgt_area[1], w.tgt_perim[2] = target, target
    _check(w, 6)


@pytest.mark.parametrize("shape,ncells,terms", [
    ((3, 5), 2, False),        # more blocks than rows
    ((61, 53), 30, True), ((17, 4), 3, False), ((4, 600), 40, True),
    ((31, 32), 12, False), ((33, 67), 20, True),
    ((256, 256), 640, False),  # two targets per lane, all blocks full
    ((375, 371), 900, True),   # rounds of draws beyond the first
    ((600, 100), 2000, False),
])
@pytest.mark.parametrize("runs", [(40,), (1, 1, 25, 13)])
def test_small_lattices_run_in_a_cluster(engine_lib, shape, ncells, terms, runs):
    """Lattices small enough to start in the cluster sweep, and the same ones
    in the grid sweep: lattice, tables and counters of the oracle, over one
    launch and over several (tables go out and come in again), and under a
    graph."""
    import gpucpm
    w = W.random_small(shape, ncells, ntypes=3, seed=70 + ncells, temperature=11.0)
    if terms:
        _terms(w, ncells)
    sim = oracle.OracleSim(w.lattice, w.ncells, **w.oracle_kwargs(), seed=6).run(sum(runs))
    for fill in (None, gpucpm.FILL_PARITY):
        e = make_engine(w, seed=6)
        if fill is not None:
            e.set_fill(fill)
        else:
            # (3 columns are below the cluster sweep's least width)
            assert (e.sweep_config()["grid"] <= 16) or shape[1] < 4
        for i, mcs in enumerate(runs):
            (e.run_graph if i % 2 else e.run_mcs)(mcs)
        finish(e)
        assert_same(e, sim)


@pytest.mark.parametrize("shape,cells,mcs", [
    ((64, 50), 399, 20), ((64, 50), 440, 20),        # rows on both sides of sites / 8
    ((16, 14, 18), 480, 12), ((16, 14, 18), 720, 12),
    ((1301, 1025), 170000, 1),                       # four rows side by side, listed rows
])
@pytest.mark.parametrize("terms", [False, True])
def test_tables_scanned_and_listed(engine_lib, shape, cells, mcs, terms):
    """Few rows are replayed by a scan of the tables, many from lists of the
    changed ones: the oracle's results either way, alone and in a batch of
    two lattices of different sizes."""
    import gpucpm
    w = W.random_small(shape, cells, ntypes=3, seed=33, temperature=14.0)
    if terms:
        _terms(w, 5)
    sim = oracle.OracleSim(w.lattice, w.ncells, **w.oracle_kwargs(), seed=12).run(mcs)
    e = make_engine(w, seed=12)
    e.set_fill(gpucpm.FILL_PARITY)
    e.run_mcs(mcs)
    finish(e)
    assert_same(e, sim)
    if terms or w.lattice.size > 100000:
        return
    v = W.random_small(tuple(s + 3 for s in shape), cells, ntypes=3, seed=34, temperature=14.0)
    b = _batch([w, v], seed=12, stream0=0)
    b.set_dispatch(gpucpm.DISPATCH_GRID)
    b.run_mcs(mcs)
    for r, (x, (lat, a, p, c, cnt)) in enumerate(zip([w, v], _batch_state(b, 2))):
        o = oracle.OracleSim(x.lattice, x.ncells, **x.oracle_kwargs(), seed=12, stream=r).run(mcs)
        np.testing.assert_array_equal(lat.view(np.uint32), o.lattice)
        np.testing.assert_array_equal(a, o.area)
        np.testing.assert_array_equal(p, o.perim)
        np.testing.assert_array_equal(c, o.csum)
        assert cnt["accepted"] == int(o.counters[2])


@pytest.mark.parametrize("ndim", [2, 3])
@pytest.mark.parametrize("variant", [0, 1, 2, 3])
def test_batches_of_many_replicas(engine_lib, ndim, variant):
    """More replicas than a warp searches at once, of sides from a few columns
    to several tasks, in tasks of 2 to 32 rows: each as the oracle has it."""
    import gpucpm
    g = np.random.default_rng(8)
    n = 70 if ndim == 2 else 35
    lo, hi = ((5, 90) if ndim == 2 else (4, 14))
    ws = [W.random_small(tuple(int(k) for k in g.integers(lo, hi, ndim)), 4 + i % 9,
                         seed=200 + i, temperature=5.0 + i % 7) for i in range(n)]
    b = _batch(ws, seed=3, stream0=11)
    b.set_variant(variant)
    b.set_dispatch(gpucpm.DISPATCH_GRID)
    b.run_mcs(4)
    for r, (x, (lat, a, p, c, cnt)) in enumerate(zip(ws, _batch_state(b, n))):
        o = oracle.OracleSim(x.lattice, x.ncells, **x.oracle_kwargs(), seed=3,
                             stream=11 + r).run(4)
        np.testing.assert_array_equal(lat.view(np.uint32), o.lattice)
        np.testing.assert_array_equal(a, o.area)
        np.testing.assert_array_equal(p, o.perim)
        np.testing.assert_array_equal(c, o.csum)
        assert cnt["accepted"] == int(o.counters[2])


def test_scores_of_long_and_short_tasks(engine_lib):
    """Scores over tasks of 8 rows (four side by side) and of 2 (two): the same
    lattices, and sums that differ by their order only (FP32)."""
    import torch

    import gpucpm
    ws = [W.sorting_2d(n=40 + 8 * i, ncells=20 + 5 * i, seed=60 + i) for i in range(4)]
    spec = gpucpm.ScoreSpec.make(((1, 1), (2, 2), (1, 2)), lambda_perim=True)
    res = []
    for variant in (1, 3):
        b = _batch(ws, seed=4, stream0=0)
        b.set_variant(variant)
        b.set_dispatch(gpucpm.DISPATCH_GRID)
        sc = torch.zeros((len(ws), 6, gpucpm.SCORE_MAX), device="cuda")
        torch.cuda.synchronize()
        b.run_scores(6, sc.data_ptr(), 0, 6, spec)
        res.append((_batch_state(b, len(ws)), sc.cpu().numpy()))
    for r in range(len(ws)):
        np.testing.assert_array_equal(res[0][0][r][0], res[1][0][r][0])
    scale = np.abs(res[0][1]).max(axis=(0, 1)) + 1e-6
    assert (np.abs(res[0][1] - res[1][1]) / scale).max() < 1e-4
