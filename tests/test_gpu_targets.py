"""Target areas and perimeters at the ends of 32 bits, where the difference of a
table entry and its target needs more: every sweep has the oracle's results, so
that none depends on the kernel that runs."""
import numpy as np
import pytest

import oracle
from gpucpm import workloads as W
from test_gpu_batch import _batch, _batch_state
from test_gpu_parity import assert_same, finish, make_engine

pytestmark = pytest.mark.gpu

TARGETS = [2**31 - 1, -2**31, -2**31 + 40]


def _far(shape, target, seed=9):
    w = W.random_small(shape, 20, seed=seed, temperature=15.0)
    w.tgt_area = w.tgt_area.copy()
    w.tgt_perim = w.tgt_perim.copy()
    # energies of the order of the temperature
    w.lam_area = w.lam_area * np.float32(3e-9)
    w.lam_perim = w.lam_perim * np.float32(1e-9)
    w.tgt_area[1], w.tgt_perim[2] = target, target
    return w


@pytest.mark.parametrize("target", TARGETS)
@pytest.mark.parametrize("shape,fill,act", [
    ((40, 50), "cluster", False), ((40, 50), "parity", False), ((40, 50), "parity", True),
    ((16, 14, 18), "parity", False), ((16, 14, 18), "parity", True),
])
def test_targets_at_the_ends_of_32_bits(engine_lib, shape, fill, act, target):
    import gpucpm
    w = _far(shape, target)
    if act:
        w.act_lambda = np.array([0, 10, 0], np.float32)
        w.act_max = np.array([0, 20, 0], np.int32)
    e = make_engine(w, seed=5)
    e.set_fill({"cluster": gpucpm.FILL_CLUSTER, "parity": gpucpm.FILL_PARITY}[fill])
    e.run_mcs(6)
    finish(e)
    sim = oracle.OracleSim(w.lattice, w.ncells, **w.oracle_kwargs(), seed=5).run(6)
    assert_same(e, sim)
    assert int(sim.counters[2]) > 0


@pytest.mark.parametrize("target", TARGETS)
def test_targets_in_batches_and_scores(engine_lib, target):
    import torch

    import gpucpm
    ws = [_far((40, 50), target, seed=9), _far((33, 35), target, seed=10)]
    pairs = ((1, 1), (2, 2), (1, 2))
    b = _batch(ws, seed=21, stream0=5)
    b.set_dispatch(gpucpm.DISPATCH_GRID)
    mcs = 6
    sc = torch.zeros((2, mcs, gpucpm.SCORE_MAX), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    b.run_scores(mcs, sc.data_ptr(), 0, mcs,
                 gpucpm.ScoreSpec.make(pairs, lambda_perim=True))
    b.run_mcs(3)
    state = _batch_state(b, 2)
    for r, w in enumerate(ws):
        sim = oracle.OracleSim(w.lattice, w.ncells, **w.oracle_kwargs(), seed=21, stream=5 + r)
        want = sim.run_scores(mcs, oracle.ScoreSpec.make(pairs, lambda_perim=True))
        sim.run(3)
        np.testing.assert_array_equal(state[r][0].view(np.uint32), sim.lattice)
        # FP32 terms and sums against FP64, relative to the parameter's largest
        # score, as for ordinary targets
        scale = np.abs(want).max(axis=0) + 1e-6
        assert (np.abs(sc[r].cpu().numpy() - want) / scale).max() < 2e-3
