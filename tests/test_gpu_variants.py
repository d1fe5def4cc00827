"""What an explicit variant does where it does not fit: runs with the act or
persistence term keep variant 0, as they always did, and fixed rows give way
where warps would be left without tasks."""
import numpy as np
import pytest

from gpucpm import workloads as W
from test_gpu_batch import _batch, _batch_state

pytestmark = pytest.mark.gpu


def _replicas(n, side, ndim=2):
    return [W.random_small((side - i % 5,) * ndim, 12, seed=i, temperature=9.0) for i in range(n)]


def _tile(b):
    c = b.sweep_config()
    return c["tile"], c["warps_per_block"], c["grid"]


@pytest.mark.parametrize("ndim,term", [(2, "act"), (3, "act"), (3, "persist")])
@pytest.mark.parametrize("dispatch", [0, 1])
def test_act_and_persistence_runs_keep_variant_0(engine_lib, ndim, term, dispatch):
    ws = _replicas(20, 60 if ndim == 2 else 24, ndim)
    states, tiles = [], []
    for variant in (0, 2):
        b = _batch(ws, seed=4, stream0=0)
        for r in range(len(ws)):
            if term == "act":
                b.set_act(r, 1, 20, 30.0)
            else:
                b.set_persistence(r, 1, 0, 0.5, 10.0)
        b.set_dispatch(dispatch)
        b.set_variant(variant)
        b.run_mcs(3)
        tiles.append(_tile(b))
        states.append(_batch_state(b, len(ws)))
    assert tiles[0] == tiles[1]
    for x, y in zip(*states):
        np.testing.assert_array_equal(x[0], y[0])


def test_autotuned_variants_of_act_runs_are_used(engine_lib):
    """The tuner's choice for act runs holds for them, a caller's later one
    does not."""
    b = _batch(_replicas(20, 60), seed=4, stream0=0)
    b.set_act(0, 1, 20, 30.0)
    b.run_mcs(2)
    default = _tile(b)
    v, _ = b.autotune(2)
    assert b.sweep_config()["variant"] == v
    b.set_dispatch(0)
    b.set_variant(2)
    assert _tile(b) == default


@pytest.mark.parametrize("dispatch", [0, 1, 2])
@pytest.mark.parametrize("variant", [1, 2, 3])
@pytest.mark.parametrize("n,side,ndim", [(20, 60, 2), (200, 60, 2), (12, 24, 3)])
def test_fixed_rows_leave_no_warps_without_tasks(engine_lib, n, side, ndim, variant, dispatch):
    """Batches of small replicas in variants of fixed rows: no task of more than
    16 rows in grid dispatch, the rows that the size gives in replica dispatch,
    and the results of variant 0."""
    import gpucpm
    ws = _replicas(n, side, ndim)
    states, tiles = [], []
    for v in (0, variant):
        b = _batch(ws, seed=4, stream0=0)
        b.set_dispatch(dispatch)
        b.set_variant(v)
        b.run_mcs(2)
        tiles.append(_tile(b))
        states.append(_batch_state(b, n))
    if dispatch == gpucpm.DISPATCH_REPLICA and variant == 3 and ndim == 3:
        assert tiles[1][0][1] == 1  # 144 rows for 24 warps: one-row tasks are many
    elif dispatch == gpucpm.DISPATCH_REPLICA:
        assert tiles[0] == tiles[1]
    else:
        assert tiles[1][0][1] <= 16
    for x, y in zip(*states):
        for s, t in zip(x[:4], y[:4]):
            np.testing.assert_array_equal(s, t)


def test_fixed_rows_of_large_replicas(engine_lib):
    """Where every warp gets a task the fixed rows hold, in both dispatches."""
    import gpucpm
    for dispatch, variant, rows in ((0, 1, 8), (0, 2, 32), (1, 1, 8), (1, 2, 16), (1, 3, 1)):
        b = gpucpm.Batch(2, [(1600, 1500)] * 8, [100] * 8)
        b.set_dispatch(dispatch)
        b.set_variant(variant)
        assert b.sweep_config()["tile"][1] == rows
