"""What an explicit variant does where it does not fit: runs with the act or
persistence term keep variant 0, as they always did."""
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
