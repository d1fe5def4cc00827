"""Batches of even and odd sides under replica and hybrid dispatch: a replica
of even sides has no targets in the slots that only the odd ones fill."""
import numpy as np
import pytest

import oracle
from gpucpm import workloads as W
from test_gpu_batch import _batch, _batch_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim,n,lo,hi", [(2, 70, 5, 90), (2, 200, 4, 40), (3, 35, 4, 14),
                                          (3, 170, 3, 9)])
@pytest.mark.parametrize("dispatch", ["DISPATCH_REPLICA", "DISPATCH_HYBRID"])
def test_even_and_odd_sides(engine_lib, ndim, n, lo, hi, dispatch):
    import gpucpm
    g = np.random.default_rng(n)
    ws = [W.random_small(tuple(int(k) for k in g.integers(lo, hi, ndim)), 3 + i % 9,
                         seed=300 + i, temperature=5.0 + i % 7) for i in range(n)]
    b = _batch(ws, seed=3, stream0=11)
    b.set_dispatch(getattr(gpucpm, dispatch))
    b.run_mcs(4)
    for r, (x, (lat, a, p, c, cnt)) in enumerate(zip(ws, _batch_state(b, n))):
        o = oracle.OracleSim(x.lattice, x.ncells, **x.oracle_kwargs(), seed=3,
                             stream=11 + r).run(4)
        np.testing.assert_array_equal(lat.view(np.uint32), o.lattice)
        np.testing.assert_array_equal(a, o.area)
        np.testing.assert_array_equal(p, o.perim)
        np.testing.assert_array_equal(c, o.csum)
        assert cnt["accepted"] == int(o.counters[2])
