"""The cluster sweep of lattices whose tables no block holds whole: rows dealt
over the blocks, against the oracle, over one launch and several and under a
graph; and what the engine reports and tunes."""
import numpy as np
import pytest

import oracle
from gpucpm import workloads as W
from test_gpu_parity import assert_same, finish, make_engine
from test_gpu_rowtiles import _terms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,ncells,rows,terms", [
    ((72, 66), 60, 20000, False),
    ((173, 120), 9000, 9000, False),      # cells of two sites, odd ny
    ((101, 180), 400, 12345, True),       # rows that do not divide evenly
    ((181, 203), 5000, 16389, True),      # odd sides, two rounds of targets
    ((17, 4), 3, 30001, False),           # more blocks than rows of sites
])
@pytest.mark.parametrize("runs", [(24,), (1, 1, 13, 9)])
def test_dealt_tables_match_oracle(engine_lib, shape, ncells, rows, terms, runs):
    import gpucpm
    w = W.random_small(shape, ncells, ntypes=3, seed=70 + ncells, temperature=11.0)
    if terms:
        _terms(w, ncells)
    w.ncells = rows
    e = make_engine(w, seed=6)
    assert e.sweep_config()["fill"] == "parity"  # not by itself
    e.set_fill(gpucpm.FILL_CLUSTER)
    c = e.sweep_config()
    assert c["fill"] == "cluster" and c["warps_per_block"] == 16
    for i, mcs in enumerate(runs):
        (e.run_graph if i % 2 else e.run_mcs)(mcs)
    finish(e)
    sim = oracle.OracleSim(w.lattice, w.ncells, **w.oracle_kwargs(), seed=6).run(sum(runs))
    assert_same(e, sim)
    assert int(sim.counters[2]) > 0


def test_autotuned_lattices_of_many_rows(engine_lib):
    """Whatever the tuner picks runs, also where a caller's cluster fill would
    not, and the trajectory goes on."""
    import gpucpm
    w = W.random_small((256, 256), 640, ntypes=3, seed=5, temperature=9.0)
    w.ncells = 16000
    e = make_engine(w, seed=6)
    e.set_fill(gpucpm.FILL_CLUSTER)
    assert e.sweep_config()["fill"] == "parity"
    e.run_mcs(3)
    e.autotune(4)
    assert (e.sweep_config()["fill"] == "cluster") == (e.fill == gpucpm.FILL_CLUSTER)
    e.run_mcs(9)
    finish(e)
    sim = oracle.OracleSim(w.lattice, w.ncells, **w.oracle_kwargs(), seed=6).run(12)
    assert_same(e, sim)
