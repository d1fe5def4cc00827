"""Which sweep runs, and that the engine says so: small 2D lattices start in
the cluster sweep whatever their sides, can be taken out of it and put back,
and a lattice that no cluster holds with its tables runs the grid sweep under
every fill."""
import numpy as np
import pytest

import oracle
from gpucpm import workloads as W
from test_gpu_parity import assert_same, finish, make_engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,ncells", [
    ((17, 4), 3), ((31, 32), 12), ((64, 64), 40), ((50, 200), 60), ((80, 70), 30),
    ((101, 200), 120), ((256, 256), 640),
])
def test_cluster_sweep_is_reported_and_can_be_asked_for(engine_lib, shape, ncells):
    import gpucpm
    w = W.random_small(shape, ncells, ntypes=3, seed=ncells, temperature=9.0)
    e = make_engine(w, seed=8)
    default = e.fill
    assert default in (gpucpm.FILL_PARITY, gpucpm.FILL_TMA)
    c = e.sweep_config()
    assert c["fill"] == "cluster" and c["warps_per_block"] == 16 and c["grid"] in (8, 16)
    e.run_mcs(3)
    e.set_fill(gpucpm.FILL_PARITY)
    assert e.sweep_config()["fill"] == "parity" and e.fill == gpucpm.FILL_PARITY
    e.run_mcs(3)
    e.set_fill(gpucpm.FILL_CLUSTER)
    assert e.sweep_config()["fill"] == "cluster" and e.fill == gpucpm.FILL_CLUSTER
    e.run_mcs(3)
    finish(e)
    sim = oracle.OracleSim(w.lattice, w.ncells, **w.oracle_kwargs(), seed=8).run(9)
    assert_same(e, sim)


def test_lattices_that_no_cluster_holds(engine_lib):
    import gpucpm
    # the rows fit, 20,000 rows of tables do not: accepted, and the grid sweep runs
    e = gpucpm.create_box(256, 256, 1, 2, 20000, 10.0)
    assert e.sweep_config()["fill"] == "parity"
    e.set_fill(gpucpm.FILL_CLUSTER)
    assert e.fill == gpucpm.FILL_CLUSTER and e.sweep_config()["fill"] == "parity"
    assert e.sweep_config()["grid"] > 16
    # neither fits
    for shape in ((1024, 1024), (600, 601)):
        e = gpucpm.create_box(*shape, 1, 2, 500, 10.0)
        assert e.sweep_config()["fill"] == "parity"
        with pytest.raises(gpucpm.CpmError, match="cluster"):
            e.set_fill(gpucpm.FILL_CLUSTER)
    for e in (gpucpm.create_box(32, 32, 32, 3, 20, 10.0),
              gpucpm.Batch(2, [(64, 64), (64, 64)], [10, 10])):
        assert e.sweep_config()["fill"] == "parity"
        with pytest.raises(gpucpm.CpmError, match="cluster"):
            e.set_fill(gpucpm.FILL_CLUSTER)


def test_act_runs_report_the_grid_sweep(engine_lib):
    w = W.random_small((64, 64), 40, ntypes=3, seed=3, temperature=9.0)
    w.act_lambda = np.array([0, 10, 0, 0], np.float32)
    w.act_max = np.array([0, 20, 0, 0], np.int32)
    e = make_engine(w, seed=8)
    e.run_mcs(2)
    assert e.sweep_config()["fill"] == "parity"
    e.set_act(0, 1, 0, 0.0)
    e.run_mcs(2)
    assert e.sweep_config()["fill"] == "cluster"
    finish(e)


def test_autotune_keeps_the_fill_that_it_did_not_time(engine_lib):
    """The cluster sweep is no candidate of act runs, so tuning one decides
    nothing about the runs after it."""
    import gpucpm
    w = W.random_small((64, 64), 40, ntypes=3, seed=3, temperature=9.0)
    w.act_lambda = np.array([0, 10, 0, 0], np.float32)
    w.act_max = np.array([0, 20, 0, 0], np.int32)
    for fill in (None, gpucpm.FILL_CLUSTER):
        e = make_engine(w, seed=8)
        if fill is not None:
            e.set_fill(fill)
        before = e.fill
        e.autotune(probe_mcs=2)
        assert e.fill == before
        e.set_act(0, 1, 0, 0.0)
        e.run_mcs(2)
        assert e.fill == before and e.sweep_config()["fill"] == "cluster"
        finish(e)


def test_autotune_keeps_the_fill_after_an_error(engine_lib):
    """A site of an unknown cell, which the sweep reports and skips, ends the
    tuning; variant and fill are as before it."""
    import gpucpm
    w = W.random_small((64, 64), 40, ntypes=3, seed=3, temperature=9.0)
    e = make_engine(w, seed=8)
    before, config = e.fill, e.sweep_config()
    e.synchronize()
    e.device_lattice(0)[10, 10] = w.ncells + 5 + (1 << 24)
    import torch
    torch.cuda.synchronize()
    with pytest.raises(gpucpm.CpmError, match="autotune"):
        e.autotune(probe_mcs=2)
    assert e.fill == before and e.sweep_config() == config
