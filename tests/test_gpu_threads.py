"""Engines in several host threads at once, each with its own handle, while
another thread makes and frees engines.  A kernel's shared-memory limit belongs
to the function, not to a handle, so a launch must not depend on the sizes that
other threads launch or plan with: no call fails, and every engine ends where
it ends when it runs alone."""
import threading

import numpy as np
import pytest

from gpucpm import workloads as W
from test_gpu_parity import finish, make_engine

pytestmark = pytest.mark.gpu


def _state(e):
    finish(e)
    return (e.lattice(0).copy(),) + e.tables(0)


@pytest.mark.parametrize("shapes,ncells", [
    (((64, 64), (256, 256)), (40, 655)),                # cluster sweep, by the lattice
    (((1200, 1200), (2048, 2048)), (14400, 41943)),     # grid sweep, by the plan's warps
])
def test_two_engines_in_two_threads(engine_lib, shapes, ncells):
    import gpucpm
    ws = [W.random_small(s, n, ntypes=3, seed=n, temperature=9.0) for s, n in zip(shapes, ncells)]
    runs = 400
    want = []
    for w in ws:
        e = make_engine(w, seed=21)
        e.run_mcs(runs)
        want.append(_state(e))
    engines = [make_engine(w, seed=21) for w in ws]
    errors, done = [], threading.Event()
    gate = threading.Barrier(len(ws) + 1)

    def run(e):
        gate.wait()
        for _ in range(runs):
            try:
                e.run_mcs(1)
                e.synchronize()
            except gpucpm.CpmError as exc:
                errors.append(str(exc))
                return

    def churn():
        gate.wait()
        k = 0
        while not done.is_set():
            k += 1
            try:
                gpucpm.create_box(40 + k % 200, 48, 1, 2, 20, 8.0)
            except gpucpm.CpmError as exc:
                errors.append(str(exc))
                return

    threads = [threading.Thread(target=run, args=(e,)) for e in engines]
    maker = threading.Thread(target=churn)
    for t in threads + [maker]:
        t.start()
    for t in threads:
        t.join()
    done.set()
    maker.join()
    assert not errors, errors[:3]
    for e, state in zip(engines, want):
        for got, ref in zip(_state(e), state):
            np.testing.assert_array_equal(got, ref)
