"""Act runs where device memory has no room for the second copies of lattice
and stamps: they run with one copy, as large lattices always did, and end where
runs with two end."""
import numpy as np
import pytest

from gpucpm import workloads as W
from test_gpu_batch import _batch
from test_gpu_parity import make_engine

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _leave(megabytes):
    """Tensors that leave about that much of the device's memory free."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = []
    for _ in range(64):
        free = torch.cuda.mem_get_info()[0]
        spare = (free - megabytes * MB) // (2 * MB) * 2 * MB
        if spare < 12 * MB:
            break
        try:
            held.append(torch.empty(spare - (32 * MB if len(held) == 0 else 0),
                                    dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            held.append(torch.empty(spare // 2, dtype=torch.uint8, device="cuda"))
    return held


def _engine(ws, dispatch):
    for w in ws:
        nt = w.J.shape[0]
        w.act_lambda, w.act_max = np.zeros(nt, np.float32), np.zeros(nt, np.int32)
        w.act_lambda[1], w.act_max[1] = 30.0, 20
        w.act_lambda[2], w.act_max[2] = 12.0, 8
    if len(ws) == 1:
        return make_engine(ws[0], seed=6)
    b = _batch(ws, seed=6, stream0=0)
    b.set_dispatch(dispatch)
    return b


def _end(e, n):
    e.synchronize()
    e.pull_from_gpu()
    return [(e.lattice(r).copy(), e.act_lattice(r).copy(), *e.tables(r),
             e.counters(r)["accepted"]) for r in range(n)]


@pytest.mark.parametrize("shape,replicas,dispatch,room", [
    ((1536, 1501), 1, 0, 20),      # 3 B a site of lists fit (7 MB), 16 B of copies (37) do not
    ((100, 120, 128), 1, 0, 8),    # 3D: 2 MB, 18 MB
    ((128, 128), 160, 0, 20),      # batches, each dispatch: 8 MB, 41 MB
    ((128, 128), 160, 1, 20),
    ((127, 128), 160, 2, 20),
])
def test_act_runs_without_room_for_second_copies(engine_lib, shape, replicas, dispatch, room):
    import torch
    cells = int(np.prod(shape)) // 100
    ws = [W.random_small(shape, cells, ntypes=2, seed=50 + i % 3, temperature=12.0)
          for i in range(replicas)]
    roomy = _engine(ws, dispatch)
    for mcs in (3, 2):
        roomy.run_mcs(mcs)
    want = _end(roomy, replicas)
    tight = _engine(ws, dispatch)
    tight.act_lattice(0)  # (the stamps themselves)
    held = _leave(room)
    try:
        assert torch.cuda.mem_get_info()[0] < (room + 14) * MB
        for mcs in (3, 2):
            tight.run_mcs(mcs)
        got = _end(tight, replicas)
    finally:
        del held
        torch.cuda.empty_cache()
    assert sum(s[-1] for s in want) > 0
    for g, w in zip(got, want):
        for x, y in zip(g, w):
            np.testing.assert_array_equal(x, y)
