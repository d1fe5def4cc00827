"""A call that fails for want of device memory leaves nothing behind: the calls
after it, of other engines in the same thread, succeed."""
import numpy as np
import pytest

from gpucpm import workloads as W
from test_gpu_parity import finish, make_engine

pytestmark = pytest.mark.gpu


def test_engine_after_a_failed_creation(engine_lib):
    import gpucpm
    with pytest.raises(gpucpm.CpmError):
        gpucpm.Batch(3, [(1250, 1250, 1250)] * 45, [10] * 45)  # 350 GB of lattices
    w = W.random_small((14, 15, 13), 20, seed=3, temperature=8.0)
    e = make_engine(w, seed=4)
    e.run_mcs(2)
    finish(e)


def test_engine_after_a_failed_seeding(engine_lib):
    import torch

    import gpucpm
    w = W.random_small((14, 15, 13), 20, seed=3, temperature=8.0)
    e = make_engine(w, seed=4)
    e.run_mcs(1)
    n = 2_000_000  # 128 MB of scratch
    big = gpucpm.create_box(1024, 1024, 1, 2, n, 10.0)
    rng = np.random.default_rng(1)
    pts, vals = rng.random((n, 2)) * 1024.0, ((np.arange(n) + 1) | (1 << 24)).astype(np.uint32)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    held = torch.empty(free - (64 << 20), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(gpucpm.CpmError):
            big.seed_voronoi(0, pts, vals)
        e.recount()
        e.run_mcs(1)
        finish(e)
    finally:
        del held
        torch.cuda.empty_cache()
    big.seed_voronoi(0, pts, vals)
