"""Device memory after seeding from many points: a call's scratch (64 bytes a
point) is given back where it is large."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.mark.parametrize("npoints,kept", [(1_000_000, 256), (6_000_000, 32)])
def test_seeding_gives_large_scratch_back(engine_lib, npoints, kept):
    import torch

    import gpucpm
    n = 4096
    e = gpucpm.create_box(n, n, 1, 2, npoints, 10.0)
    rng = np.random.default_rng(npoints)
    vals = ((np.arange(npoints) + 1) | (1 << 24)).astype(np.uint32)
    e.seed_voronoi(0, rng.random((100, 2)) * n, vals[:100])  # (kernels loaded)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    e.seed_voronoi(0, rng.random((npoints, 2)) * n, vals)
    assert free - torch.cuda.mem_get_info()[0] <= kept * MB
    e.seed_voronoi(0, rng.random((100, 2)) * n, vals[:100])  # (and it can be used again)
    e.recount()
    e.synchronize()
    e.pull_from_gpu()
    assert len(np.unique(e.lattice(0))) == 100
