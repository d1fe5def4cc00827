"""Seeding of lattices so long that FP32 distances are coarse against a bucket:
those just short of the double-only search and those in it, against a k-d tree
in double.  Every point is there twice under two indices; the lower one wins."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,npoints", [
    ((3, 450000), 330000),     # 3 ferr = 1.93, buckets 2.02 wide: FP32 first
    ((3, 600000), 450000),     # 2.57 against 1.5: double alone
    ((600000, 3), 450000),
    ((3, 4, 300000), 200000),  # 3D: 1.29 against 2
    ((4, 3, 700000), 900000),  # 3.00 against 2
])
def test_long_lattices_take_their_nearest_points(engine_lib, shape, npoints):
    spatial = pytest.importorskip("scipy.spatial")
    import gpucpm
    nd = len(shape)
    rng = np.random.default_rng(npoints)
    size = np.array(shape[::-1], np.float64)
    pts = rng.random((npoints, nd)) * size
    pts = np.concatenate([pts, pts])
    rng.shuffle(pts)
    ids = np.arange(len(pts)) + 1
    e = gpucpm.create_box(*((shape[::-1] + (1,))[:3]), nd, len(pts), 10.0)
    e.seed_voronoi(0, pts, (ids | (1 << 24)).astype(np.uint32))
    e.recount()
    e.synchronize()
    e.pull_from_gpu()
    got = (e.lattice(0).view(np.uint32) & 0xFFFFFF).astype(np.int64).ravel() - 1
    uniq, first = np.unique(pts, axis=0, return_index=True)  # the lower index of each pair
    grids = np.meshgrid(*[np.arange(n, dtype=np.float64) for n in shape], indexing="ij")
    sites = np.stack([g.ravel() for g in grids[::-1]], axis=1)
    _, near = spatial.cKDTree(uniq, boxsize=size).query(sites, workers=-1)
    bad = np.flatnonzero(got != first[near])
    # (the tree's own rounding may decide between points at one distance)

    def dist2(k, s):
        d = np.abs(sites[s] - pts[k])
        return (np.minimum(d, size - d) ** 2).sum(axis=1)
    worse = dist2(got[bad], bad) > dist2(first[near[bad]], bad)
    assert not worse.any(), (len(bad), sites[bad[worse]][:3])
    assert len(bad) < 10
