"""A rebuild that the GPU builder refuses leaves the accel as it was: the same hits and statistics as
before, whether the refused mesh is smaller or larger than the tree's and whether its list of clusters
goes through the passes over all blocks or only the last ones."""
import numpy as np
import pytest

from test_bvh_host import _rays, _soup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("built,refused", [(1000, 9), (5000, 1000), (5000, 1024), (5000, 1025), (9, 1000), (300, 1025), (300, 20000)])
def test_refused_rebuild_keeps_the_tree(lm, built, refused):
    from lightmetrica._native import LmGpuError
    acc = lm.load_accel("acc", "sahbvh", builder="ploc")
    acc.build_triangles(_soup(built, 3))
    rays = _rays(20000, 5)
    before, stats = acc.intersect_batch(rays).tobytes(), acc.stats()
    for value in (np.nan, np.inf):
        bad = _soup(refused, 4)
        bad[refused // 2, 4] = value
        with pytest.raises(LmGpuError, match="non-finite"):
            acc.build_triangles(bad)
        assert acc.intersect_batch(rays).tobytes() == before
    now = acc.stats()
    assert all(now[k] == stats[k] for k in ("num_tris", "num_nodes", "max_depth"))
    acc.build_triangles(_soup(refused, 4))  # the accel still takes a mesh
    fresh = lm.load_accel("fresh", "sahbvh", builder="sah")
    fresh.build_triangles(_soup(refused, 4))
    assert acc.intersect_batch(rays).tobytes() == fresh.intersect_batch(rays).tobytes()


def _overflowing(a, b):
    """A flat mesh (z = 0) of finite coordinates: `a` triangles whose merged boxes have infinite areas and,
    across a gap beyond the float range, `b` without area. The collapse makes the first set one leaf of
    `a` > 3 triangles beside an inner node over the second."""
    t = np.zeros((a + b, 3, 3), np.float32)
    k = np.arange(a)
    t[:a, :, 0] = np.stack([k * 1e36 - 3e38, np.full(a, -1e38), np.full(a, -2e38)], 1)
    t[:a, :, 1] = np.stack([np.zeros(a), np.full(a, 1e30), -1e30 * (k + 1)], 1)
    t[a:, :, 0] = 3e38
    t[a:, :, 1] = np.arange(b)[:, None] * 10 + np.arange(3)
    return t.reshape(-1, 9)


@pytest.mark.parametrize("a,b", [(5, 5), (6, 200), (40, 300), (4, 1000), (500, 500)])
def test_areas_beyond_the_float_range(lm, a, b):
    """The emission stops at the level whose nodes it cannot lay out; the accel takes the next mesh."""
    from lightmetrica._native import LmGpuError
    acc = lm.load_accel("acc", "sahbvh", builder="ploc")
    for _ in range(2):
        with pytest.raises(LmGpuError, match="wide node layout"):
            acc.build_triangles(_overflowing(a, b))
    rays = _rays(5000, 5)
    acc.build_triangles(_soup(2000, 4))
    fresh = lm.load_accel("fresh", "sahbvh", builder="sah")
    fresh.build_triangles(_soup(2000, 4))
    assert acc.intersect_batch(rays).tobytes() == fresh.intersect_batch(rays).tobytes()


@pytest.mark.parametrize("built", [9, 5000])  # larger and smaller buffers than the refused mesh takes
def test_rebuild_refused_late(lm, built):
    """An emission that fails has overwritten the accel's tree: queries are refused until the next build."""
    from lightmetrica._native import LmGpuError
    acc = lm.load_accel("acc", "sahbvh", builder="ploc")
    acc.build_triangles(_soup(built, 3))
    with pytest.raises(LmGpuError, match="wide node layout"):
        acc.build_triangles(_overflowing(6, 200))
    rays = _rays(5000, 5)
    with pytest.raises(LmGpuError, match="not built"):
        acc.intersect_batch(rays)
    acc.build_triangles(_soup(2000, 4))
    fresh = lm.load_accel("fresh", "sahbvh", builder="sah")
    fresh.build_triangles(_soup(2000, 4))
    assert acc.intersect_batch(rays).tobytes() == fresh.intersect_batch(rays).tobytes()
