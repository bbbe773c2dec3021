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
