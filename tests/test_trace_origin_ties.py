"""Rays that start on a surface (tmin 0): the hit lies at t = +0 or -0, several triangles share it, and
the smallest index wins, whichever of them is tested first. A range [0, -0] holds that hit too. Integer
coordinates: every test is exact, so the expected index needs no arithmetic."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDE = 24  # quads along a side; vertices at integer points of the plane z = 0


def _grid(seed):
    """Triangles in shuffled order with shuffled corners (both windings: both signs of zero), and per grid
    vertex the smallest index among those that touch it."""
    rng = np.random.default_rng(seed)
    x, y = (a.reshape(-1) for a in np.meshgrid(np.arange(SIDE), np.arange(SIDE), indexing="ij"))
    a, b, c, d = (np.stack([x + i, y + j], 1) for i, j in ((0, 0), (1, 0), (1, 1), (0, 1)))
    tri = np.concatenate([np.stack([a, b, c], 1), np.stack([a, c, d], 1)])
    tri = tri[rng.permutation(len(tri))]
    for t in tri:
        t[:] = t[rng.permutation(3)]
    first = np.full((SIDE + 1, SIDE + 1), len(tri), np.int64)
    for k in range(3):
        np.minimum.at(first, (tri[:, k, 0], tri[:, k, 1]), np.arange(len(tri)))
    p = np.zeros((len(tri), 3, 3), np.float32)
    p[:, :, :2] = tri
    return p.reshape(-1, 9), first


@pytest.mark.parametrize("copies", [1, 400])  # eight lanes per ray; full warps
@pytest.mark.parametrize("two_level", [False, True])
@pytest.mark.parametrize("tmax", [1e10, 0.0, -0.0])
@pytest.mark.parametrize("tmin", [0.0, -0.0])
def test_smallest_index_at_the_origin(lm, native_lib, tmin, tmax, two_level, copies):
    import torch
    from lightmetrica import _native as N
    tri, first = _grid(3)
    accel = lm.load_accel("accel", "embreeinstanced" if two_level else "sahbvh")
    if two_level:
        accel.build_instanced(tri, [0, len(tri)], [(0, np.eye(4))])
    else:
        accel.build_triangles(tri)
    x, y = (a.reshape(-1) for a in np.meshgrid(np.arange(SIDE + 1), np.arange(SIDE + 1), indexing="ij"))
    rays = np.zeros((2 * len(x), 8), np.float32)
    rays[:, 0], rays[:, 1] = np.tile(x, 2), np.tile(y, 2)
    rays[:, 3], rays[:, 7] = tmin, tmax
    rays[:len(x), 6], rays[len(x):, 6] = 1.0, -1.0
    rays = np.tile(rays, (copies, 1))
    h = accel.intersect_batch(rays)
    assert np.array_equal(h["prim"], np.tile(first[x, y], 2 * copies))
    assert (h["t"] == 0.0).all()
    d = torch.from_numpy(rays).cuda()
    occ = torch.zeros(len(rays), dtype=torch.uint8, device="cuda")
    N.check(native_lib.lmgpu_accel_occluded_device(accel._h, d.data_ptr(), len(rays), occ.data_ptr(), C.c_void_p(0)))
    assert bool((occ != 0).all())
