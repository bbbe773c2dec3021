"""Ray batches at the sizes where the batch trace changes how it runs: eight lanes per ray for a
few rays, fewer rays per warp than lanes, full warps, and every batch's last rays (eight lanes per
ray again). Hits do not depend on the size of the batch a ray is in: bit-exact against the oracle's
exhaustive fp32 test, and bit-identical (exact ties and non-finite rays included) to the same rays
inside a larger batch."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WARP_ROOM = 152 * 32  # warps in flight on the chip; the switch points are multiples of it
SIZES = [1, 2, 3, 4, 5, 8, 31, 33, 127, 129, 4 * WARP_ROOM - 1, 4 * WARP_ROOM + 1, 8 * WARP_ROOM + 3, 32 * WARP_ROOM + 5]


def _soup(n, seed):
    rng = np.random.default_rng(seed)
    c = rng.random((n, 1, 3))
    t = (c + rng.uniform(-0.08, 0.08, (n, 3, 3))).astype(np.float32)
    t[n // 2:n // 2 + n // 8] = t[:n // 8]  # exact duplicates: ties go to the smaller index
    return t.reshape(-1, 9)


def _rays(n, seed):
    rng = np.random.default_rng(seed)
    r = np.empty((n, 8), np.float32)
    r[:, :3] = rng.uniform(-0.2, 1.2, (n, 3))
    r[:, 3] = 1e-3
    d = rng.normal(size=(n, 3))
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 7] = np.where(rng.random(n) < 0.2, 0.2, 1e10)
    return r


def _occluded(lib, accel, rays):
    import torch
    d = torch.from_numpy(rays).cuda()
    out = torch.full((len(rays) + 8,), 7, dtype=torch.uint8, device="cuda")
    from lightmetrica import _native as N
    N.check(lib.lmgpu_accel_occluded_device(accel._h, d.data_ptr(), len(rays), out.data_ptr(), C.c_void_p(0)))
    out = out.cpu().numpy()
    assert (out[len(rays):] == 7).all(), "wrote past the batch"
    return out[:len(rays)]


@pytest.mark.parametrize("two_level", [False, True])
def test_batch_sizes(lm, native_lib, oracle_mod, two_level):
    tri = _soup(700, 5)
    accel = lm.load_accel("accel", "embreeinstanced" if two_level else "sahbvh")
    if two_level:
        m = np.eye(4)
        m[:3, 3] = [0.4, -0.1, 0.2]
        accel.build_instanced(tri, [0, 300, 700], [(0, np.eye(4)), (1, np.eye(4)), (1, m)])
    else:
        accel.build_triangles(tri)
    rays = _rays(max(SIZES), 9)
    rays[7, 0] = np.nan
    rays[11, 7] = np.inf
    rays[13, 4:7] = 0.0
    big = accel.intersect_batch(rays)
    occ = _occluded(native_lib, accel, rays)
    assert np.array_equal(occ != 0, big["prim"] >= 0) and 0 < occ.mean() < 1
    for n in SIZES:
        assert accel.intersect_batch(rays[:n]).tobytes() == big[:n].tobytes(), n
        assert np.array_equal(_occluded(native_lib, accel, rays[:n]), occ[:n]), n
    if not two_level:
        from parity_util import compare_bitexact
        scene = lm.load_scene("scene", "default", accel=lm.load_accel("a2", "sahbvh"))
        k = np.arange(3 * len(tri))
        mesh = lm.load_mesh("soup", "raw", ps=tri.reshape(-1, 3), ns=[0, 0, 1], ts=[0, 0], fs={"p": k, "n": 0 * k, "t": 0 * k})
        scene.add_primitive(mesh=mesh, material=lm.load_material("m", "diffuse"))
        S = oracle_mod.from_lm_scene(scene, double=False)
        S.build(robust=True)
        ok = np.ones(len(rays), bool)
        ok[[7, 11, 13]] = False
        t, uv, ids, _ = S.intersect(rays[ok], brute=True, refine_t=True)
        compare_bitexact(big[ok], t, uv, ids, rays[ok], S.triangles())


@pytest.mark.parametrize("far", [0.0, 0.5, 0.97, 1.0])  # rays from far away: all but a few miss
@pytest.mark.parametrize("n", [32 * WARP_ROOM + 1, 64 * WARP_ROOM + 31, 500001])
def test_distance_pass(lm, n, far):
    """Larger batches take the hit distances in a pass of its own, whose warps collect the hits of the
    rays they pass: the bits of the same rays in batches whose trace launch takes them."""
    accel = lm.load_accel("accel", "sahbvh")
    accel.build_triangles(_soup(700, 5))
    rays = _rays(n, 17)
    rays[:, :3] = 0.5
    rays[np.random.default_rng(3).random(n) < far, :3] = 50.0
    rays[:, 7] = 1e10
    out = accel.intersect_batch(rays)
    step = 100003
    parts = b"".join(accel.intersect_batch(rays[i:i + step]).tobytes() for i in range(0, n, step))
    assert out.tobytes() == parts
