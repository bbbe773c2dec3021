"""The GPU builder where its passes change form: lists short enough for the one-block passes, just
longer ones, and lists that take several batches of passes; one-child and full nodes. The layout's
invariants, and hits equal to the host builder's tree bit for bit."""
import numpy as np
import pytest

import bvh8_sim as sim
from test_bvh_host import _check_structure, _rays, _soup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 9, 1023, 1024, 1025, 2500])
def test_structure_at_pass_boundaries(native_lib, n):
    tri_p = _soup(n, n)
    nodes, tris, depth = sim.build_gpu(native_lib, tri_p)
    assert depth >= 1 and len(nodes) >= 1
    _check_structure(nodes, tris, tri_p)


@pytest.mark.parametrize("n,copies", [(30, 1), (1025, 1), (40000, 1), (300, 20)])
def test_hits_equal_host_builder(lm, n, copies):
    tri = np.tile(_soup(n, 3), (copies, 1))  # copies: clusters of identical boxes
    rays = _rays(30000, 5)
    hits = []
    for b in ("sah", "ploc"):
        acc = lm.load_accel("acc_" + b, "sahbvh", builder=b)
        acc.build_triangles(tri)
        acc.build_triangles(tri)  # a rebuild reuses the accel's buffers
        hits.append(acc.intersect_batch(rays).tobytes())
    assert hits[0] == hits[1]
