"""The pass counts of a run, read with each chunk for short tables and after the last one for longer: the
status of every job after single chunks and at the end, at both sides of the line, and the images."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spp", [[1023], [1024], [1025], [512, 512], [512, 513], [700, 1, 2000]])
def test_status_follows_the_run(lm, spp):
    from lightmetrica import synthetic as syn
    from lightmetrica.serving import BatchRenderer
    scene, _ = syn.box_scene(seed=3, w=8, h=8, prefix="pc_")
    scene.build()
    films = [lm.load_film(f"pc_film{k}", "bitmap", w=8, h=8) for k in range(len(spp))]
    batch = BatchRenderer(queue_paths=1 << 14)
    jobs = [batch.submit(scene, f, max_verts=7, spp=n, seed=3) for f, n in zip(films, spp)]
    before, left = [0] * len(jobs), 1
    while left:
        left = batch.run(1)
        now = [batch.status(j) for j in jobs]
        assert all(a <= p <= n and done == (p == n) for a, (p, done), n in zip(before, now, spp))
        assert all(done for _, done in now) == (left == 0)
        before = [p for p, _ in now]
    images = []
    for j, f in zip(jobs, films):
        batch.resolve(j)
        images.append(f.buffer().copy())
    batch.reset()
    jobs = [batch.submit(scene, f, max_verts=7, spp=n, seed=3) for f, n in zip(films, spp)]
    assert batch.run(0) == 0 and all(batch.status(j) == (n, True) for j, n in zip(jobs, spp))
    for j, f, image in zip(jobs, films, images):
        batch.resolve(j)
        # the same paths; fp32 additions in another order: n of them, at most 2^-24 relative each
        np.testing.assert_allclose(f.buffer(), image, rtol=max(spp) * 7 * 2.0 ** -24, atol=1e-6)
    batch.close()
