"""renderer::pt and renderer::lt where the wavefront changes how it runs: waves around a block's 256
queue entries (the shade kernels order a block's entries), path lengths around the longest chunk of
iterations, image mode (shadow rays from the camera vertex), queues smaller than the job. Against the
oracle on matched Philox streams, at the image parity bar (relative L1 2e-3)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(lm, w, h):
    from lightmetrica import synthetic as syn
    scene, film, _ = syn.spheres_scene(n_spheres=8, subdiv=2, ground_quads=8, w=w, h=h)
    scene.build()
    return scene, film


def _err(a, b):
    return np.abs(a - b).sum() / max(np.abs(b).sum(), 1e-12)


@pytest.mark.parametrize("w,h,spp,max_verts,mode,wave", [
    (1, 1, 1, 6, "pixel", 0), (51, 5, 1, 8, "pixel", 0), (16, 16, 1, 8, "pixel", 0), (257, 1, 1, 8, "pixel", 0),
    (24, 16, 3, 2, "pixel", 0), (24, 16, 3, 3, "image", 0), (24, 16, 3, 17, "pixel", 0), (24, 16, 3, 18, "image", 0),
    (24, 16, 3, 21, "pixel", 0), (24, 16, 8, 9, "pixel", 700), (24, 16, 8, 9, "image", 257)])
def test_pt_sizes(lm, oracle_mod, w, h, spp, max_verts, mode, wave):
    scene, film = _scene(lm, w, h)
    lm.load_renderer("r", "pt", scene=scene, output=film, max_verts=max_verts, seed=3, scheduler="sample", spp=spp,
                     primary_ray_sampling_mode=mode, wave_paths=wave).render()
    S = oracle_mod.from_lm_scene(scene, double=True)
    S.build()
    ref, _, _, _ = S.render_pt(w, h, spp, max_verts, seed=3, primary_mode=mode, rng="philox")
    assert _err(film.buffer(), ref) < 2e-3


@pytest.mark.parametrize("samples,max_verts,wave", [(1, 6, 0), (255, 6, 0), (256, 6, 0), (257, 3, 0), (5000, 9, 700)])
def test_lt_sizes(lm, oracle_mod, samples, max_verts, wave):
    scene, film = _scene(lm, 24, 16)
    lm.load_renderer("r", "lt", scene=scene, output=film, max_verts=max_verts, seed=3, scheduler="sample", num_samples=samples,
                     wave_paths=wave).render()
    S = oracle_mod.from_lm_scene(scene, double=True)
    S.build()
    ref = S.render_lt(24, 16, samples, max_verts, seed=3, rng="philox")[0]
    assert np.abs(film.buffer() - ref).sum() <= 2e-3 * np.abs(ref).sum()
