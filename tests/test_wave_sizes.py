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


@pytest.mark.parametrize("order", ["pip", "ipi", "pbp", "ibi", "bpib"])
def test_plain_and_instanced_in_turn(lm, oracle_mod, order):
    """Plain (p) and instanced (i) scenes and batches of both (b) one after another: each table runs the
    chunk of its own kind. The plain image against the oracle (2e-3); the instanced image against its
    flattened build, whose paths differ by fp32 rounding (the bar of the instancing test, 2 %)."""
    from lightmetrica import synthetic as syn
    from lightmetrica.serving import BatchRenderer
    plain, pfilm = _scene(lm, 32, 24)
    S = oracle_mod.from_lm_scene(plain, double=True)
    S.build()
    ref = S.render_pt(32, 24, 4, 8, seed=3, primary_mode="pixel", rng="philox")[0]
    built = [syn.instanced_scene(n_instances=6, n_lat=10, n_lon=14, n_lights=3, w=32, h=24, env_w=32, env_h=16, seed=11,
                                 spread=3.0, accel=a, prefix=f"turn_{a}_") for a in ("embreeinstanced", "sahbvh")]
    for scene, _, _ in built:
        scene.build()
    (inst, ifilm, _), (flat, ffilm, _) = built

    def render(scene, film):
        lm.load_renderer(f"turn_{id(film)}", "pt", scene=scene, output=film, max_verts=8, seed=3, scheduler="sample",
                         spp=4, primary_ray_sampling_mode="pixel").render()

    render(flat, ffilm)
    iref = ffilm.buffer().copy()
    batch = BatchRenderer(queue_paths=1024)
    jobs = {"p": (plain, pfilm), "i": (inst, ifilm)}
    for kind in order:
        table = [jobs[k] for k in ("pi" if kind == "b" else kind)]
        for own in (True, False):  # a batch of its own, reset between tables; the device's
            if own:
                batch.reset()
                batch.render([dict(scene=s, film=f, max_verts=8, spp=4, seed=3) for s, f in table])
            else:
                for s, f in table:
                    render(s, f)
            if kind in "pb":
                assert _err(pfilm.buffer(), ref) < 2e-3
            if kind in "ib":
                assert np.abs(ifilm.buffer() - iref).mean() <= 0.02 * np.abs(iref).mean()
    batch.close()
