"""A context launches the graph of its last pass again when the next one has the same
shape. Every image must be what a context that never rendered before gives: over
seeds, cameras, outputs, scenes of the same size, film forms, tunings, limits, wave
counts, path-kernel passes, and two contexts that take turns."""

import numpy as np
import pytest

import lambda_b200 as lb
from lambda_b200 import scenes, surrogate

pytestmark = pytest.mark.gpu

FORMS = [lb.RENDER_THINFILM_EXACT, lb.RENDER_THINFILM_FP64, lb.RENDER_THINFILM_SURROGATE]


def _scenes(directory):
    out = []
    for seed in (3, 4):  # the same sizes, other spheres
        sc = scenes.thinfilm_spheres(directory, 64, 36, 4, depth=5, seed=seed, name=f"plan_{seed}.lrd")
        out.append(lb.HostScene.parse(sc.lrd))
    sc = scenes.cornell(directory, 64, 36, 4, depth=5, name="plan_cornell.lrd")
    out.append(lb.HostScene.parse(sc.lrd))
    return out


def _fresh(scene, desc, tuning):
    with lb.Context(0) as c:
        surrogate.install(c)
        c.upload(scene)
        c.set_tuning(*tuning)
        img = c.render(desc)
        return img, c.stats()


def _same(a, b):
    return np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("path_pixels", [0, 1 << 20])
def test_kept_plans_render_what_fresh_contexts_do(scene_dir, path_pixels):
    worlds = _scenes(scene_dir)
    wave = (128, 128, 1, 0, 4, path_pixels)
    steps = []
    for scene in (0, 0, 1, 0, 2, 1):  # the same scene again, one of the same size, another
        for seed, flags, samples in ((1, FORMS[0], 4), (2, FORMS[0], 4), (2, FORMS[1], 4), (2, FORMS[2], 4), (2, FORMS[0], 9)):
            steps.append((scene, seed, flags, samples, wave))
    steps += [(0, 7, FORMS[0], 4, (256, 64, 2, 0, 8, path_pixels)), (0, 7, FORMS[0], 4, wave),
              (0, 7, FORMS[0], 4, (64, 128, 1, 0, 4, path_pixels, 1)), (0, 7, FORMS[0], 4, wave)]
    contexts = [lb.Context(0), lb.Context(0)]
    try:
        for c in contexts:
            surrogate.install(c)
        held = [None, None]
        for k, (scene, seed, flags, samples, tuning) in enumerate(steps):
            desc = worlds[scene].render_desc(seed=seed, flags=flags, samples=samples)
            want, stats = _fresh(worlds[scene], desc, tuning)
            for j, c in enumerate(contexts):
                if held[j] != scene or k % 7 == 0:
                    c.upload(worlds[scene])
                    held[j] = scene
                c.set_tuning(*tuning)
                assert _same(c.render(desc), want), (k, j)
                got = c.stats()
                assert (got.segments, got.shadow_rays, got.thinfilm_hits, got.waves, got.kernel_launches) == (
                    stats.segments, stats.shadow_rays, stats.thinfilm_hits, stats.waves, stats.kernel_launches)
    finally:
        for c in contexts:
            c.close()


def test_plans_survive_limits_batches_and_profiles(scene_dir):
    scene = _scenes(scene_dir)[0]
    with lb.Context(0) as c:
        surrogate.install(c)
        c.upload(scene)
        c.set_tuning(128, 128, 1, 0, 4, 0)
        desc = scene.render_desc(seed=5, flags=lb.RENDER_THINFILM_SURROGATE)
        want = c.render(desc)
        c.set_limits(mma_polls=0)
        with pytest.raises(lb.LambdaError):
            c.render(desc)
        c.reset_limits()
        assert _same(c.render(desc), want)
        # a larger frame moves the buffers that the plan names; a profiled one runs no graph
        big = scene.render_desc(seed=5, flags=lb.RENDER_THINFILM_SURROGATE)
        big.settings.width, big.settings.height = 400, 300
        c.render(big)
        assert _same(c.render(desc), want)
        lb.stage_profile(c, desc, np.empty_like(want))
        assert _same(c.render(desc), want)
        imgs = c.render_batch([desc, desc])
        assert _same(imgs[0], want) and _same(imgs[1], want)
        assert _same(c.render(desc), want)
        # other weights in the same buffers
        p, r = c.surrogate_get()
        c.surrogate_set(p * np.float32(0.5), r)
        assert not _same(c.render(desc), want)
        c.surrogate_set(p, r)
        assert _same(c.render(desc), want)


def test_query_staging_grows_shrinks_and_repeats(scene_dir):
    scene = _scenes(scene_dir)[2]
    rng = np.random.default_rng(0)
    rays = rng.normal(size=(300_000, 6)).astype(np.float32)
    pick = np.arange(len(rays)) % len(scene.light_instances)
    with lb.Context(0) as c:
        c.upload(scene)
        full = c.trace_closest(rays)
        occ = c.trace_shadow(rays, scene.light_instances[pick], scene.light_objects[pick])
        for n in (1, 300_000, 17, 70_000, 300_000):
            for a, b in zip(c.trace_closest(rays[:n]), full):
                assert np.array_equal(a, b[:n])
            assert np.array_equal(c.trace_shadow(rays[:n], scene.light_instances[pick][:n], scene.light_objects[pick][:n]),
                                  occ[:n])
        for bad in ((-1, 0), (0, -1), (len(scene.instances_array()), 0), (0, len(scene.objects_array())), (-2, -1)):
            with pytest.raises(lb.LambdaError):
                c.trace_shadow(rays[:3], np.array([-1, bad[0], -1]), np.array([-1, bad[1], -1]))
        assert np.array_equal(c.trace_shadow(rays[:3], scene.light_instances[pick][:3], scene.light_objects[pick][:3]), occ[:3])
