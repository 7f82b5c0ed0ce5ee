"""Closest-hit queries take rays lane by lane from a counter: a ray's answer does not
depend on how many are asked, from one ray to more than the GPU holds at once, and a
scene of one leaf, missed by most rays, answers like the fixed per-ray form."""

import numpy as np
import pytest

import lambda_b200 as lb
from lambda_b200 import scenes
from oracle import port
from tests.helpers import random_rays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("compressed", [0, 1])
def test_answers_do_not_depend_on_the_batch(scene_dir, ctx, compressed):
    sc = scenes.instanced_meshes(scene_dir, 8, 8, 1, depth=2, instances=50, segments=16, rings=9, box=10.0,
                                 name="query_sizes.lrd")
    scene = lb.HostScene.parse(sc.lrd)
    ctx.upload(scene)
    nodes = scene.nodes_array()
    n_max = 148 * 16 * 128 + 5
    rays = random_rays(n_max, nodes["min"][0] - 1, nodes["max"][0] + 1, 77)
    t = ctx.tuning()
    try:
        ctx.set_tuning(t.trace_block, t.shade_block, t.grid_scale, t.max_pixels, t.bvh_width, t.path_kernel_pixels,
                       t.lane_fetch, compressed)
        full = ctx.trace_closest(rays)
        for n in (1, 2, 31, 32, 33, 127, 128, 129, 148 * 128, 148 * 128 + 1):
            for a, b in zip(ctx.trace_closest(rays[:n]), full):
                assert np.array_equal(a, b[:n]), n
    finally:
        ctx.set_tuning(t.trace_block, t.shade_block, t.grid_scale, t.max_pixels, t.bvh_width, t.path_kernel_pixels,
                       t.lane_fetch, t.compressed_nodes)
    k = 3000
    for a, b in zip(full, port.hit(scene, rays[:k])):
        assert np.array_equal(a[:k], b)
    assert (full[0] >= 0).any() and (full[0] < 0).any()
