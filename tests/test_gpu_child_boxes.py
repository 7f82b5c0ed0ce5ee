"""Wide nodes by plane (child_boxes): the exact layout's hits at every width equal those
of the compressed layout, which tests each child's own record with the scalar slab
test, on nodes with unused slots, on trees that are a single leaf, and on rays that
start on node planes with direction components that are exactly zero of either sign."""

import os

import numpy as np
import pytest

import lambda_b200 as lb
from lambda_b200 import scenes
from tests.helpers import random_rays

pytestmark = pytest.mark.gpu

ONE_QUAD = """Render 8 8 2 1 380 780
Material grey lambertian 0.5
Object wall quad grey (-1 -1 0) (2 0 0) (0 2 0)
Instance wall default (0 0 0) (0 0 0) (1 1 1)
Background equirectangular 1
Camera (0 0 -3) (-0.5 0.5 -2) (1 0 0) (0 -1 0)
"""


def _scene(directory, name):
    if name == "one_quad":
        path = os.path.join(directory, "child_boxes_quad.lrd")
        with open(path, "w") as f:
            f.write(ONE_QUAD)
        return path
    if name == "cornell":
        return scenes.cornell(directory, 8, 8, 1, name="child_boxes_cornell.lrd").lrd
    if name == "instanced":
        return scenes.instanced_meshes(directory, 8, 8, 1, depth=2, instances=37, segments=12, rings=7, box=8.0,
                                       name="child_boxes_instanced.lrd").lrd
    levels = int(name[4:])
    return scenes.perlin_sphere(directory, 8, 8, 1, depth=2, levels=levels, name=f"child_boxes_{name}.lrd").lrd


def _rays(scene, n, seed):
    nodes = scene.nodes_array()
    lo, hi = nodes["min"][0], nodes["max"][0]
    r = random_rays(n, lo - 0.5, hi + 0.5, seed)
    rng = np.random.default_rng(seed + 1)
    k = np.arange(n)
    # a third start on a node's plane, a third have a zero component (of either sign)
    node, axis = rng.integers(0, len(nodes), n), rng.integers(0, 3, n)
    on = k % 3 == 0
    r[k[on], axis[on]] = np.where(rng.integers(0, 2, n) == 0, nodes["min"][node, axis], nodes["max"][node, axis])[on]
    zero = k % 3 != 1
    r[k[zero], 3 + axis[zero]] = np.where(rng.integers(0, 2, n) == 0, 0.0, -0.0)[zero]
    dead = (r[:, 3:] == 0).all(axis=1)
    r[dead, 3] = 1.0
    return np.ascontiguousarray(r, dtype=np.float32)


@pytest.mark.parametrize("name", ["one_quad", "cornell", "mesh0", "mesh1", "mesh3", "instanced"])
@pytest.mark.parametrize("width", [2, 4, 8])
def test_plane_nodes_find_the_compressed_layouts_hits(scene_dir, ctx, name, width):
    scene = lb.HostScene.parse(_scene(scene_dir, name))
    ctx.upload(scene)
    rays = _rays(scene, 6000, 31 + width)
    pick = np.arange(len(rays)) % len(scene.light_instances)
    light = scene.light_instances[pick], scene.light_objects[pick]
    t = ctx.tuning()
    got = {}
    try:
        for compressed in (1, 0):
            ctx.set_tuning(t.trace_block, t.shade_block, t.grid_scale, t.max_pixels, width, t.path_kernel_pixels,
                           t.lane_fetch, compressed)
            got[compressed] = (*ctx.trace_closest(rays), ctx.trace_shadow(rays, *light))
    finally:
        ctx.set_tuning(t.trace_block, t.shade_block, t.grid_scale, t.max_pixels, t.bvh_width, t.path_kernel_pixels,
                       t.lane_fetch, t.compressed_nodes)
    for a, b in zip(got[0], got[1]):
        assert np.array_equal(a, b)
    assert (got[0][0] >= 0).any()
