"""Renders through both closest-hit walks (a warp's 32 rays to the end, in the separate,
fused and path kernels; lane by lane with TLAS and BLAS in one loop) with cameras whose
rays start on BVH node planes and have direction components that are exactly zero, of
either sign: the same images and statistics bit for bit at every BVH width, and the CPU
oracle's images. No film is involved, so matched streams leave rounding alone (the
device's sine and cosine differ from the C library's in the last place): 1e-5."""

import os

import numpy as np
import pytest

import lambda_b200 as lb
from lambda_b200 import scenes
from oracle import port

pytestmark = pytest.mark.gpu

# spheres in instances of their own put node planes at 0 on every axis
PLANES = """Render 24 16 3 4 380 780
Material a lambertian 0.7
Material b mirror 0.8
Material c lambertian 0.3
Object w quad a (-0.9 -1 -1) (0 2 0) (0 0 2)
Object w quad b (-1 -0.8 -1) (0 0 2) (2 0 0)
Object w quad c (-1 -1 0.9) (1 0 0) (0 1 0)
Object w quad a (0 0 0.9) (1 0 0) (0 1 0)
Object s sphere c (0.5 0.5 0.5) 0.5
Object t sphere a (-0.25 -0.25 -0.25) 0.25
Instance w default (0 0 0) (0 0 0) (1 1 1)
Instance s default (0 0 0) (0 0 0) (1 1 1)
Instance t default (0 0 0) (0 0 0) (1 1 1)
Background equirectangular 0.6
Camera (0 0 -3) (-0.5 0.5 -2) (1 0 0) (0 -1 0)
"""


def _lrd(directory, name):
    if name == "planes":
        path = os.path.join(directory, "walk_planes.lrd")
        with open(path, "w") as f:
            f.write(PLANES)
        return path
    if name == "cornell":
        return scenes.cornell(directory, 24, 16, 4, depth=3, name="walk_cornell.lrd").lrd
    if name == "mesh":
        return scenes.perlin_sphere(directory, 24, 16, 4, depth=3, levels=3, name="walk_mesh.lrd").lrd
    return scenes.instanced_meshes(directory, 24, 16, 4, depth=3, instances=37, segments=12, rings=7, box=8.0,
                                   name="walk_instanced.lrd").lrd


def _cameras(scene, n, seed):
    """(position, corner, horizontal, vertical) of cameras on node planes: rays fan out
    within the plane or, every fourth, all run along one axis."""
    rng = np.random.default_rng(seed)
    nodes = scene.nodes_array()
    lo, hi = nodes[0]["min"], nodes[0]["max"]
    out = []
    for k in range(n):
        a = rng.integers(0, 3)
        b, c = (a + 1) % 3, (a + 2) % 3
        on = nodes["min" if k % 2 else "max"][:, a]
        zeros = on[on == 0]
        pos = rng.uniform(lo, hi).astype(np.float32)
        pos[a] = zeros[0] if len(zeros) and k % 3 else rng.choice(on)
        if k % 3 == 0:  # from outside, grazing the plane
            pos[b] = lo[b] - np.float32(0.5)
        aim = (lo + hi) / 2 + rng.uniform(-0.3, 0.3, 3) * (hi - lo) - pos
        fwd, across = np.zeros(3), np.zeros(3)
        if k % 4 != 3:
            angle = np.arctan2(aim[c], aim[b])
            fwd[b], fwd[c] = np.cos(angle), np.sin(angle)
            across[b], across[c] = -np.sin(angle), np.cos(angle)
        else:
            fwd[b] = np.sign(aim[b])
            across = 0.2 * fwd
        down = 0.3 * fwd
        corner = (pos + fwd - 0.5 * across).astype(np.float32)
        corner[a] = across[a] = down[a] = 0.0 if k % 2 else -0.0  # the direction's zero: + or -
        if pos[a] != 0:
            corner[a] = pos[a]
        out.append((pos, corner, across, down))
    return out


@pytest.mark.parametrize("name", ["planes", "cornell", "mesh", "instanced"])
def test_both_walks_render_grazing_cameras_alike(scene_dir, ctx, name):
    lrd = _lrd(scene_dir, name)
    with open(lrd) as f:
        lines = f.read().splitlines()
    keep = ctx.tuning()
    hits = 0
    base = lb.HostScene.parse(lrd)
    for k, view in enumerate(_cameras(base, 16, 5)):
        parallel = k % 4 == 3  # a camera that scene files do not allow: no oracle
        if parallel:
            scene = base
        else:
            camera = "Camera " + " ".join("(" + " ".join(repr(float(x)) for x in v) + ")" for v in view)
            path = os.path.join(scene_dir, f"walk_{name}_{k}.lrd")
            with open(path, "w") as f:
                f.write("\n".join(camera if line.startswith("Camera") else line for line in lines) + "\n")
            scene = lb.HostScene.parse(path)
        ctx.upload(scene)
        desc = scene.render_desc(seed=3)
        for field, v in zip(("position", "corner", "horizontal", "vertical"), view):
            getattr(desc.settings.camera, field)[:] = [float(x) for x in v]
        first = None
        try:
            for width in (2, 4, 8):
                for path_pixels, fetch, fused in ((0, 0, 0), (0, 0, 1), (1 << 20, 0, 0), (0, 1, 0)):
                    ctx.set_tuning(keep.trace_block, keep.shade_block, keep.grid_scale, keep.max_pixels, width,
                                   path_pixels, fetch, 0, fused)
                    img = ctx.render(desc)
                    st = ctx.stats()
                    got = img, (st.paths, st.segments, st.shadow_rays)
                    first = first or got
                    form = (k, width, path_pixels, fetch, fused)
                    assert got[1] == first[1], form
                    assert np.array_equal(got[0], first[0], equal_nan=True), form
        finally:
            ctx.set_tuning(keep.trace_block, keep.shade_block, keep.grid_scale, keep.max_pixels, keep.bvh_width,
                           keep.path_kernel_pixels, keep.lane_fetch, keep.compressed_nodes, keep.fused_bounce)
        hits += first[1][1] - first[1][0]
        if parallel:
            continue
        want = port.render(scene, 3)
        fine = np.isfinite(want)
        assert np.array_equal(np.isfinite(first[0]), fine)
        assert (np.abs(first[0] - want) <= 1e-5 * (np.abs(want) + 1))[fine].mean() > 0.99, k
    assert hits > 1000
