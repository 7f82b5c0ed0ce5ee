"""Quads through their precomputed normals against the CPU oracle: hit ids, distances and
shadow answers bit for bit, and images, over axis-aligned, skewed, tiny and huge quads
seen from both sides, under identity, translated and rotated instances, with a quad
light. Image tolerance: no film is involved, so matched streams leave rounding alone (the
device's sine and cosine differ from the C library's in the last place): 1e-5."""

import os

import numpy as np
import pytest

import lambda_b200 as lb
from oracle import port
from tests.helpers import random_rays

pytestmark = pytest.mark.gpu

QUADS = {
    "aligned": ["(-1 -1 0.5) (2 0 0) (0 2 0)", "(-1 -1 -1) (0 0 2) (2 0 0)", "(1 -1 -1) (0 2 0) (0 0 2)"],
    "skewed": ["(-1.1 -0.7 0.3) (1.7 0.2 0.4) (0.3 1.9 -0.5)", "(-1 -1 -1) (0.1 0.2 1.9) (1.8 -0.3 0.1)"],
    "tiny_and_huge": ["(-0.01 0.2 0.1) (0.02 0.001 0) (0 0.03 0.002)", "(-60 -1.2 -60) (0 0.3 120) (120 0 0.1)"],
}
INSTANCES = {
    "identity": "(0 0 0) (0 0 0) (1 1 1)",
    "translated": "(0.1 -0.2 0.3) (0 0 0) (1 1 1)",
    "rotated": "(0.1 0 -0.1) (0.3 0.7 -0.4) (1.5 1.5 1.5)",
}


@pytest.mark.parametrize("quads", sorted(QUADS))
@pytest.mark.parametrize("instance", sorted(INSTANCES))
def test_quads_match_the_oracle(scene_dir, ctx, quads, instance):
    lines = ["Render 40 30 5 4 380 780", "Material grey lambertian 0.6", "Material glass dielectric 1.0 1.5",
             "Material shiny mirror 0.8", "Material lamp emissive 6"]
    lines += [f"Object walls quad {m} {q}" for m, q in zip(("grey", "shiny", "glass"), QUADS[quads])]
    lines += ["Object light quad lamp (-0.4 1.3 -0.5) (0.8 0.1 0) (0 0.05 0.9)",
              f"Instance walls default {INSTANCES[instance]}", "Instance light default (0 0 0) (0 0 0) (1 1 1)",
              "Background equirectangular 0.3", "Camera (0 0.1 -3) (-0.5 0.45 -2) (1 0 0) (0 -0.75 0)"]
    path = os.path.join(scene_dir, f"quads_{quads}_{instance}.lrd")
    with open(path, "w") as f:
        f.write("\n".join(lines) + "\n")
    scene = lb.HostScene.parse(path)
    ctx.upload(scene)
    rays = random_rays(8000, np.array([-2, -2, -2], np.float32), np.array([2, 2, 2], np.float32), 5)
    for a, b in zip(ctx.trace_closest(rays), port.hit(scene, rays)):
        assert np.array_equal(a, b)
    pick = np.arange(len(rays)) % len(scene.light_instances)
    light = scene.light_instances[pick], scene.light_objects[pick]
    assert np.array_equal(ctx.trace_shadow(rays, *light), port.shadow(scene, rays, *light))
    got, want = ctx.render(scene.render_desc(seed=4)), port.render(scene, 4)
    assert np.linalg.norm(got - want) <= 1e-2 * np.linalg.norm(want)
    assert (np.abs(got - want) <= 1e-5 * (np.abs(want) + 1)).mean() > 0.99
