"""Renders through the records that stand for chains of lookups (spectrum textures,
one-layer film thickness, lights) against the CPU oracle, which looks everything up:
constant and checker textures of flat and of dispersive spectra, scalar textures, one
and several lights, films of one and two layers with constant, Perlin and Worley
thickness, under constant, checker and Perlin skies.

Tolerance: matched random streams make the images equal but for rounding (1e-6
relative) unless a rounding difference of the FP32 film flips a reflect/refract choice;
the repository's 1 % bound on linear values covers a flipped pixel in these frames."""

import os

import numpy as np
import pytest

import lambda_b200 as lb
from oracle import port

pytestmark = pytest.mark.gpu

SKIES = {"constant": "0.4", "checker": "tiles", "perlin": "sky", "black": "0"}
LIGHTS = {
    "none": [],
    "one": ["Object lamp0 quad glow (-0.5 1.9 -0.5) (1 0 0) (0 0 1)"],
    "three": ["Object lamp0 quad glow (-0.5 1.9 -0.5) (1 0 0) (0 0 1)", "Object lamp1 quad warm (-1.9 0 0) (0 0 0.5) (0 0.5 0)",
              "Object lamp2 sphere tiled_glow (1.2 1.2 0) 0.2"],
}


def _write(directory, sky, lights):
    names = sorted({line.split()[1] for line in LIGHTS[lights]})
    lines = [
        "Render 48 32 6 4 380 780",
        "Texture red spectrum constant (360 0.05 599 0.05 600 0.65 830 0.65)",
        "Texture blue spectrum constant (360 0.6 480 0.6 520 0.1 830 0.1)",
        "Texture tiles spectrum checker 0.8 0.2 0.25",
        "Texture redblue spectrum checker (360 0.05 600 0.6 830 0.65) (360 0.6 520 0.1 830 0.1) 0.3",
        "Texture cloud scalar perlin 0.2 0.9 3",
        "Texture sky scalar perlin 0.2 1.0 1",
        "Texture thickworley scalar worley 200 800 3",
        "Texture thickperlin scalar perlin 250 600 2",
        "Material m0 lambertian 0.5", "Material m1 lambertian red", "Material m2 lambertian tiles",
        "Material m3 lambertian redblue", "Material m4 lambertian cloud", "Material m5 mirror tiles",
        "Material m6 mirror 0.9", "Material m7 thinfilm [1 1.33 1.5] [thickworley]",
        "Material m8 thinfilm [1 1.33 1.5] [400]", "Material m9 thinfilm [1 1.33 1.5] [thickperlin]",
        "Material m10 thinfilm [1 1.38 2.1 1.5] [100 thickperlin]", "Material m11 dielectric 1.0 1.5",
        "Material glow emissive 8", "Material warm emissive red", "Material tiled_glow emissive tiles",
        "Object floor quad m0 (-3 -0.5 -3) (0 0 6) (6 0 0)",
    ]
    for k in range(1, 12):
        lines.append(f"Object balls sphere m{k} ({(k % 4) * 0.9 - 1.4} {(k // 4) * 0.8 - 0.1} {(k % 3) * 0.4}) 0.35")
    lines += LIGHTS[lights]
    lines += [f"Instance {n} default (0 0 0) (0 0 0) (1 1 1)" for n in ["floor", "balls"] + names]
    lines += [f"Background equirectangular {SKIES[sky]}", "Camera (0 0.6 -4) (-0.75 1.1 -3) (1.5 0 0) (0 -1 0)"]
    path = os.path.join(directory, f"records_{sky}_{lights}.lrd")
    with open(path, "w") as f:
        f.write("\n".join(lines) + "\n")
    return path


@pytest.mark.parametrize("sky,lights", [("constant", "none"), ("checker", "one"), ("perlin", "three"), ("black", "three")])
@pytest.mark.parametrize("path_pixels", [0, 1 << 20])
def test_records_render_what_the_lookups_do(scene_dir, ctx, sky, lights, path_pixels):
    scene = lb.HostScene.parse(_write(scene_dir, sky, lights))
    ctx.upload(scene)
    t = ctx.tuning()
    want = port.render(scene, 11)
    try:
        ctx.set_tuning(128, 128, 1, 0, 4, path_pixels)
        got = ctx.render(scene.render_desc(seed=11))
    finally:
        ctx.set_tuning(t.trace_block, t.shade_block, t.grid_scale, t.max_pixels, t.bvh_width, t.path_kernel_pixels,
                       t.lane_fetch, t.compressed_nodes)
    fine = np.isfinite(want)
    assert np.array_equal(fine, np.isfinite(got))
    assert np.linalg.norm((got - want)[fine]) <= 1e-2 * np.linalg.norm(want[fine])
    assert (np.abs(got - want) <= 1e-5 * (np.abs(want) + 1))[fine].mean() > 0.97
