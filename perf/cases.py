"""Workloads of the renderer, timed through the package's public entry points.

A case is a dict of plain values; `listed()` names twelve, `draw(rng)` gives others of
the same ranges. `prepare` makes what a program holds before the call (the context with
its uploaded scene, weights and launch shapes; rays or film queries), `run` is one call,
`work` the bytes and operations it cannot do without, and `exact` the float64 values of
the outputs that have a closed form.

Kinds:
  render   lambda_render of one of the four scene families of lambda_b200/scenes.py
  batch    lambda_render_batch of many views of one scene
  rays     lambda_trace_closest and lambda_trace_shadow on the same rays (host arrays)
  film     film queries: the FP32 or FP64 transfer matrix or the tensor-core surrogate
  train    a training run of the surrogate: labels, optimiser steps, audit
"""

import math
import os
import tempfile

import numpy as np
import torch

import lambda_b200 as lb
from lambda_b200 import _native, scenes, surrogate

FORMS = {"exact": lb.RENDER_THINFILM_EXACT, "surrogate": lb.RENDER_THINFILM_SURROGATE, "fp64": lb.RENDER_THINFILM_FP64}
HUGE = 1e29  # a hit distance above this is a miss


def listed():
    return [
        # a preview after an edit: one sample of a thumbnail, the image back in host memory
        {"name": "preview_160x90", "kind": "render", "scene": "thinfilm", "width": 160, "height": 90, "depth": 16,
         "spp": 1, "form": "exact", "host": True, "lane_fetch": False, "detail": 0},
        # the Cornell box of the benchmark's configurations: mixed materials, few pixels
        {"name": "cornell_256", "kind": "render", "scene": "cornell", "width": 256, "height": 256, "depth": 8,
         "spp": 16, "form": "exact", "host": True, "lane_fetch": False, "detail": 0},
        # the headline frame (thin-film spheres at 1080p) at a part of its 256 samples
        {"name": "thinfilm_1080p", "kind": "render", "scene": "thinfilm", "width": 1920, "height": 1080, "depth": 16,
         "spp": 16, "form": "exact", "host": False, "lane_fetch": False, "detail": 0},
        # the same frame with the learned film
        {"name": "thinfilm_1080p_surrogate", "kind": "render", "scene": "thinfilm", "width": 1920, "height": 1080,
         "depth": 16, "spp": 4, "form": "surrogate", "host": False, "lane_fetch": False, "detail": 0},
        # a check frame in the double-precision film form, at an odd size
        {"name": "thinfilm_fp64_641x363", "kind": "render", "scene": "thinfilm", "width": 641, "height": 363,
         "depth": 16, "spp": 9, "form": "fp64", "host": True, "lane_fetch": False, "detail": 0},
        # the mesh configuration: 1,048,576 triangles (9 subdivisions), 1024 x 1024, depth 12
        {"name": "mesh_1024", "kind": "render", "scene": "mesh", "width": 1024, "height": 1024, "depth": 12, "spp": 4,
         "form": "exact", "host": False, "lane_fetch": False, "detail": 9},
        # the instanced configuration (10,000 instances of 100,000 triangles) at a draft
        # size, in the launch shapes the autotuner picks for it (rays taken lane by lane)
        {"name": "instanced_960x540", "kind": "render", "scene": "instanced", "width": 960, "height": 540, "depth": 32,
         "spp": 1, "form": "surrogate", "host": False, "lane_fetch": True, "detail": 10000},
        # many uneven views of one scene in one call (turntables, training-data renders)
        {"name": "batch_24_views", "kind": "batch", "scene": "thinfilm", "views": 24, "spp": 16, "form": "exact",
         "detail": 0},
        # picking and visibility queries of a host program against a mesh
        {"name": "rays_200k", "kind": "rays", "scene": "mesh", "n": 200003, "detail": 8},
        # film reflectance for a table of spectra, device to device
        {"name": "film_exact_4m", "kind": "film", "form": "exact", "n": 4194304, "host": False},
        # the same through the learned film, an odd count
        {"name": "film_surrogate_3m", "kind": "film", "form": "surrogate", "n": 3000001, "host": False},
        # a short training run of the surrogate at its usual batch
        {"name": "train_262k", "kind": "train", "samples": 262144, "epochs": 1, "batch": 8192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render"] * 5 + ["batch", "rays", "film", "film", "train"])
    if kind == "render":
        scene = rng.choice(["thinfilm", "thinfilm", "cornell", "mesh", "instanced"])
        pixels = _log_int(rng, 96 * 54, 1920 * 1080 if scene != "instanced" else 640 * 360)
        aspect = rng.choice([1.0, 4 / 3, 16 / 9])
        width = max(8, int(math.sqrt(pixels * aspect)))
        height = max(8, int(width / aspect))
        most = {"thinfilm": 16, "cornell": 16, "mesh": 9, "instanced": 1}[scene]
        spp = rng.choice([s for s in (1, 4, 9, 16) if s <= most])
        form = rng.choice(["exact", "exact", "surrogate", "fp64"]) if scene in ("thinfilm", "instanced") else "exact"
        if form == "fp64":  # the double-precision form costs about twice the others
            spp = min(spp, 4)
        detail = {"thinfilm": 0, "cornell": 0, "mesh": rng.choice([5, 7, 8]),
                  "instanced": _log_int(rng, 20, 2000)}[scene]
        return {"kind": kind, "scene": scene, "width": width, "height": height, "depth": rng.randint(2, 24),
                "spp": spp, "form": form, "host": rng.random() < 0.5, "lane_fetch": scene == "instanced",
                "detail": detail}
    if kind == "batch":
        scene = rng.choice(["thinfilm", "mesh"])
        return {"kind": kind, "scene": scene, "views": rng.randint(2, 24), "spp": rng.choice([1, 4, 16]),
                "form": "exact", "detail": 0 if scene == "thinfilm" else 7}
    if kind == "rays":
        scene = rng.choice(["cornell", "thinfilm", "mesh", "instanced"])
        return {"kind": kind, "scene": scene, "n": _log_int(rng, 100, 200000),
                "detail": {"mesh": 7, "instanced": 300}.get(scene, 0)}
    if kind == "film":
        host = rng.random() < 0.4
        return {"kind": kind, "form": rng.choice(["exact", "fp64", "surrogate"]),
                "n": _log_int(rng, 64, 200000 if host else 4000000), "host": host}
    return {"kind": kind, "samples": _log_int(rng, 20000, 262144), "epochs": 1, "batch": rng.choice([2048, 4096, 8192])}


# ---------------------------------------------------------------------------
# What a program has in hand before the call
# ---------------------------------------------------------------------------

_assets = None


def _asset_dir():
    """Scene files of this process (meshes are written once, as a user's are on disk)."""
    global _assets
    if _assets is None:
        _assets = tempfile.TemporaryDirectory(prefix="lambda_cases_")
    return _assets.name


def _scene(case, seed, ctx, width=64, height=64, depth=4, spp=1):
    d, kind = _asset_dir(), case["scene"]
    kw = dict(width=width, height=height, depth=depth, spp=spp)
    if kind == "cornell":
        sc = scenes.cornell(d, **kw)
    elif kind == "thinfilm":  # the seed places the spheres
        sc = scenes.thinfilm_spheres(d, seed=seed, **kw)
    elif kind == "mesh":
        sc = scenes.perlin_sphere(d, levels=case["detail"], **kw)
    else:  # the seed places the instances; the mesh file is the same for every seed
        obj = os.path.join(d, "latlong_250x201.obj")
        if not os.path.exists(obj):
            scenes.write_latlong_sphere_obj(obj, 250, 201)
        # the density of the full configuration, whatever the instance count
        box = 100.0 * (case["detail"] / 10000.0) ** (1.0 / 3.0)
        sc = scenes.instanced_meshes(d, instances=case["detail"], box=box, seed=seed, **kw)
    return lb.HostScene.parse_gpu(ctx, sc.lrd)


def _film_queries(n, seed):
    """Uniform queries of the trained box, as [n, 5] float32 on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lb.default_film_range()
    lo = torch.tensor([getattr(r, k)[0] for k in surrogate.RANGE_KEYS], device="cuda")
    hi = torch.tensor([getattr(r, k)[1] for k in surrogate.RANGE_KEYS], device="cuda")
    return lo + (hi - lo) * torch.rand(n, 5, device="cuda", generator=g)


def prepare(case, seed):
    kind = case["kind"]
    ctx = lb.Context(0)
    s = {"kind": kind, "ctx": ctx}
    if kind == "render":
        scene = _scene(case, seed, ctx, case["width"], case["height"], case["depth"], case["spp"])
        ctx.upload(scene)
        flags = FORMS[case["form"]]
        if case["form"] == "surrogate":
            surrogate.install(ctx)
        if case["lane_fetch"]:
            ctx.set_tuning(64, 128, 2, 0, 4, lane_fetch=1)
        shape = (case["height"], case["width"], 3)
        if case["host"]:
            s["out"] = np.zeros(shape, np.float32)
        else:
            flags |= lb.RENDER_OUTPUT_DEVICE
            s["out"] = torch.zeros(shape, dtype=torch.float32, device="cuda")
        s["desc"] = scene.render_desc(seed=seed, flags=flags)
        s["scene"] = scene
    elif kind == "batch":
        scene = _scene(case, seed, ctx)
        ctx.upload(scene)
        view = {} if case["scene"] == "thinfilm" else dict(target=(0.0, 0.0, 0.0), distance=(2.6, 4.0),
                                                           height=(-1.0, 1.5), jitter=0.2)
        # the views' sizes, depths and cameras are the case's; their noise is the seed's
        descs = scenes.random_pose_jobs(scene, case["views"], seed=4, resolutions=(128, 256, 512),
                                        spps=[v for v in (1, 4, 16) if v <= case["spp"]], flags=FORMS[case["form"]],
                                        **view)
        for i, d in enumerate(descs):
            d.seed = seed * 1000 + i
        s["descs"] = descs
        s["outs"] = [np.zeros((d.settings.height, d.settings.width, 3), np.float32) for d in descs]
        s["scene"] = scene
    elif kind == "rays":
        scene = _scene(case, seed, ctx)
        ctx.upload(scene)
        rng = np.random.default_rng(seed)
        n = case["n"]
        # from a sphere around the scene towards points inside it
        node = scene.nodes_array()[0]
        mid, half = (node["min"] + node["max"]) / 2, (node["max"] - node["min"]) / 2
        o = rng.normal(size=(n, 3))
        o = mid + o / np.linalg.norm(o, axis=1, keepdims=True) * np.linalg.norm(half) * 1.2
        d = mid + rng.uniform(-0.8, 0.8, (n, 3)) * half - o
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        s["rays"] = np.concatenate([o, d], 1).astype(np.float32)
        # visibility of a light per ray: the scene's lights in turn (the last is the sky)
        pick = np.arange(n) % len(scene.light_instances)
        s["light"] = (scene.light_instances[pick], scene.light_objects[pick])
        s["scene"] = scene
    elif kind == "film":
        if case["form"] == "surrogate":
            surrogate.install(ctx)
        q = _film_queries(case["n"], seed)
        s["call"] = {"exact": ctx.thinfilm_exact, "fp64": ctx.thinfilm_fp64, "surrogate": ctx.surrogate_eval}[case["form"]]
        s["out"] = None
        if case["host"]:
            q = q.cpu().numpy()
        else:
            dt = torch.float64 if case["form"] == "fp64" else torch.float32
            s["out"] = torch.zeros(case["n"], 4, dtype=dt, device="cuda")
        s["q"] = q
    else:
        s["args"] = dict(samples=case["samples"], epochs=case["epochs"], batch=case["batch"], lr=2e-3, seed=seed)
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "render":
        return ctx.render(s["desc"], out=s["out"])
    if kind == "batch":
        return ctx.render_batch(s["descs"], outs=s["outs"])
    if kind == "rays":
        inst, obj, t = ctx.trace_closest(s["rays"])
        return inst, obj, t, ctx.trace_shadow(s["rays"], *s["light"])
    if kind == "film":
        return s["call"](s["q"], s["out"])
    rep = ctx.surrogate_train(**s["args"])
    return ctx.surrogate_get()[0], rep.final_loss, rep.mean_abs_error


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

_MLP_FLOPS = 2 * (5 * 64 + 64 * 64 + 64 * 64 + 64 * 4)
# bytes of one triangle's record and of its share of the tree, read once
_TRI_BYTES = 116 + 2 * 32
# segments per path and operations per segment (ray setup, box and primitive tests of
# one root-to-leaf walk, scatter) of a typical path of each scene
_SEGMENTS = {"thinfilm": 3.3, "cornell": 5.0, "mesh": 1.7, "instanced": 1.7}
_OPS = 400


def _scene_bytes(case):
    return {"thinfilm": 64 * 180, "cornell": 8 * 180, "mesh": 4 * 4 ** case["detail"] * _TRI_BYTES,
            "instanced": 100000 * _TRI_BYTES + case["detail"] * 144}[case["scene"]]


def _batch_shape(case):
    """Pixels and paths of the batch's views (random_pose_jobs draws them from seed 4)."""
    rng = np.random.default_rng(4)
    spps = [v for v in (1, 4, 16) if v <= case["spp"]]
    pixels = paths = 0
    for _ in range(case["views"]):
        res, spp = int(rng.choice((128, 256, 512))), int(rng.choice(spps))
        rng.integers(4, 25)
        rng.uniform(size=7)  # azimuth, distance, height, target, field of view
        pixels += res * res
        paths += res * res * spp
    return pixels, paths


def work(case):
    kind = case["kind"]
    if kind in ("render", "batch"):
        if kind == "render":
            pixels = case["width"] * case["height"]
            paths = pixels * case["spp"]
        else:
            pixels, paths = _batch_shape(case)
        segments = paths * min(_SEGMENTS[case["scene"]], case.get("depth", 24) + 1)
        flops = segments * _OPS
        if case["form"] == "surrogate" and case["scene"] in ("thinfilm", "instanced"):
            flops += paths * 4 * _MLP_FLOPS  # about one film hit per path
        return {"bytes": pixels * 12 + _scene_bytes(case), "flops": flops}
    if kind == "rays":
        return {"bytes": case["n"] * (24 + 12 + 24 + 8 + 4) + _scene_bytes(case), "flops": 2 * case["n"] * _OPS}
    if kind == "film":
        per = {"exact": 80, "fp64": 80, "surrogate": _MLP_FLOPS + 40}[case["form"]]
        return {"bytes": case["n"] * (20 + (32 if case["form"] == "fp64" else 16)), "flops": case["n"] * per}
    # forward and backward of every sample (three products per weight) and the FP64 labels
    # of the samples and the 2^18 audit queries, which the network also evaluates
    n, audit = case["samples"] * case["epochs"], 1 << 18
    return {"bytes": n * 36 + case["samples"] * 36 + audit * 52,
            "flops": 3 * n * _MLP_FLOPS + (case["samples"] + audit) * 80 + audit * _MLP_FLOPS}


# ---------------------------------------------------------------------------
# Float64 values
# ---------------------------------------------------------------------------

def _film_exact(q):
    """(R_s, R_p, T_s, T_p) of a film of index n_film between air and n_sub, from the
    characteristic matrices, in complex128."""
    lam, c0, d, nf, ns = (q.double()[:, i].to(torch.complex128) for i in range(5))
    n = [torch.ones_like(nf), nf, ns]
    s2 = 1 - c0 * c0
    cos = [c0, torch.sqrt(1 - s2 / (nf * nf)), torch.sqrt(1 - s2 / (ns * ns))]
    phase = torch.exp(1j * 2 * math.pi / lam * nf * d * cos[1])

    def stack(pol):
        m = None
        for j in range(2):
            a, b = (n[j] * cos[j], n[j + 1] * cos[j + 1]) if pol == "s" else (n[j + 1] * cos[j], n[j] * cos[j + 1])
            t = 2 * n[j] * cos[j]
            i00, i01 = (a + b) / t, (a - b) / t
            if m is None:
                m = (i00 / phase, i01 * phase)
            else:
                m = (m[0] * i00 + m[1] * i01, m[0] * i01 + m[1] * i00)
        r = (m[1] / m[0]).abs() ** 2
        trans = (n[2] * cos[2]).real / (n[0] * cos[0]).real * (1 / m[0]).abs() ** 2
        return r, trans

    # M01 and M10 of the product agree in modulus for a lossless stack, so the first row is enough
    (rs, ts), (rp, tp) = stack("s"), stack("p")
    return torch.stack([rs, rp, ts, tp], 1)


def _film_network(q):
    """The surrogate network of the shipped weights, in float64."""
    p, r = surrogate.load()
    p = torch.from_numpy(p).cuda().double()
    lo = [getattr(r, k)[0] for k in surrogate.RANGE_KEYS]
    hi = [getattr(r, k)[1] for k in surrogate.RANGE_KEYS]
    lam, c0, d, nf, ns = (q.double()[:, i] for i in range(5))
    cf = torch.sqrt(torch.clamp(1 - (1 - c0 * c0) / (nf * nf), min=0))
    delta = 4 * math.pi * nf * d * cf / lam
    norm = [2 * (v - lo[k]) / (hi[k] - lo[k]) - 1 for k, v in ((1, c0), (3, nf), (4, ns))]
    h = torch.stack([torch.cos(delta), torch.sin(delta)] + norm, 1)
    at = 0
    for k, (out, inp) in enumerate(((64, 5), (64, 64), (64, 64), (4, 64))):
        w = p[at:at + out * inp].reshape(out, inp)
        at += out * inp
        h = h @ w.T + p[at:at + out]
        at += out
        h = torch.relu(h) if k < 3 else h
    return h


def exact(case, seed):
    if case["kind"] != "film":
        return None  # path-traced images, hit ids and trained weights have no closed form
    q = _film_queries(case["n"], seed)
    return _film_network(q) if case["form"] == "surrogate" else _film_exact(q)
