"""The work that programs have the framework do, as cases to time: frames of the progressive
renderer, ray queries, forward light walks and gradient steps, through the public entry points
(owe_cuda.CudaBackend / Renderer, owe_cuda.Context, owe_autograd).

A case is a dict of plain values; `kind` says which program it stands for. `prepare` makes what such a
program holds before the call (the scene on the device with its BVH, rays, heights), `run` is one pass
of it. Scenes are the repository's own (scenes.py), with the camera, the ray set or the heights moved
by the seed. Run from the repository's root.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "optical-pathtracer_b200"))

import owe_autograd  # noqa: E402
import owe_cuda  # noqa: E402
import owec_abi as A  # noqa: E402
import scenes  # noqa: E402

PRECISIONS = {"mixed": A.PRECISION_MIXED, "fp32": A.PRECISION_FP32, "fp64": A.PRECISION_FP64}
WAVELENGTHS = {"hero4": A.WAVELENGTHS_HERO4, "uniform1": A.WAVELENGTHS_UNIFORM1}


def frame(name, scene, width, height, spp, depth=12, rr=6, precision="mixed", wavelengths="hero4", integrator="path",
          mesh=0, pinned=True):
    """A frame of the renderer: one pass of spp samples per pixel of a fresh film and its image.
    mesh: meridians of the scene's triangle meshes, where it has any (2 * mesh * mesh / 2 triangles)."""
    return {"name": name, "kind": "frame", "scene": scene, "width": width, "height": height, "spp": spp, "depth": depth,
            "rr": rr, "precision": precision, "wavelengths": wavelengths, "integrator": integrator, "mesh": mesh,
            "pinned": pinned}


def listed():
    return [
        # a viewer's thumbnail while the camera moves: the smallest frame, all launches and latency
        frame("glass_preview", "glass", 64, 48, 1, depth=16, rr=4, pinned=False),
        # the small plain-method configuration: a 256 x 256 film, 64 samples, one wavelength a path
        frame("glass_256_64spp", "glass", 256, 256, 64, depth=16, rr=4, wavelengths="uniform1"),
        # the benchmark's own frame: 2^20 triangles, 1920 x 1080, one sample
        frame("room_1080p", "room", 1920, 1080, 1, mesh=1024),
        # the reference-grade rendering mode, an odd film
        frame("room_fp64", "room", 641, 359, 3, precision="fp64", mesh=512),
        # the fast mode, an ordinary film
        frame("room_fp32", "room", 960, 541, 1, precision="fp32", mesh=512),
        # a product shot with the renderer's default depths: dispersive, rough and metal spheres, a box
        # of fog behind null boundaries, lamp and sun
        frame("gallery_default", "gallery", 480, 270, 2, depth=64, rr=6),
        # the other integrator, as caustics are rendered
        frame("room_light", "room", 960, 540, 1, integrator="light", mesh=512),
        # a lens analyser's spot diagram: ghosts and all through a cemented achromat
        {"name": "lens_walks", "kind": "lens", "walks": 1 << 22, "bins": 1024, "splat": "nearest"},
        # one step of the differentiable caustic: heights set, walks, their adjoint, heights updated
        {"name": "caustic_step", "kind": "caustic", "n": 256, "bins": 512, "walks": 1 << 22},
        # one step of the camera-film optimisation in the fog room: heights set, a pass, its adjoint
        {"name": "camera_step", "kind": "camera", "width": 640, "height": 360, "spp": 2, "n": 256, "mesh": 256},
        # ray queries of a program's own: a batch from host arrays, and a handful (a picker, a probe)
        {"name": "rays_batch", "kind": "rays", "n": 1 << 20, "mesh": 512, "precision": "mixed"},
        {"name": "rays_few", "kind": "rays", "n": 257, "mesh": 256, "precision": "mixed"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _film(rng, paths_lo, paths_hi):
    """(width, height, spp) of a film with that many paths in a pass, of any aspect up to 2:1."""
    paths = _log(rng, paths_lo, paths_hi)
    spp = rng.choice([1, 1, 2, 3, 4, 8, 16])
    pixels = max(64, paths // spp)
    aspect = rng.uniform(0.8, 2.0)
    width = max(8, int(math.sqrt(pixels * aspect)))
    return width, max(8, pixels // width), spp


def draw(rng):
    kind = rng.choice(["glass", "room", "room", "gallery", "light", "lens", "caustic", "camera", "rays"])
    if kind == "glass":
        w, h, spp = _film(rng, 1 << 11, 1 << 22)
        c = frame("", "glass", w, h, spp, depth=rng.randint(8, 16), rr=4,
                  wavelengths=rng.choice(["hero4", "uniform1"]), precision=rng.choice(["mixed", "mixed", "fp32", "fp64"]),
                  pinned=rng.random() < 0.5)
    elif kind == "room":
        precision = rng.choice(["mixed", "mixed", "fp32", "fp64"])
        w, h, spp = _film(rng, 1 << 12, 1 << (20 if precision == "fp64" else 21))
        c = frame("", "room", w, h, spp, depth=rng.randint(6, 12), rr=rng.randint(3, 6), precision=precision,
                  mesh=rng.choice([128, 256, 384, 512]), pinned=rng.random() < 0.5)
    elif kind == "gallery":
        w, h, spp = _film(rng, 1 << 12, 1 << 18)
        c = frame("", rng.choice(["gallery", "gallery", "shapes", "textures", "fog"]), w, h, spp,
                  depth=rng.choice([12, 24, 64]), rr=6, mesh=128)
    elif kind == "light":
        w, h, spp = _film(rng, 1 << 12, 1 << 20)
        c = frame("", "room", w, h, spp, depth=rng.randint(6, 12), rr=rng.randint(3, 6), integrator="light",
                  mesh=rng.choice([128, 256, 384]))
    elif kind == "lens":
        c = {"kind": "lens", "walks": _log(rng, 1 << 12, 1 << 23), "bins": _log(rng, 64, 1024),
             "splat": rng.choice(["nearest", "bilinear"])}
    elif kind == "caustic":
        c = {"kind": "caustic", "n": _log(rng, 32, 320), "bins": _log(rng, 64, 512), "walks": _log(rng, 1 << 14, 1 << 23)}
    elif kind == "camera":
        w, h, spp = _film(rng, 1 << 13, 1 << 19)
        c = {"kind": "camera", "width": w, "height": h, "spp": spp, "n": _log(rng, 32, 320),
             "mesh": rng.choice([64, 128, 256])}
    else:
        c = {"kind": "rays", "n": _log(rng, 1 << 7, 3 << 19), "mesh": rng.choice([64, 128, 256, 512]),
             "precision": rng.choice(["mixed", "mixed", "fp64", "fp32"])}
    c.pop("name", None)
    return c


def _scene(case, seed):
    """The case's scene description, seen from a camera a little off its place by the seed."""
    rng = np.random.default_rng(seed)
    w, h = case.get("width", 8), case.get("height", 8)
    if case["scene"] == "glass":
        sb = scenes.glass_sphere_on_floor(w, h)
    elif case["scene"] == "room":
        sb = scenes.bvh_stress_room(w, h, case["mesh"], case["mesh"] // 2)
    elif case["scene"] == "gallery":
        sb = scenes.materials_gallery(w, h)
    elif case["scene"] == "shapes":
        sb = scenes.shape_gallery(w, h)
    elif case["scene"] == "textures":
        sb = scenes.texture_gallery(w, h)
    else:
        sb = scenes.fog_room(w, h, case["mesh"], case["mesh"] // 2, 64)
    for k in range(3):
        sb.detector.position[k] += rng.uniform(-0.05, 0.05)
    return sb.desc()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        settings = A.make_settings(seed=seed, max_depth=case["depth"], rr_depth=case["rr"],
                                   wavelength_mode=WAVELENGTHS[case["wavelengths"]],
                                   precision=PRECISIONS[case["precision"]])
        renderer = owe_cuda.CudaBackend().create_renderer(_scene(case, seed), settings, case["integrator"])
        out = torch.empty(case["height"], case["width"], 3, dtype=torch.float64, pin_memory=True).numpy() if case["pinned"] else None
        return {"kind": kind, "renderer": renderer, "spp": case["spp"], "out": out}
    ctx = owe_cuda.Context()
    if kind == "rays":
        ctx.upload(_scene({"scene": "room", "mesh": case["mesh"]}, seed))
        ctx.set_settings(A.make_settings(precision=PRECISIONS[case["precision"]]))
        ctx.build_bvh()
        o, d = scenes.random_rays(case["n"], seed, (-2.5, -2.5, 0.3), (2.5, 2.5, 3.7), (-1.2, -1.2, 0.1), (1.2, 1.2, 2.4))
        return {"kind": kind, "ctx": ctx, "o": o, "d": d}
    if kind == "lens":
        sb, info = scenes.achromat_scene(film=case["bins"])
        walk = scenes.achromat_walk(info, seed=seed, splat=A.SPLAT_NEAREST if case["splat"] == "nearest" else A.SPLAT_BILINEAR)
        ctx.upload(sb.desc())
        ctx.build_bvh()
        return {"kind": kind, "ctx": ctx, "walk": walk, "walks": case["walks"]}
    n = case["n"]
    rng = np.random.default_rng(seed)
    # a smooth surface of a few waves, flat at its edge, a tenth of a millimetre high
    x = np.linspace(0.0, 1.0, n)
    h = np.zeros((n, n))
    for _ in range(4):
        kx, ky, ph = rng.integers(1, 5), rng.integers(1, 5), rng.uniform(0, 2 * math.pi)
        h += np.sin(2 * math.pi * kx * x + ph)[None, :] * np.sin(math.pi * ky * x)[:, None]
    h *= 2.5e-5 * (np.sin(math.pi * x)[None, :] * np.sin(math.pi * x)[:, None])
    h[0, :] = h[-1, :] = 0.0
    h[:, 0] = h[:, -1] = 0.0
    heights = torch.from_numpy(h.ravel().copy())
    if kind == "caustic":
        sb, info = scenes.caustic_slab_scene(n=n, wall_bins=case["bins"])
        ctx.upload(sb.desc())
        ctx.build_bvh()
        target = torch.from_numpy(scenes.gaussian_blobs(case["bins"], count=16, seed=seed, sigma_range=(0.01 * case["bins"], 0.04 * case["bins"])))
        return {"kind": kind, "ctx": ctx, "heights": heights, "hf": (info["heightfield"], info["thickness"]),
                "walk": scenes.caustic_walk(info, seed=seed), "walks": case["walks"], "target": target}
    sb, info = scenes.caustic_room(width=case["width"], height=case["height"], n_lon=case["mesh"], n_lat=case["mesh"] // 2, panel_n=n)
    ctx.set_settings(A.make_settings(seed=seed, max_depth=24, rr_depth=6))
    ctx.upload(sb.desc())
    ctx.build_bvh()
    target = torch.from_numpy(rng.uniform(0.0, 0.2, (case["height"], case["width"], 3)))
    return {"kind": kind, "ctx": ctx, "heights": heights, "hf": (info["heightfield"], info["base_z"]), "spp": case["spp"],
            "target": target}


def run(state):
    kind = state["kind"]
    if kind == "frame":
        r = state["renderer"]
        r.reset_observer()
        r.run_pass(state["spp"])
        return r.resolve(out=state["out"])
    ctx = state["ctx"]
    if kind == "rays":
        return ctx.cast_rays(state["o"], state["d"])
    if kind == "lens":
        ctx.walk_reset()
        ctx.walk(state["walk"], 0, state["walks"])
        bins, stats = ctx.walk_resolve()
        return bins, stats["binned"], stats["escaped"], stats["events"]
    # a gradient step: the loss of the film to its target, and the heights moved down it by at most
    # a nanometre
    heights = state["heights"].requires_grad_(True)
    boundary, base_z = state["hf"]
    if kind == "caustic":
        film = owe_autograd.walk_film(heights, ctx, boundary, base_z, state["walk"], 0, state["walks"])
        loss = ((film - state["target"] * film.detach().mean()) ** 2).sum()
    else:
        film = owe_autograd.camera_film(heights, ctx, boundary, base_z, 0, state["spp"])
        loss = ((film - state["target"]) ** 2).sum()
    loss.backward()
    grad = heights.grad
    with torch.no_grad():
        moved = heights - grad * (1e-9 / grad.abs().max().clamp_min(1e-30))
    state["heights"] = moved
    return film.detach(), grad, moved


# What one query of each kind of scene does at the least: closest-hit and any-hit queries per path
# (averages of the renderer's own counts), each a walk from the root to a leaf of an 8-wide tree (192
# flops a node) and one or two primitive tests (40 flops) and a shading event (about 400 flops).
QUERIES = {"glass": 6.0, "room": 13.0, "gallery": 9.0, "shapes": 6.0, "textures": 6.0, "fog": 18.0}


def _query_flops(triangles):
    return 192.0 * max(1.0, math.log(max(8.0, triangles), 8) / 2) + 80.0


def _scene_bytes(triangles, rays):
    """The triangles read once, or where the rays are few the one leaf triangle each of them meets."""
    return 48.0 * min(triangles, rays)


def work(case):
    kind = case["kind"]
    if kind == "frame":
        paths = case["width"] * case["height"] * case["spp"]
        tris = case["mesh"] ** 2
        return {"bytes": 24.0 * case["width"] * case["height"] + _scene_bytes(tris, paths * QUERIES[case["scene"]]),
                "flops": paths * QUERIES[case["scene"]] * (_query_flops(tris) + 400.0)}
    if kind == "rays":
        tris = case["mesh"] ** 2
        return {"bytes": 64.0 * case["n"] + _scene_bytes(tris, case["n"]), "flops": case["n"] * (2 * _query_flops(tris) + 100.0)}
    if kind == "lens":
        return {"bytes": 8.0 * case["bins"] ** 2, "flops": case["walks"] * 4.5 * 500.0}
    tris = 4 * case["n"] ** 2
    if kind == "caustic":
        return {"bytes": 2 * 8.0 * case["bins"] ** 2 + 3 * 8.0 * case["n"] ** 2 + _scene_bytes(tris, 6 * case["walks"]),
                "flops": 2 * case["walks"] * 3 * (_query_flops(tris) + 300.0)}
    tris += 2 * case["mesh"] ** 2
    paths = case["width"] * case["height"] * case["spp"]
    return {"bytes": 2 * 24.0 * case["width"] * case["height"] + 3 * 8.0 * case["n"] ** 2 + _scene_bytes(tris, paths * QUERIES["fog"]),
            "flops": 2 * paths * QUERIES["fog"] * (_query_flops(tris) + 400.0)}


def exact(case, seed):
    """The ray queries' distances, by testing every triangle and every wall in 64 bits. The other
    kinds are sums over random paths, which have no such value."""
    if case["kind"] != "rays" or case["n"] * case["mesh"] ** 2 > 5e9:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    o, d = scenes.random_rays(case["n"], seed, (-2.5, -2.5, 0.3), (2.5, 2.5, 3.7), (-1.2, -1.2, 0.1), (1.2, 1.2, 2.4))
    o, d = torch.from_numpy(o).to(dev), torch.from_numpy(d).to(dev)
    best = torch.full((case["n"],), math.inf, dtype=torch.float64, device=dev)
    # the walls, and the lamp below the ceiling: (axis, its value, half sizes along the other two axes)
    for axis, at, half in ((2, 0.0, 3.0), (2, 4.0, 3.0), (0, -3.0, 3.0), (0, 3.0, 3.0), (1, -3.0, 3.0), (1, 3.0, 3.0), (2, 3.98, 0.8)):
        t = (at - o[:, axis]) / d[:, axis]
        p = o + d * t[:, None]
        inside = t > 0
        for k in range(3):
            if k != axis:
                mid, h = (2.0, 2.0) if k == 2 else (0.0, half)
                inside &= (p[:, k] - mid).abs() <= h
        best = torch.where(inside & (t < best), t, best)
    v, tri = scenes.uv_sphere(case["mesh"], case["mesh"] // 2)
    v = torch.from_numpy(v + np.array([0.0, 0.0, 1.2])).to(dev)
    tri = torch.from_numpy(tri.astype(np.int64)).to(dev)
    a, e1, e2 = v[tri[:, 0]], v[tri[:, 1]] - v[tri[:, 0]], v[tri[:, 2]] - v[tri[:, 0]]
    step = max(1, (1 << 24) // len(tri))
    for k in range(0, case["n"], step):
        ok, dk = o[k:k + step, None, :], d[k:k + step, None, :]
        s = ok - a
        p = torch.linalg.cross(dk.expand_as(s), e2.expand_as(s))
        det = (e1 * p).sum(-1)
        u = (s * p).sum(-1) / det
        q = torch.linalg.cross(s, e1.expand_as(s))
        w = (dk * q).sum(-1) / det
        t = (e2 * q).sum(-1) / det
        t = torch.where((u >= 0) & (w >= 0) & (u + w <= 1) & (t > 0), t, math.inf)
        best[k:k + step] = torch.minimum(best[k:k + step], t.min(-1).values)
    return None, None, best.cpu().numpy()
