"""Timed cases of the path tracer, each through its public entry points.

Every case is what a program that embeds the library has it do: batches of
rays against a built scene, the ray sort, a scene whose instances move, a mesh
built from scratch, frames of the render loop read back, a batch of scenes,
and a gradient step of the differentiable form. Geometry, rays, materials and
parameters come from the seed; the sizes come from the case.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from raydemo_b200 import api, capi, diff, scenes

TMAX = 10.0  # rays start in or near the unit cube: past everything, and a miss stays on the scale of a hit


def listed():
    return [
        # picking and visibility queries: a handful of rays, where launches and latency are the cost
        {"name": "trace_1k", "kind": "trace", "tris": 20000, "rays": 1000, "order": "incoherent", "mem": "device", "obj": True},
        # a bake's gather over a mid-sized mesh, neither count a multiple of anything
        {"name": "trace_262k", "kind": "trace", "tris": 300007, "rays": 262147, "order": "incoherent", "mem": "device", "obj": True},
        # the closest-hit microbenchmark: every ray its own way through 2M triangles
        {"name": "trace_4m", "kind": "trace", "tris": 2097152, "rays": 4194304, "order": "incoherent", "mem": "device", "obj": False},
        # one camera ray per pixel of a 2048 x 2048 view
        {"name": "trace_coherent_4m", "kind": "trace", "tris": 2097152, "rays": 4194304, "order": "coherent", "mem": "device", "obj": False},
        # rays that come from and go back to a host program's page-locked buffers
        {"name": "trace_host_1m", "kind": "trace", "tris": 2097152, "rays": 1048583, "order": "incoherent", "mem": "host", "obj": False},
        # a dynamic scene: a few instances move, the next batch of rays sees them moved
        {"name": "instances_1k", "kind": "moving", "instances": 1024, "level": 3, "moved": 64, "rays": 262144},
        # the ray sort over one camera's rays (1280 x 720)
        {"name": "sort_921k", "kind": "sort", "rays": 921600, "gather": True},
        # a mesh that a program generates: added, committed (BVH build) and probed
        {"name": "build_131k", "kind": "build", "tris": 131071, "rays": 65536},
        # the smallest frame: an interactive preview, one sample a pass, pixels read back
        {"name": "cornell_256", "kind": "render", "scene": "cornell", "w": 256, "h": 256, "bounces": 4, "samples": 1},
        # the large frame: metallic-roughness materials, area lights, long paths, pixels read back
        {"name": "atrium_720p", "kind": "render", "scene": "atrium", "w": 1280, "h": 720, "bounces": 8, "samples": 4},
        # many scenes of very different sizes rendered together, pixels kept on the device
        {"name": "batch_16", "kind": "batch", "first": 0, "scenes": 16, "samples": 4},
        # a gradient step: forward render and adjoint of one view
        {"name": "diff_256", "kind": "diff", "w": 256, "h": 256, "samples": 8, "bounces": 4, "texture": 512},
    ]


def _log(rng, lo, hi):
    """An integer from lo to hi, spread over its logarithm; odd ones as likely as even ones."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "trace", "sort", "moving", "build", "render", "render", "batch", "diff"])
    if kind == "trace":
        return {"kind": kind, "tris": _log(rng, 1000, 2097152), "rays": _log(rng, 500, 4194304),
                "order": rng.choice(["incoherent", "coherent"]), "mem": rng.choice(["device", "device", "host"]), "obj": rng.random() < 0.5}
    if kind == "sort":
        return {"kind": kind, "rays": _log(rng, 1000, 4194304), "gather": rng.random() < 0.5}
    if kind == "moving":
        n = _log(rng, 33, 4096)
        return {"kind": kind, "instances": n, "level": rng.randint(1, 4), "moved": rng.randint(1, min(n, 128)), "rays": _log(rng, 1000, 1048576)}
    if kind == "build":
        return {"kind": kind, "tris": _log(rng, 1000, 262144), "rays": _log(rng, 500, 65536)}
    if kind == "render":
        scene = rng.choice(["cornell", "lightmap", "atrium"])
        w = _log(rng, 64, 640)
        h = w if scene == "lightmap" else rng.randint(max(48, w // 2), w)
        return {"kind": kind, "scene": scene, "w": w, "h": h, "bounces": rng.randint(1, 8), "samples": rng.randint(1, 4)}
    if kind == "batch":
        return {"kind": kind, "first": rng.randint(16, 4000), "scenes": rng.randint(2, 6), "samples": rng.randint(1, 4)}
    w = _log(rng, 64, 256)
    return {"kind": "diff", "w": w, "h": rng.randint(w // 2, w), "samples": rng.randint(1, 8), "bounces": rng.randint(2, 4),
            "texture": _log(rng, 64, 512)}


# ---------------------------------------------------------------- inputs


def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed(1000003 * (seed + 1) + salt)


def _soup(case, seed):
    """Random triangles in the unit cube (n, 3, 3), lognormal edges that shrink as the count grows."""
    n, g = case["tris"], _gen(seed, 1)
    mean = 0.005 * (2097152 / n) ** (1.0 / 3.0)
    c = torch.rand((n, 1, 3), generator=g, device="cuda")
    d = torch.randn((n, 3, 3), generator=g, device="cuda")
    d = d / d.norm(dim=2, keepdim=True)
    return c + d * torch.exp(math.log(mean) + 0.5 * torch.randn((n, 3, 1), generator=g, device="cuda"))


def _rays(n, seed, order="incoherent"):
    """(n, 8) rays: through the unit cube in every direction, or a pinhole view of it in pixel order."""
    g = _gen(seed, 2)
    r = torch.zeros((n, 8), device="cuda")
    if order == "coherent":
        w = max(1, math.isqrt(n))
        k = math.tan(math.radians(22.5))
        i = torch.arange(n, device="cuda")
        eye = torch.tensor([0.5, 0.5, -1.5], device="cuda") + 0.1 * (torch.rand(3, generator=g, device="cuda") - 0.5)
        x = (((i % w).float() + 0.5) / w * 2 - 1) * k
        y = (1 - ((i // w).float() + 0.5) / (n / w) * 2) * k
        d = torch.stack([x, y, torch.ones_like(x)], dim=1)
        r[:, 0:3] = eye
    else:
        r[:, 0:3] = torch.rand((n, 3), generator=g, device="cuda")
        d = torch.randn((n, 3), generator=g, device="cuda")
    r[:, 3] = TMAX
    r[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    return r


def _soup_attrs(tris, layout):
    """Vertex attributes of a triangle soup: positions, one normal, (a tangent), texture coordinates."""
    n = len(tris) * 3
    a = torch.zeros((n, 11 if layout == 2 else 8), device="cuda")
    a[:, 0:3] = tris.reshape(-1, 3)
    a[:, 5] = 1.0
    if layout == 2:
        a[:, 6] = 1.0
    else:
        a[:, 6:8] = tris.reshape(-1, 3)[:, 0:2]
    return a.cpu().numpy(), np.arange(n, dtype=np.uint32)


def _scene(r, spec):
    sc = r.CreateScene()
    sc.SetEnvironment(**spec["env"])
    for rgba, srgb, mips in spec["textures"]:
        sc.AddTexture(rgba, is_srgb=srgb, generate_mipmaps=mips)
    for m in spec["materials"]:
        sc.AddMaterial(**m)
    for attrs, idx, shapes, layout in spec["meshes"]:
        sc.AddMesh(attrs, idx, shapes, layout=layout)
    for mesh, xf in spec["instances"]:
        sc.AddMeshInstance(mesh, xf)
    for l in spec["lights"]:
        sc.AddLight(**l)
    sc.set_current_cam(sc.AddCamera(api.CameraDesc(**spec["camera"])))
    sc.Commit()
    return sc


def _batch_spec(index, seed):
    """Scene `index` of the batched configuration (its sizes fixed by the index), its colours, sun and placement from the seed."""
    spec = scenes.batch_scene(index)
    rng = np.random.default_rng([seed, index])
    for m in spec["materials"]:
        m["main_color"] = tuple(float(v) for v in rng.uniform(0.2, 0.9, 3))
    for k in range(1, len(spec["instances"])):
        mesh, xf = spec["instances"][k]
        xf = np.array(xf, np.float32)
        xf[12] += rng.uniform(-1.0, 1.0)
        xf[14] += rng.uniform(-1.0, 1.0)
        spec["instances"][k] = (mesh, xf)
    sun = rng.normal(size=3)
    sun[1] = -abs(sun[1]) - 1.0
    spec["lights"][0]["direction"] = tuple(float(v) for v in sun / np.linalg.norm(sun))
    return spec


def _hits(buf, obj=None):
    """A hit buffer (n, 4) int32 as its triangle ids and its float t, u, v."""
    out = {"prim": buf[:, 0], "tuv": buf.view(torch.float32)[:, 1:]}
    if obj is not None:
        out["obj"] = obj
    return out


class _DevicePixels:
    """A renderer's framebuffer in device memory, as torch reads it; a tensor made of it keeps the renderer."""

    def __init__(self, ptr, renderer):
        self.renderer = renderer
        w, h = renderer.size()
        self.__cuda_array_interface__ = {"shape": (h, w, 4), "typestr": "<f4", "data": (ptr, False), "version": 3}


def prepare(case, seed):
    kind = case["kind"]
    world = seed % 100003  # the procedural scenes hash their seed in 64 bits
    s = {"kind": kind, "case": case, "stream": torch.cuda.Stream()}
    if kind in ("trace", "moving", "build"):
        s["renderer"] = r = api.Renderer(16, 16)
    if kind == "trace":
        attrs, idx = _soup_attrs(_soup(case, seed), 2)
        s["scene"] = sc = r.CreateScene()
        m = sc.AddMaterial()
        sc.AddMeshInstance(sc.AddMesh(attrs, idx, [(m, 0, len(idx))], layout=2))
        sc.Commit()
        s["rays"] = rays = _rays(case["rays"], seed, case["order"])
        if case["mem"] == "host":
            s["rays"] = rays.cpu().pin_memory()
        where = {"pin_memory": True} if case["mem"] == "host" else {"device": "cuda"}
        s["hits"] = torch.zeros((case["rays"], 4), dtype=torch.int32, **where)
        s["obj"] = torch.zeros(case["rays"], dtype=torch.int32, **where) if case["obj"] else None
    elif kind == "moving":
        rng = np.random.default_rng(seed)
        a, i = scenes.displaced_sphere(case["level"], world)
        s["scene"] = sc = r.CreateScene()
        m = sc.AddMaterial()
        mesh = sc.AddMesh(a, i, [(m, 0, len(i))])
        n = case["instances"]
        size = 0.35 / n ** (1.0 / 3.0)
        xf = np.tile(np.eye(4, dtype=np.float32), (n, 1, 1))
        ang, sc_k, pos = rng.uniform(0, 2 * np.pi, n), rng.uniform(0.5, 2.0, n) * size, rng.uniform(0, 1, (n, 3))
        xf[:, 0, 0] = xf[:, 2, 2] = np.cos(ang) * sc_k
        xf[:, 0, 2] = -np.sin(ang) * sc_k
        xf[:, 2, 0] = np.sin(ang) * sc_k
        xf[:, 1, 1] = sc_k
        xf[:, 3, 0:3] = pos
        for k in range(n):
            sc.AddMeshInstance(mesh, xf[k])
        sc.Commit()
        who = rng.choice(n, case["moved"], replace=False)
        there = xf[who].copy()
        there[:, 3, 0:3] = rng.uniform(0, 1, (case["moved"], 3))
        s["moves"] = [(int(k), there[j].reshape(-1)) for j, k in enumerate(who)]
        s["rays"] = _rays(case["rays"], seed)
        s["hits"] = torch.zeros((case["rays"], 4), dtype=torch.int32, device="cuda")
        s["obj"] = torch.zeros(case["rays"], dtype=torch.int32, device="cuda")
    elif kind == "sort":
        s["renderer"] = api.Renderer(16, 16)
        n = case["rays"]
        s["rays"] = _rays(n, seed)
        s["keys"], s["perm"] = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
        s["sorted"] = torch.zeros((n, 8), device="cuda") if case["gather"] else None
    elif kind == "build":
        s["attrs"], s["idx"] = _soup_attrs(_soup(case, seed), 0)
        s["rays"] = _rays(case["rays"], seed).cpu().numpy()
    elif kind == "render":
        w, h, b = case["w"], case["h"], case["bounces"]
        spec = (scenes.cornell_box(world, w, h, b) if case["scene"] == "cornell"
                else scenes.lightmap_box(world, w, b) if case["scene"] == "lightmap" else scenes.atrium(world, w, h, b))
        s["renderer"] = api.Renderer(w, h)
        s["scene"] = _scene(s["renderer"], spec)
    elif kind == "batch":
        specs = [_batch_spec(case["first"] + k, seed) for k in range(case["scenes"])]
        s["renderers"] = [api.Renderer(*sp["size"]) for sp in specs]
        for r in s["renderers"]:
            r.set_stream(s["stream"].cuda_stream)
        s["scenes"] = [_scene(r, sp) for r, sp in zip(s["renderers"], specs)]
    else:
        spec = scenes.diff_atrium(world, case["w"], case["h"], case["bounces"], tex_res=case["texture"])
        s["renderer"] = api.Renderer(case["w"], case["h"])
        s["scene"] = _scene(s["renderer"], spec)
        s["slots"] = spec["material_slot"]
        s["albedo"] = torch.from_numpy(spec["albedo_target"]).cuda().requires_grad_()
        s["rough"] = torch.from_numpy(spec["rough_target"]).cuda().requires_grad_()
        s["d_image"] = torch.randn((case["h"], case["w"], 3), generator=_gen(seed, 3), device="cuda") / (case["w"] * case["h"])
    return s


# ---------------------------------------------------------------- one pass


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "trace" and case["mem"] == "host":
        capi.check(capi.lib().ray_scene_trace_closest(s["scene"].handle, s["rays"].data_ptr(), case["rays"], s["hits"].data_ptr(),
                                                      s["obj"].data_ptr() if case["obj"] else None, capi.RAY_MEM_HOST,
                                                      s["stream"].cuda_stream))
        return _hits(s["hits"], s["obj"])
    if kind in ("trace", "moving"):
        if kind == "moving":
            for k, xf in s["moves"]:
                s["scene"].SetMeshInstanceTransform(k, xf)
        s["scene"].trace_closest_device(s["rays"].data_ptr(), case["rays"], s["hits"].data_ptr(),
                                        s["obj"].data_ptr() if s["obj"] is not None else 0, s["stream"].cuda_stream)
        return _hits(s["hits"], s["obj"])
    if kind == "sort":
        s["renderer"].sort_rays_device(s["rays"].data_ptr(), case["rays"], (0.0, 0.0, 0.0), (1.0 / 255.0,) * 3, s["perm"].data_ptr(),
                                       s["keys"].data_ptr(), s["sorted"].data_ptr() if case["gather"] else 0, s["stream"].cuda_stream)
        out = {"keys": s["keys"], "perm": s["perm"]}
        return dict(out, rays=s["sorted"]) if case["gather"] else out
    if kind == "build":
        sc = s["renderer"].CreateScene()
        m = sc.AddMaterial()
        sc.AddMeshInstance(sc.AddMesh(s["attrs"], s["idx"], [(m, 0, len(s["idx"]))]))
        sc.Commit()
        h = sc.trace_closest(s["rays"])
        return {"prim": h["prim"], "tuv": np.stack([h["t"], h["u"], h["v"]], axis=1)}
    if kind == "render":
        r, region = s["renderer"], api.RegionContext()
        r.Clear()
        for _ in range(case["samples"]):
            r.RenderScene(s["scene"], region)
        return r.get_pixels_ref()
    if kind == "batch":
        for r in s["renderers"]:
            r.Clear()
        api.render_batch(s["renderers"], s["scenes"], [api.RegionContext() for _ in s["renderers"]], case["samples"])
        out = []
        for r in s["renderers"]:
            p = C.c_void_p()
            capi.check(capi.lib().ray_get_pixels(r.handle, C.byref(p), 1))
            out.append(torch.as_tensor(_DevicePixels(p.value, r), device="cuda"))
        return out
    s["albedo"].grad = s["rough"].grad = None
    image = diff.render(s["albedo"], s["rough"], s["renderer"], s["scene"], s["slots"], 1, case["samples"])
    image.backward(s["d_image"])
    return {"image": image.detach(), "albedo": s["albedo"].grad, "rough": s["rough"].grad}


# ---------------------------------------------------------------- what a pass cannot do without


def _trace_work(rays, tris, out_bytes):
    """Rays read, hits written, and of the triangles (48 B) and the wide nodes
    (80 B, one for every three triangles) what the rays touch, each once; per
    ray about two and a quarter node tests per doubling of the triangle count
    (8 boxes of 15 operations) and 7 triangle tests of 40."""
    nodes = 1.4 * math.log2(max(tris, 2))
    return {"bytes": rays * (32 + out_bytes) + min(tris, 7 * rays) * 48 + min(tris / 3, nodes * rays) * 80,
            "flops": rays * (nodes * 120 + 7 * 40)}


def work(case):
    kind = case["kind"]
    if kind == "trace":
        return _trace_work(case["rays"], case["tris"], 20 if case["obj"] else 16)
    if kind == "moving":
        w = _trace_work(case["rays"], 20 * 4 ** case["level"], 20)
        return {"bytes": w["bytes"] + 96 * case["instances"], "flops": w["flops"] + case["rays"] * 30 * math.log2(case["instances"])}
    if kind == "sort":
        return {"bytes": case["rays"] * (32 + 8 + (32 if case["gather"] else 0)), "flops": case["rays"] * 24}
    if kind == "build":
        w = _trace_work(case["rays"], case["tris"], 16)
        return {"bytes": w["bytes"] + case["tris"] * (3 * 32 + 12 + 48 + 27), "flops": w["flops"] + case["tris"] * 400}
    # rays per pixel sample (closest hit and shadow), each traced and shaded (about 600 operations); the pixels read and written
    if kind == "batch":
        px = sum(int(np.prod(_batch_size(case["first"] + k))) for k in range(case["scenes"]))
        rays = 4.0
    else:
        px, rays = case["w"] * case["h"], {"cornell": 4.5, "lightmap": 4.0, "atrium": 5.8}.get(case.get("scene"), 5.0)
    n = px * case["samples"] * min(rays, 1.0 + case.get("bounces", 6))
    w = _trace_work(n, {"cornell": 1316, "lightmap": 1316}.get(case.get("scene"), 20000 if kind == "batch" else 327692), 0)
    w = {"bytes": px * 16 * case["samples"], "flops": w["flops"] + n * 600}
    if kind == "diff":
        w = {"bytes": w["bytes"] + 2 * case["texture"] ** 2 * 12, "flops": 2 * w["flops"]}
    return w


def _batch_size(index):
    """The frame size of scene `index` of the batched configuration, without its geometry (the same first draws)."""
    rng = np.random.default_rng(1000 + index)
    rng.uniform()
    res = int(rng.choice([64, 128, 256, 512, 1024]))
    return res, res


# ---------------------------------------------------------------- in 64 bits


def _exact_hits(tris, rays):
    """Closest hits in 64 bits: every ray against every triangle. t, u, v (n, 3); a miss keeps (tmax, 0, 0)."""
    v = tris.double()
    p0, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    out = torch.zeros((len(rays), 3), dtype=torch.float64, device=rays.device)
    out[:, 0] = rays[:, 3].double()
    step = max(1, 20_000_000 // max(1, len(tris)))
    for b in range(0, len(rays), step):
        o, d = rays[b:b + step, None, 0:3].double(), rays[b:b + step, None, 4:7].double()
        h = torch.linalg.cross(d.expand(-1, len(v), -1), e2[None].expand(len(d), -1, -1))
        det = (e1 * h).sum(-1)
        q = o - p0
        u = (q * h).sum(-1) / det
        h = torch.linalg.cross(q, e1[None].expand(len(d), -1, -1))
        w = (d * h).sum(-1) / det
        t = (e2 * h).sum(-1) / det
        t = torch.where((det != 0) & (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 0) & (t < out[b:b + step, 0:1]), t, math.inf)
        best, at = t.min(dim=1)
        at, hit = at[:, None], torch.isfinite(best)
        got = torch.stack([best, u.gather(1, at)[:, 0], w.gather(1, at)[:, 0]], dim=1)
        out[b:b + step] = torch.where(hit[:, None], got, out[b:b + step])
    return out


def exact(case, seed):
    if case["kind"] not in ("trace", "build") or case["tris"] * case["rays"] > 1_000_000_000:
        return None
    tuv = _exact_hits(_soup(case, seed), _rays(case["rays"], seed, case.get("order", "incoherent")))
    out = {"prim": None, "tuv": tuv}
    return dict(out, obj=None) if case.get("obj") else out
