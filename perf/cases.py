"""The work that programs have libkgr do, as measurable cases.

Each case is one pass through the public entry points: ray buffers traced
against a resident scene, frames of the attachments, the denoising of a
frame, the radiance-cache network's inference and training, and an animated
scene's refit.  Sizes are those of the benchmark configurations and of the
tests, with ragged ones between them.

Scenes are a program's resident assets: each is generated and uploaded once
per process.  Everything that a pass reads besides them (rays, camera, frame
number, network, deformation) comes from the seed.
"""
import ctypes
import math

import numpy as np
import torch

from artemis_gb300 import kgr

# triangles and vertices of the procedural scenes (seed 1)
SCENES = {"box4k": (4236, 12708), "terrain_s": (260096, 133921), "terrain": (1165312, 590241)}

_generated = {}
_scenes = {}


def _generate(name):
    if name not in _generated:
        _generated[name] = kgr.Generated(name, 1)
    return _generated[name]


def _scene(name, owner=""):
    """The resident scene; `owner` keeps the animated copy apart from the still one."""
    key = (name, owner)
    if key not in _scenes:
        _scenes[key] = kgr.Scene.from_generated(_generate(name))
    return _scenes[key]


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # a picking or probing tool: one small batch of rays, where the call's own latency counts
        {"name": "trace_small", "kind": "trace", "scene": "box4k", "rays": "camera", "any": False, "n": 4096},
        # second-bounce rays of a 1080p frame from a program that does its own shading
        {"name": "trace_bounce", "kind": "trace", "scene": "terrain", "rays": "bounce", "any": False, "n": 2073600},
        # shadow rays of a compacted queue: a ragged count, any hit
        {"name": "trace_shadow", "kind": "trace", "scene": "terrain_s", "rays": "shadow", "any": True, "n": 777777},
        # the headline frame: 1080p, 4 spp, depth 8, roulette from depth 3
        {"name": "pt_1080p", "kind": "pt", "scene": "terrain", "w": 1920, "h": 1080, "spp": 4, "depth": 8, "rr": True},
        # a thumbnail or the smallest served request: launches and tails count
        {"name": "pt_small", "kind": "pt", "scene": "box4k", "w": 321, "h": 243, "spp": 1, "depth": 4, "rr": False},
        # 1080p through the radiance cache (network kept as it is), one sample a pixel
        {"name": "pt_cached", "kind": "cached", "scene": "terrain", "w": 1920, "h": 1080, "spp": 1, "depth": 8,
         "dtype": "bf16"},
        # ReSTIR DI as its configuration has it: 256 x 256, 32 candidates, temporal and one spatial pass
        {"name": "restir_di", "kind": "di", "scene": "box4k", "w": 256, "h": 256, "depth": 2, "passes": 1,
         "neighbors": 5},
        # ReSTIR GI with its configuration's reuse settings
        {"name": "restir_gi", "kind": "gi", "scene": "terrain", "w": 1920, "h": 1080, "depth": 8, "iterations": 3,
         "neighbors": 8},
        # the denoiser behind a noisy 1080p frame, with every guide
        {"name": "denoise_1080p", "kind": "denoise", "scene": "terrain", "w": 1920, "h": 1080, "iterations": 5,
         "guides": 7},
        # the cache network's inference over a 1080p frame's queries
        {"name": "mlp_forward", "kind": "forward", "dtype": "bf16", "n": 2073600},
        # online training: four Adam steps on a full batch, then the weights
        {"name": "mlp_train", "kind": "train", "dtype": "fp16", "n": 65536, "steps": 4},
        # a deforming mesh: new positions, refit, and the visibility of a small view
        {"name": "refit", "kind": "refit", "scene": "terrain", "mode": "positions", "n": 65536},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _extent(rng, pixels_lo, pixels_hi):
    """A ragged extent of a common aspect ratio."""
    pixels = math.exp(rng.uniform(math.log(pixels_lo), math.log(pixels_hi)))
    aspect = rng.choice([1.0, 4 / 3, 16 / 9])
    w = max(16, int(round(math.sqrt(pixels * aspect))))
    h = max(16, int(pixels / w))
    return w, h


def draw(rng):
    kind = rng.choice(["trace", "trace", "pt", "cached", "di", "gi", "denoise", "forward", "train", "refit"])
    scene = rng.choice(sorted(SCENES))
    hd = 1920 * 1080
    if kind == "trace":
        rays = rng.choice(["camera", "bounce", "shadow"])
        return {"kind": kind, "scene": scene, "rays": rays, "any": rays == "shadow", "n": _log(rng, 1000, hd)}
    if kind == "pt":
        w, h = _extent(rng, 64 * 64, hd // 4)
        return {"kind": kind, "scene": scene, "w": w, "h": h, "spp": rng.randint(1, 4), "depth": rng.randint(1, 8),
                "rr": rng.random() < 0.5}
    if kind == "cached":
        w, h = _extent(rng, 128 * 128, hd)
        return {"kind": kind, "scene": scene, "w": w, "h": h, "spp": 1, "depth": rng.randint(2, 8),
                "dtype": rng.choice(["bf16", "fp16"])}
    if kind == "di":
        w, h = _extent(rng, 128 * 128, hd // 4)
        return {"kind": kind, "scene": scene, "w": w, "h": h, "depth": rng.randint(0, 4), "passes": rng.randint(1, 2),
                "neighbors": rng.randint(3, 8)}
    if kind == "gi":
        w, h = _extent(rng, 128 * 128, hd // 2)
        return {"kind": kind, "scene": scene, "w": w, "h": h, "depth": rng.randint(1, 8),
                "iterations": rng.randint(1, 3), "neighbors": rng.randint(3, 8)}
    if kind == "denoise":
        w, h = _extent(rng, 64 * 64, hd)
        return {"kind": kind, "scene": scene, "w": w, "h": h, "iterations": rng.randint(1, 6),
                "guides": rng.randint(1, 7)}
    if kind == "forward":
        return {"kind": kind, "dtype": rng.choice(["bf16", "fp16"]), "n": _log(rng, 1000, hd)}
    if kind == "train":
        return {"kind": kind, "dtype": rng.choice(["bf16", "fp16"]), "n": _log(rng, 2000, 65536),
                "steps": rng.randint(1, 4)}
    return {"kind": "refit", "scene": rng.choice(["box4k", "terrain_s", "terrain"]),
            "mode": rng.choice(["positions", "transforms"]), "n": _log(rng, 1000, 65536)}


# ------------------------------------------------------------------- inputs

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _view(name, aspect, seed):
    """A camera on an orbit of up to 20 degrees around the scene's own."""
    g = _generate(name)
    a = math.radians(20.0 * (np.random.default_rng(seed).random() - 0.5))
    d = g.eye.astype(np.float64) - g.target
    eye = g.target + np.array([d[0] * math.cos(a) + d[2] * math.sin(a), d[1], -d[0] * math.sin(a) + d[2] * math.cos(a)])
    return kgr.camera(eye.astype(np.float32), g.target, g.fov, aspect)


def _camera_rays(name, n, seed):
    """Jittered pinhole rays of an image of n pixels, row by row."""
    w = max(1, int(math.sqrt(n * 16 / 9)))
    h = -(-n // w)
    c = _view(name, w / h, seed).camera
    u, v, f, o = (torch.tensor(list(x), dtype=torch.float32, device="cuda") for x in (c.ax_u, c.ax_v, c.ax_w, c.center))
    i = torch.arange(n, device="cuda")
    j = torch.rand((n, 2), generator=_generator(seed), device="cuda")
    x = 2 * ((i % w).float() + j[:, 0]) / w - 1
    y = 2 * ((i // w).float() + j[:, 1]) / h - 1
    d = torch.nn.functional.normalize(x[:, None] * u + y[:, None] * v + f, dim=1)
    rays = torch.zeros((n, 8), device="cuda")
    rays[:, 0:3], rays[:, 4:7], rays[:, 7] = o, d, math.inf
    return rays


def _secondary_rays(name, n, seed, shadow):
    """Rays that leave the camera rays' hits, in pixel order: cosine-distributed bounces, or shadow rays to points
    on the scene's lights."""
    g, sc = _generate(name), _scene(name)
    first = _camera_rays(name, n, seed)
    hits = torch.zeros((n, 4), device="cuda")
    sc.trace_closest(first.data_ptr(), n, hits.data_ptr(), stream=_stream())
    rnd = _generator(seed + 1)
    found = torch.nonzero(hits[:, 0].view(torch.int32) >= 0)[:, 0]
    pick = torch.sort(torch.randint(0, len(found), (n,), generator=rnd, device="cuda"))[0]
    k = found[pick]
    d = first[k, 4:7]
    tri = torch.from_numpy(g.indices.astype(np.int64)).cuda()[hits[k, 0].view(torch.int32).long()]
    p = torch.from_numpy(g.positions).cuda()[tri]
    nrm = torch.nn.functional.normalize(torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]), dim=1)
    nrm = torch.where((nrm * d).sum(1, keepdim=True) > 0, -nrm, nrm)
    x = first[k, 0:3] + hits[k, 1:2] * d + 1e-3 * nrm
    rays = torch.zeros((n, 8), device="cuda")
    rays[:, 0:3] = x
    r = torch.rand((n, 3), generator=rnd, device="cuda")
    if shadow:
        lights = torch.from_numpy(sc.lights()).cuda()
        light = lights[(r[:, 2] * len(lights)).long().clamp(max=len(lights) - 1)]
        fold = r[:, :2].sum(1, keepdim=True) > 1
        uv = torch.where(fold, 1 - r[:, :2], r[:, :2])
        to = light[:, 0:3] + uv[:, :1] * light[:, 3:6] + uv[:, 1:] * light[:, 6:9] - x
        dist = to.norm(dim=1, keepdim=True)
        rays[:, 4:7], rays[:, 7] = to / dist, dist[:, 0] - 0.05
    else:
        phi, z = 2 * math.pi * r[:, 0], 2 * r[:, 1] - 1
        s = (1 - z * z).clamp(min=0).sqrt()
        sphere = torch.stack([s * phi.cos(), s * phi.sin(), z], dim=1)
        rays[:, 4:7] = torch.nn.functional.normalize(nrm * 1.0001 + sphere, dim=1)
        rays[:, 7] = math.inf
    return rays


def _buffers(n):
    return [torch.zeros((n, 4), device="cuda") for _ in range(4)]


def _attachment(kind, case, options):
    att = kgr.Attachment(kind)
    att.attach(case["w"], case["h"])
    for k, v in options.items():
        att.set_option(k, v)
    att.load()
    return att


def _frame_state(case, seed, att):
    w, h = case["w"], case["h"]
    return {"case": case, "att": att, "scene": _scene(case["scene"]), "cam": _view(case["scene"], w / h, seed),
            "bufs": _buffers(w * h), "frame": 16 * int(seed) % (1 << 20)}


def _features(n, seed, dtype):
    """Network inputs as the cache's queries have them: sines and cosines of positions, unit vectors, albedos."""
    g = _generator(seed)
    p = torch.rand((n, 3), generator=g, device="cuda")
    cols = [torch.sin(2.0 ** k * math.pi * p) for k in range(12)] + [torch.cos(2.0 ** k * math.pi * p) for k in range(4)]
    cols += [torch.nn.functional.normalize(torch.randn((n, 3), generator=g, device="cuda"), dim=1) for _ in range(2)]
    cols += [torch.rand((n, 5), generator=g, device="cuda"), p, torch.zeros((n, 2), device="cuda")]
    return torch.cat(cols, dim=1).to(_half(dtype)).contiguous()


def _half(dtype):
    return torch.bfloat16 if dtype == "bf16" else torch.float16


def _targets(n, seed):
    """Outgoing radiance: mostly dim, a bright tail."""
    t = torch.zeros((n, 4), device="cuda")
    t[:, :3] = torch.exp(torch.randn((n, 3), generator=_generator(seed + 7), device="cuda") - 1.5)
    return t


def prepare(case, seed):
    kind = case["kind"]
    if kind == "trace":
        n = case["n"]
        rays = (_camera_rays(case["scene"], n, seed) if case["rays"] == "camera"
                else _secondary_rays(case["scene"], n, seed, case["rays"] == "shadow"))
        out = torch.zeros(n, dtype=torch.int32, device="cuda") if case["any"] else torch.zeros((n, 4), device="cuda")
        return {"case": case, "scene": _scene(case["scene"]), "rays": rays, "out": out}
    if kind == "pt":
        opts = {"spp": case["spp"], "russian_roulette": case["rr"], "rr_start_depth": 3}
        return _frame_state(case, seed, _attachment("path_tracer", case, opts))
    if kind == "cached":
        opts = {"spp": case["spp"], "russian_roulette": True, "rr_start_depth": 3, "cache": True,
                "cache_dtype": case["dtype"], "cache_train": False}
        return _frame_state(case, seed, _attachment("path_tracer", case, opts))
    if kind == "di":
        opts = {"candidates": 32, "temporal": True, "temporal_mcap": 20, "spatial_passes": case["passes"],
                "spatial_neighbors": case["neighbors"], "spatial_radius": 30}
        return _frame_state(case, seed, _attachment("restir_di", case, opts))
    if kind == "gi":
        opts = {"candidates": 32, "gi_mcap": 30, "gi_spatial_iterations": case["iterations"],
                "gi_neighbors": case["neighbors"], "russian_roulette": True, "rr_start_depth": 3}
        return _frame_state(case, seed, _attachment("restir_gi", case, opts))
    if kind == "denoise":
        # the frame to denoise: one sample a pixel of the plain tracer, with its AOVs
        state = _frame_state(case, seed, _attachment("path_tracer", case, {"spp": 1}))
        info = kgr.launch_info(state["cam"], case["w"], case["h"], [b.data_ptr() for b in state["bufs"]], max_depth=3,
                               frame=state["frame"])
        state["att"].render(info, state["scene"], _stream())
        torch.cuda.synchronize()
        state.pop("att").close()
        state["denoiser"] = kgr.Denoiser(case["w"], case["h"], case["guides"])
        state["result"] = torch.as_tensor(_Result(state["denoiser"], case["w"] * case["h"]), device="cuda")
        return state
    if kind == "forward":
        n = case["n"]
        return {"case": case, "mlp": kgr.Mlp(case["dtype"], seed=int(seed)), "x": _features(n, seed, case["dtype"]),
                "out": torch.zeros((n, 4), device="cuda")}
    if kind == "train":
        n = case["n"]
        return {"case": case, "mlp": kgr.Mlp(case["dtype"], seed=int(seed)), "x": _features(n, seed, case["dtype"]),
                "targets": _targets(n, seed)}
    if kind == "refit":
        g, n = _generate(case["scene"]), case["n"]
        rng = np.random.default_rng(seed)
        state = {"case": case, "scene": _scene(case["scene"], "animated"), "rays": _camera_rays(case["scene"], n, seed),
                 "out": torch.zeros((n, 4), device="cuda")}
        if case["mode"] == "positions":
            # a standing wave a few triangles high
            p = torch.from_numpy(g.positions).cuda()
            phase = torch.from_numpy(rng.random(3).astype(np.float32) * 6.0).cuda()
            state["positions"] = (p + 0.01 * torch.sin(9.0 * p[:, [2, 0, 1]] + phase)).contiguous()
        else:
            a = rng.uniform(-0.2, 0.2)
            m = np.eye(4, dtype=np.float32)
            m[0, 0], m[0, 2], m[2, 0], m[2, 2] = math.cos(a), math.sin(a), -math.sin(a), math.cos(a)
            m[:3, 3] = rng.uniform(-0.1, 0.1, 3)
            state["model"] = m
        return state
    raise ValueError("unknown case: %r" % (case,))


class _Result:
    """The denoiser's own result buffer, as torch.as_tensor reads it; the tensor keeps the denoiser alive."""

    def __init__(self, denoiser, n):
        self.denoiser = denoiser
        self.__cuda_array_interface__ = {"data": (denoiser.result(), False), "shape": (n, 4), "typestr": "<f4",
                                         "version": 3}


# ------------------------------------------------------------------ one pass

def _hits(out):
    return {"prim": out[:, 0].view(torch.int32), "t": out[:, 1], "b": out[:, 2:4]}


def run(state):
    case = state["case"]
    kind, st = case["kind"], _stream()
    if kind == "trace":
        if case["any"]:
            state["scene"].trace_any(state["rays"].data_ptr(), case["n"], state["out"].data_ptr(), stream=st)
            return {"occluded": state["out"]}
        state["scene"].trace_closest(state["rays"].data_ptr(), case["n"], state["out"].data_ptr(), stream=st)
        return _hits(state["out"])
    if kind in ("pt", "cached", "di", "gi"):
        info = kgr.launch_info(state["cam"], case["w"], case["h"], [b.data_ptr() for b in state["bufs"]],
                               max_depth=case["depth"], frame=state["frame"])
        state["frame"] += 1
        state["att"].render(info, state["scene"], st)
        return dict(zip(("color", "normal", "albedo", "position"), state["bufs"]))
    if kind == "denoise":
        color, normal, albedo, position = (b.data_ptr() for b in state["bufs"])
        state["denoiser"].denoise(color, normal, albedo, position, iterations=case["iterations"], stream=st)
        return {"image": state["result"]}
    if kind == "forward":
        state["mlp"].forward(state["x"].data_ptr(), case["n"], state["out"].data_ptr(), st)
        return {"y": state["out"][:, :3]}
    if kind == "train":
        for _ in range(case["steps"]):
            state["mlp"].train_step(state["x"].data_ptr(), state["targets"].data_ptr(), case["n"], 1e-3, st)
        return {"weights": state["mlp"].weights()}
    if kind == "refit":
        sc = state["scene"]
        if case["mode"] == "positions":
            sc.refit(state["positions"].data_ptr(), stream=st)
        else:
            sc.set_transforms([0], [state["model"]], st)
        sc.trace_closest(state["rays"].data_ptr(), case["n"], state["out"].data_ptr(), stream=st)
        return _hits(state["out"])
    raise ValueError("unknown case: %r" % (case,))


# -------------------------------------------------------------------- bounds

def _ray_flops(tris):
    """A ray cannot do without the boxes of one root-to-leaf path and a leaf: two slab tests a level, four triangles."""
    return 2 * math.log2(tris) * 24 + 4 * 50


def work(case):
    kind = case["kind"]
    if kind == "forward":
        return {"bytes": case["n"] * (128 + 12) + 42e3, "flops": case["n"] * 2.0 * (5 * 64 * 64 + 64 * 3)}
    if kind == "train":
        flops = case["n"] * 3 * 2.0 * (5 * 64 * 64 + 64 * 3)
        return {"bytes": case["steps"] * (case["n"] * (128 + 12) + 24 * 20672), "flops": case["steps"] * flops}
    tris, verts = SCENES[case["scene"]]
    scene = 12 * verts + 12 * tris
    if kind in ("trace", "refit"):
        n = case["n"]
        b = n * (28 + (4 if kind == "trace" and case["any"] else 16)) + scene
        if kind == "refit":
            b += 12 * verts + 2 * 24 * tris  # the new positions, and a box for each node of a binary tree
        return {"bytes": b, "flops": n * _ray_flops(tris)}
    px = case["w"] * case["h"]
    if kind == "denoise":
        inputs = 12 + 12 + (12 if case["guides"] & 2 else 0) + (12 if case["guides"] & 4 else 0)
        return {"bytes": px * (inputs + 16), "flops": px * (case["iterations"] * 25 * 30 + 30)}
    # rays a path casts: the camera's, and a bounce and a shadow ray at each of about one and a half vertices
    rays = {"pt": 3 * case.get("spp", 1), "cached": 3 * case.get("spp", 1), "di": 3 + 2 + 6, "gi": 3 + 2 + 8}[kind]
    return {"bytes": px * 64 + scene, "flops": px * rays * _ray_flops(tris)}


# ------------------------------------------------------------- 64-bit values

def _exact_trace(case, seed):
    """Every triangle against every ray, in 64 bits."""
    if SCENES[case["scene"]][0] * case["n"] > 1 << 28:
        return None
    g, rays = _generate(case["scene"]), prepare(case, seed)["rays"].double()
    p = torch.from_numpy(g.positions).cuda().double()[torch.from_numpy(g.indices.astype(np.int64)).cuda()]
    v, e1, e2 = p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    t_all, b_all = [], []
    for part in rays.split(1024):
        o, d = part[:, None, 0:3], part[:, None, 4:7]
        s1 = torch.linalg.cross(d.expand(-1, len(v), -1), e2.expand(len(part), -1, -1))
        inv = 1 / (s1 * e1).sum(-1)
        s = o - v
        b1 = (s * s1).sum(-1) * inv
        s2 = torch.linalg.cross(s, e1.expand(len(part), -1, -1))
        b2 = (d * s2).sum(-1) * inv
        t = (e2 * s2).sum(-1) * inv
        t = torch.where((b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1) & (t > 0) & (t < part[:, 7:8]), t, math.inf)
        best, at = t.min(1)
        hit = best < math.inf
        b = torch.stack([x.gather(1, at[:, None])[:, 0] for x in (b1, b2)], dim=1)
        t_all.append(torch.where(hit, best, part[:, 7]))
        b_all.append(torch.where(hit[:, None], b, 0.0))
    return {"prim": None, "t": torch.cat(t_all), "b": torch.cat(b_all)}


def _exact_denoise(case, seed):
    """The a-trous filter of the AOV-guided denoiser, in 64 bits."""
    w, h, guides = case["w"], case["h"], case["guides"]
    bufs = prepare(case, seed)["bufs"]
    color, normal, albedo, position = (b.double().view(h, w, 4)[..., :3] for b in bufs)
    div = torch.where(albedo > float(np.float32(1e-3)), albedo, 1.0) if guides & 2 else torch.ones_like(albedo)
    lum = lambda c: c @ torch.tensor([0.2126, 0.7152, 0.0722], dtype=torch.float64, device="cuda")  # noqa: E731
    taps = [1 / 16, 1 / 4, 3 / 8, 1 / 4, 1 / 16]
    hit = (normal != 0).any(-1)
    c = color / div
    for i in range(case["iterations"]):
        step, sigma = 1 << i, 1.0 / (1 << i)
        total, weight, lp = torch.zeros_like(c), torch.zeros_like(c[..., 0]), lum(c)
        for dy in range(-2, 3):
            for dx in range(-2, 3):
                oy, ox = dy * step, dx * step
                if abs(oy) >= h or abs(ox) >= w:
                    continue
                here = (slice(max(0, -oy), h - max(0, oy)), slice(max(0, -ox), w - max(0, ox)))
                there = (slice(max(0, oy), h + min(0, oy)), slice(max(0, ox), w + min(0, ox)))
                lq = lp[there]
                k = taps[dx + 2] * taps[dy + 2] * (hit[here] == hit[there])
                k = k * torch.exp(-(lp[here] - lq).abs() / (sigma * 0.5 * (lp[here] + lq) + 1e-4))
                if guides & 1:
                    cos = (normal[here] * normal[there]).sum(-1).clamp(min=0)
                    k = torch.where(hit[here], k * cos ** 64, k)
                if guides & 4 and (dx or dy):
                    v = position[there] - position[here]
                    length = v.norm(dim=-1)
                    off = torch.where(length > 0, (normal[here] * v).sum(-1).abs() / length, 0.0)
                    k = torch.where(hit[here], k * torch.exp(-off / 0.2), k)
                total[here] += k[..., None] * c[there]
                weight[here] += k
        c = torch.where(weight[..., None] > 0, total / weight[..., None], c)
    return {"image": torch.cat([(c * div).view(-1, 3), bufs[0].double()[:, 3:]], dim=1)}


def _forward64(w, x):
    """Every layer's input, and the output, of the network in 64 bits."""
    acts = [x]
    for layer in range(5):
        acts.append((acts[-1] @ w[layer]).clamp(min=0))
    return acts, acts[-1] @ w[5][:, :3]


def exact(case, seed):
    kind = case["kind"]
    if kind == "trace" and not case["any"]:
        return _exact_trace(case, seed)
    if kind == "denoise":
        return _exact_denoise(case, seed)
    if kind == "forward":
        s = prepare(case, seed)
        w = torch.from_numpy(s["mlp"].weights()).cuda().to(_half(case["dtype"])).double()
        return {"y": torch.cat([_forward64(w, x.double())[1] for x in s["x"].split(1 << 18)])}
    if kind == "train":
        s = prepare(case, seed)
        w = torch.from_numpy(s["mlp"].weights()).cuda().double()
        m, v, n = torch.zeros_like(w), torch.zeros_like(w), case["n"]
        x, t = s["x"].double(), s["targets"].double()[:, :3]
        for step in range(1, case["steps"] + 1):
            acts, y = _forward64(w, x)
            delta = 2 * (y - t) / (y * y + 0.01) / n  # the loss's denominator is held fixed, as the relative loss has it
            grad = torch.zeros_like(w)
            grad[5, :, :3] = acts[5].T @ delta
            delta = delta @ w[5][:, :3].T * (acts[5] > 0)
            for layer in range(4, -1, -1):
                grad[layer] = acts[layer].T @ delta
                if layer:
                    delta = delta @ w[layer].T * (acts[layer] > 0)
            m, v = 0.9 * m + 0.1 * grad, 0.99 * v + 0.01 * grad * grad
            w = w - 1e-3 * (m / (1 - 0.9 ** step)) / ((v / (1 - 0.99 ** step)).sqrt() + 1e-8)
        return {"weights": w}
    return None
