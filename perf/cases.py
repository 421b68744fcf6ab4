"""Workloads whose time and outputs are compared between versions of this library.

Every case is work that an application gives the library through its public
entry points: whole bakes of a scene that is already ingested (ltr_Start ..
ltrg_Wait .. ltr_GetWorkOutput), a batch of scenes, the many-lights gather
(cold start and repeated solves, host and device buffers, each precision) and
the finalize step on caller-owned device buffers. Sizes are those of the
package's own scene generators, tests and benchmark.
"""
import ctypes as C
import math
import types

import numpy as np
import torch

from lighter_gb300 import abi, library, patches, scenes
from lighter_gb300.gather import Gather
from lighter_gb300.scene import ingest, srand


def listed():
    return [
        # the smallest bake: the reference test driver's quad scene (three 128^2 lightmaps, one light),
        # what an editor re-bakes after every change; launches and host latency count
        {"name": "quads", "kind": "quads", "lm": 128},
        # Cornell room with the reference's own per-sample radiosity (one bounce) and AO
        {"name": "room_radiosity", "kind": "room", "lm": 32, "bounces": 1},
        # one small level (1.5k triangles) at an odd lightmap size: an ordinary single bake
        {"name": "small_level", "kind": "level", "lm": 213, "boxes": 40, "spheres": 4, "bounces": 0, "ao": 16,
         "patches": 0, "precision": 0, "sampled": 0, "normals": 0},
        # a middle-sized level with the sampled soft shadows, normal maps, the FP16 patch radiosity and RGBE output
        {"name": "level_sampled", "kind": "level", "lm": 384, "boxes": 200, "spheres": 25, "bounces": 2, "ao": 17,
         "patches": 4096, "precision": 1, "sampled": 1, "normals": 1},
        # the benchmark's scene: 20.8k triangles, four 1024^2 lightmaps, sphere-traced shadows, AO, FP32 patch radiosity
        {"name": "level_full", "kind": "level", "lm": 1024, "boxes": 400, "spheres": 50, "bounces": 2, "ao": 32,
         "patches": 16384, "precision": 0, "sampled": 0, "normals": 0},
        # terrain (the large workload at a quarter of its triangles): many more samples than one level
        {"name": "terrain", "kind": "terrain", "lm": 1024, "quads": 512, "rocks": 500, "points": 8, "ao": 64},
        # many small scenes baked together (ltrg_StartBatch), sizes as the batch workload draws them
        {"name": "batch", "kind": "batch", "scenes": 16},
        # form factors of a new patch set and its first solve, host arrays (loading a level)
        {"name": "gather_cold", "kind": "gather_cold", "n": 4096, "configs": 32, "bounces": 3},
        # repeated small solves from host arrays at full refinement (a lighting tool), odd sizes
        {"name": "gather_host_bf16", "kind": "gather", "n": 2999, "configs": 15, "bounces": 3, "precision": 2,
         "refine": 2, "host": 1},
        # repeated FP32 solves on device buffers
        {"name": "gather_fp32", "kind": "gather", "n": 8192, "configs": 32, "bounces": 2, "precision": 0, "refine": 0,
         "host": 0},
        # the many-lights benchmark: 32,768 patches x 64 RGB light configurations, FP16 with split right-hand side
        {"name": "gather_fp16", "kind": "gather", "n": 32768, "configs": 64, "bounces": 4, "precision": 1, "refine": 1,
         "host": 0},
        # per-frame finishing of one lightmap on device buffers
        {"name": "finalize", "kind": "finalize", "w": 512, "h": 512, "blur": 0.5},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("quads", "room", "level", "level", "level", "terrain", "batch", "gather_cold", "gather",
                       "gather", "finalize"))
    if kind == "quads":
        return {"kind": kind, "lm": _log_int(rng, 32, 512)}
    if kind == "room":
        return {"kind": kind, "lm": rng.randint(16, 48), "bounces": rng.randint(1, 3)}
    if kind == "level":
        bounces = rng.randint(0, 2)
        return {"kind": kind, "lm": _log_int(rng, 100, 900), "boxes": _log_int(rng, 20, 400),
                "spheres": rng.randint(1, 40), "bounces": bounces, "ao": rng.choice((0, 5, 16, 17, 32)),
                "patches": _log_int(rng, 500, 12000) if bounces else 0, "precision": rng.randint(0, 2),
                "sampled": rng.randint(0, 1), "normals": rng.randint(0, 1)}
    if kind == "terrain":
        return {"kind": kind, "lm": _log_int(rng, 200, 900), "quads": rng.choice((128, 256, 384)),
                "rocks": rng.randint(50, 400), "points": rng.randint(2, 8), "ao": rng.choice((17, 32, 64))}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(4, 20)}
    if kind == "gather_cold":
        return {"kind": kind, "n": _log_int(rng, 700, 6000), "configs": rng.randint(1, 40),
                "bounces": rng.randint(1, 4)}
    if kind == "gather":
        n = _log_int(rng, 1000, 20000)
        return {"kind": kind, "n": n, "configs": rng.randint(1, 64), "bounces": rng.randint(1, 4),
                "precision": rng.choice((0, 1, 1, 2)), "refine": rng.randint(0, 2), "host": rng.randint(0, 1)}
    return {"kind": kind, "w": _log_int(rng, 40, 1024), "h": _log_int(rng, 40, 1024),
            "blur": rng.choice((0.0, 0.5, 1.7, 3.0))}


# ----------------------------------------------------------------------------- inputs

def _scene_inputs(case, seed):
    """(SceneDesc, ltrg_Options) of a single-bake case."""
    kind = case["kind"]
    rng = np.random.default_rng([seed, 11])
    if kind == "quads":
        d = scenes.basic()
        light = d.lights[0]
        light.position = (float(rng.uniform(-0.6, 0.6)), float(rng.uniform(-0.6, 0.6)), float(rng.uniform(0.8, 1.4)))
        light.color = tuple(float(v) for v in rng.uniform(0.2, 1.0, 3))
        d.fixed_lm_size = (case["lm"], case["lm"])
        d.seed = seed & 0x7fffffff
        return d, {}
    if kind == "room":
        return scenes.cornell(seed & 0x7fffffff, lm=case["lm"], bounces=case["bounces"], ao=True), {}
    if kind == "level":
        d = scenes.mid(seed & 0x7fffffff, lm=case["lm"], n_boxes=case["boxes"], n_spheres=case["spheres"],
                       bounces=case["bounces"], ao_rays=case["ao"])
        opts = {"radiosity_patches": case["patches"], "radiosity_links": 1, "radiosity_precision": case["precision"],
                "shadow_mode": case["sampled"], "encode_rgbe": case["normals"]}
        if case["normals"]:
            d.config["generate_normalmap_data"] = 1
        return d, opts
    q = case["quads"]
    d = scenes.large(seed & 0x7fffffff, lm=case["lm"], grid=(q, q // 2), tiles=(2, 2), n_rocks=case["rocks"],
                     n_points=case["points"], ao_rays=case["ao"], bounces=0)
    return d, {}


def _batch_inputs(case, seed):
    """The batch workload's first levels under new lights."""
    rng = np.random.default_rng([seed, 13])
    descs = []
    for k in range(case["scenes"]):
        d = scenes.batch_scene(k)
        for light in d.lights:
            light.position = (*(float(v) for v in rng.uniform(-30, 30, 2)), float(rng.uniform(3, 10)))
            light.color = tuple(float(v) for v in rng.uniform(0.5, 1.0, 3))
        d.seed = (seed + k) & 0x7fffffff
        descs.append(d)
    return descs


class _Scenes:
    """Ingested scenes, destroyed with the object."""

    def __init__(self, descs, opts):
        self.lib = library()
        self.seed = descs[0].seed
        self.held = []
        try:
            for d in descs:
                self.held.append(ingest(self.lib, d, gpu_options=opts))
        except BaseException:
            self.close()
            raise
        self.handles = [h for h, _ in self.held]

    def close(self):
        while self.held:
            self.lib.ltr_DestroyScene(self.held.pop()[0])

    def __del__(self):
        self.close()


def _view(owner, ctype, pointer, shape):
    """An array over the scene's own output buffer, which keeps the scene alive."""
    buf = (ctype * math.prod(shape)).from_address(C.cast(pointer, C.c_void_p).value)
    buf.owner = owner
    return np.frombuffer(buf, dtype=ctype).reshape(shape)


def _outputs(held, handle):
    """The work outputs of a finished bake."""
    out = []
    lib = held.lib
    info = abi.WorkOutputInfo()
    lib.ltr_GetWorkOutputInfo(handle, C.byref(info))
    for k in range(info.lightmap_count):
        wo = abi.WorkOutput()
        if not lib.ltr_GetWorkOutput(handle, k, C.byref(wo)):
            raise RuntimeError("ltr_GetWorkOutput failed")
        out.append(_view(held, C.c_float, wo.lightmap_rgb, (wo.height, wo.width, 3)))
        if wo.normals_xyzf:
            out.append(_view(held, C.c_float, wo.normals_xyzf, (wo.height, wo.width, 4)))
        px = C.POINTER(C.c_ubyte)()
        if lib.ltrg_GetWorkOutputRGBE(handle, k, C.byref(px)):
            out.append(_view(held, C.c_ubyte, px, (wo.height, wo.width, 4)))
    return out


def _room(case, seed):
    return patches.room(seed & 0x7fffffff, case["n"], case["configs"])


def _finalize_inputs(case, seed):
    """Scattered colours of a chart atlas: a grid of covered rectangles with gaps."""
    w, h = case["w"], case["h"]
    rng = np.random.default_rng([seed, 7])
    cell = int(rng.integers(12, 40))
    mask = np.zeros((h, w), np.uint8)
    for y in range(0, h, cell):
        for x in range(0, w, cell):
            a, b = rng.integers(1, 6, 2)
            mask[y + a:y + cell - b, x + b:x + cell - a] = 1
    rgb = rng.uniform(0.0, 2.0, (h, w, 3)).astype(np.float32) * mask[:, :, None]
    return rgb, mask


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("quads", "room", "level", "terrain"):
        desc, opts = _scene_inputs(case, seed)
        return types.SimpleNamespace(kind="bake", scenes=_Scenes([desc], opts))
    if kind == "batch":
        return types.SimpleNamespace(kind="batch", scenes=_Scenes(_batch_inputs(case, seed), {}))
    if kind == "finalize":
        rgb, mask = _finalize_inputs(case, seed)
        d = torch.from_numpy(rgb).cuda()
        return types.SimpleNamespace(kind=kind, lib=library(), rgb=d, mask=torch.from_numpy(mask).cuda(),
                                     out=torch.empty_like(d), w=case["w"], h=case["h"], blur=case["blur"])
    sc = _room(case, seed)
    if kind == "gather_cold":
        return types.SimpleNamespace(kind=kind, lib=library(), sc=sc, bounces=case["bounces"])
    g = Gather(library(), sc["tri"], sc["pos"], sc["nrm"], sc["area"])
    s = types.SimpleNamespace(kind=kind, g=g, bounces=case["bounces"], precision=case["precision"],
                              refine=case["refine"], host=case["host"], albedo=sc["albedo"], emission=sc["emission"])
    if case["host"]:
        s.out = np.empty_like(sc["emission"])
    else:
        s.albedo = torch.from_numpy(sc["albedo"]).cuda()
        s.emission = torch.from_numpy(sc["emission"]).cuda()
        s.out = torch.empty_like(s.emission)
    return s


def run(s):
    if s.kind == "bake":
        lib, handle = s.scenes.lib, s.scenes.handles[0]
        srand(s.scenes.seed)
        lib.ltr_Start(handle)
        if not lib.ltrg_Wait(handle):
            raise RuntimeError("bake failed: %r" % lib.ltrg_LastError(handle))
        return _outputs(s.scenes, handle)
    if s.kind == "batch":
        lib, handles = s.scenes.lib, s.scenes.handles
        srand(s.scenes.seed)
        if not lib.ltrg_StartBatch((C.c_void_p * len(handles))(*handles), len(handles)):
            raise RuntimeError("ltrg_StartBatch rejected the batch")
        for handle in handles:
            if not lib.ltrg_Wait(handle):
                raise RuntimeError("bake failed: %r" % lib.ltrg_LastError(handle))
        return [_outputs(s.scenes, handle) for handle in handles]
    if s.kind == "gather_cold":
        with Gather(s.lib, s.sc["tri"], s.sc["pos"], s.sc["nrm"], s.sc["area"]) as g:
            return g.solve(s.sc["albedo"], s.sc["emission"], s.bounces)[0]
    if s.kind == "gather":
        if s.host:
            return s.g.solve(s.albedo, s.emission, s.bounces, s.precision, s.refine, out=s.out)[0]
        s.g.solve_device(s.albedo.data_ptr(), s.emission.data_ptr(), s.emission.shape[1], s.bounces, s.out.data_ptr(),
                         s.precision, s.refine)
        return s.out
    stream = torch.cuda.current_stream().cuda_stream
    if s.lib.ltrg_FinalizeLightmapNoAlloc(s.rgb.data_ptr(), s.mask.data_ptr(), s.out.data_ptr(), s.w, s.h, s.blur,
                                          C.c_void_p(stream)):
        raise RuntimeError("ltrg_FinalizeLightmapNoAlloc failed")
    return s.out


# ----------------------------------------------------------------------------- algorithmic work

def work(case):
    """Scene in, images out; flops of one box or triangle test (about 50) per ray, at least ten
    tests per sphere-traced shadow; one multiply-add per form factor and right-hand side."""
    kind = case["kind"]
    if kind == "finalize":
        n = case["w"] * case["h"]
        return {"bytes": n * (12 + 1 + 12), "flops": n * 6 * (2 * math.ceil(case["blur"]) + 1) * 2}
    if kind in ("gather", "gather_cold"):
        n, r = case["n"], 3 * case["configs"]
        item = 4 if case.get("precision", 1) == 0 else 2
        io = 4 * n * (2 * r + 3)
        flops = 2.0 * n * n * r * case["bounces"]
        if kind == "gather_cold":
            return {"bytes": io + item * n * n + 36 * 2 * n, "flops": flops + 25.0 * n * n}
        return {"bytes": io + item * n * n, "flops": flops}
    if kind == "batch":   # means of the generator: lightmap side 64..512, 3 lightmaps, 4.5 lights
        tex, tris, pairs, rays = 3 * 200 * 200 * case["scenes"], 2500 * case["scenes"], 4.5, 16
    else:
        maps, tris, lights = {"quads": (3, 6, 1), "room": (8, 36, 2)}.get(kind, (4, 0, 10))
        if kind == "level":
            tris = 12 * case["boxes"] + 320 * case["spheres"] + 2
        elif kind == "terrain":
            tris, lights = case["quads"] ** 2 + 80 * case["rocks"], 1 + case["points"]
        tex = maps * case["lm"] ** 2
        pairs, rays = 0.1 * lights, case.get("ao", 17 if kind == "room" else 0)
    shadow = 64 if case.get("sampled") else 10
    out = 12 + (20 if case.get("normals") else 0)
    return {"bytes": tex * out + 96 * tris, "flops": 0.6 * tex * (pairs * shadow + rays) * 50.0}


# ----------------------------------------------------------------------------- the same in 64 bits

def _exact_finalize(case, seed):
    rgb, mask = _finalize_inputs(case, seed)
    img, cur = rgb.astype(np.float64), mask.astype(bool)
    h, w = cur.shape
    for _ in range(3):
        pad = np.zeros((h + 4, w + 4), bool)
        pad[2:-2, 2:-2] = cur
        col = np.zeros((h + 4, w + 4, 3))
        col[2:-2, 2:-2] = img
        acc, cnt = np.zeros((h, w, 3)), np.zeros((h, w), int)
        for dx, dy in ((-1, 0), (1, 0), (0, -1), (0, 1)):
            def at(a, k):
                return a[2 + k * dy:2 + k * dy + h, 2 + k * dx:2 + k * dx + w]
            one, two = at(pad, 1), at(pad, 2)
            c = np.where(two[..., None], 2.0 * at(col, 1) - at(col, 2), at(col, 1))
            acc += np.where(one[..., None], c, 0.0)
            cnt += one
        new = ~cur & (cnt > 0)
        img = np.where(new[..., None], np.maximum(acc / np.maximum(cnt, 1)[..., None], 0.0), img)
        cur = cur | new
    blur = case["blur"]
    if blur:
        ext = math.ceil(blur)
        taps = np.exp(-0.5 * (np.arange(-ext, ext + 1) / blur) ** 2)
        taps /= taps.sum()
        for axis in (1, 0):
            pad = np.pad(img, [(ext, ext) if a == axis else (0, 0) for a in range(3)], mode="edge")
            n = img.shape[axis]
            img = sum(t * np.take(pad, np.arange(k, k + n), axis=axis) for k, t in enumerate(taps))
    return img


def _exact_gather(case, seed):
    """Pair factors, visibility by testing every occluder, and the Jacobi sweeps."""
    sc = _room(case, seed)
    dev = "cuda"
    P = torch.from_numpy(sc["pos"]).to(dev).double()
    N = torch.nn.functional.normalize(torch.from_numpy(sc["nrm"]).to(dev).double(), dim=1)
    area = torch.from_numpy(sc["area"]).to(dev).double()
    tri = torch.from_numpy(sc["tri"]).to(dev).double().reshape(-1, 3, 3)
    small = 0.001
    p0, u, v = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n = torch.linalg.cross(u, v)
    big = (n.abs() >= small).any(1)
    p0, u, v, n = p0[big], u[big], v[big], n[big]
    uu, uv, vv = (u * u).sum(1), (u * v).sum(1), (v * v).sum(1)
    den = uv * uv - uu * vv
    # dual edge vectors: s = w . gs, t = w . gt
    gs = (uv[:, None] * v - vv[:, None] * u) / den[:, None]
    gt = (uv[:, None] * u - uu[:, None] * v) / den[:, None]
    nd, sd, td = (n * p0).sum(1), (gs * p0).sum(1), (gt * p0).sum(1)
    count = len(P)
    G = torch.zeros((count, count), dtype=torch.float64, device=dev)
    for i in range(count - 1):
        d = P[i + 1:] - P[i]
        da, db, l2 = d @ N[i], -(d * N[i + 1:]).sum(1), (d * d).sum(1)
        f = da * db / (l2 * l2 * math.pi)
        j = torch.nonzero((da > small) & (db > small) & (f >= small)).reshape(-1)
        if not len(j):
            continue
        dn = d[j] / l2[j].sqrt()[:, None]
        a, b = P[i] + dn * small, P[i + 1 + j] - dn * small
        hit = torch.zeros(len(j), dtype=torch.bool, device=dev)
        for k in range(0, len(j), 8192):
            o, e = a[k:k + 8192], b[k:k + 8192]
            q = e - o
            slope, off = q @ n.T, nd - o @ n.T
            r = off / slope
            s = (o @ gs.T - sd) + r * (q @ gs.T)
            t = (o @ gt.T - td) + r * (q @ gt.T)
            ok = (slope.abs() >= small) & (r >= 0) & (r < 1) & (s >= 0) & (s <= 1) & (t >= 0) & (s + t <= 1)
            hit[k:k + 8192] = ok.any(1)
        j, f = j[~hit], f[j][~hit]
        G[i, i + 1 + j] = f * area[i + 1 + j]
        G[i + 1 + j, i] = f * area[i]
    E = torch.from_numpy(sc["emission"]).to(dev).double()
    alb = torch.from_numpy(sc["albedo"]).to(dev).double()[:, torch.arange(E.shape[1], device=dev) % 3]
    B = E.clone()
    for _ in range(case["bounces"]):
        B = E + G @ (alb * B)
    return B


def exact(case, seed):
    """Finalize, and gathers small enough to test every occluder; a bake's sphere traces and sample
    pushes are defined by their 32-bit steps and have no such value."""
    if case["kind"] == "finalize":
        return _exact_finalize(case, seed)
    if case["kind"] in ("gather", "gather_cold") and case["n"] <= 4096:
        return _exact_gather(case, seed)
    return None
