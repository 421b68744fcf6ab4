"""The one-pass finalize (finalize.cuh) at the edges of its 32 x 32 tiles: sizes around one and two tiles, single
rows and columns, every halo class of the blur, in place and out of place, against a plain numpy restatement of the
sweeps and convolutions (lighter.cpp:880-961) in FP32 with the same order of operations. Every operation is an
IEEE + - * / in that order, so the results are equal bit for bit."""
import ctypes as C
import math

import numpy as np
import pytest

from lighter_gb300 import ext, scenes
from lighter_gb300.scene import bake

f32 = np.float32
_libm = C.CDLL("libm.so.6")
for _n, _a in (("expf", 1), ("powf", 2)):
    getattr(_libm, _n).restype = C.c_float
    getattr(_libm, _n).argtypes = [C.c_float] * _a


def taps_of(blur):
    e = math.ceil(blur)
    mc = f32(1.0) / np.sqrt(f32(2.0) * f32(3.14159265358979323846) * f32(blur) * f32(blur), dtype=f32)
    k = [f32(_libm.expf(f32(-0.5) * f32(_libm.powf(f32(i) / f32(blur), f32(2.0))))) * mc for i in range(-e, e + 1)]
    total = f32(0)
    for v in k:
        total = f32(total + v)
    return e, [f32(v / total) for v in k]


def finish(rgb, mask, blur):
    img, cur = rgb.astype(f32).copy(), mask.astype(bool)
    h, w = cur.shape
    for _ in range(3):
        pm = np.pad(cur, 2)
        pc = np.pad(img, ((2, 2), (2, 2), (0, 0)))
        acc, cnt = np.zeros((h, w, 3), f32), np.zeros((h, w), np.int32)
        for dx, dy in ((-1, 0), (1, 0), (0, -1), (0, 1)):
            def at(a, k):
                return a[2 + k * dy:2 + k * dy + h, 2 + k * dx:2 + k * dx + w]
            c = np.where(at(pm, 2)[..., None], at(pc, 2) * f32(-1.0) + at(pc, 1) * f32(2.0), at(pc, 1))
            acc = np.where(at(pm, 1)[..., None], acc + c, acc)
            cnt += at(pm, 1)
        new = ~cur & (cnt > 0)
        v = acc / np.maximum(cnt, 1)[..., None].astype(f32)
        img = np.where(new[..., None], np.where(v > 0, v, f32(0)), img)
        cur = cur | new
    if blur:
        e, k = taps_of(blur)
        for axis in (1, 0):
            n = img.shape[axis]
            out = np.zeros_like(img)
            for i in range(-e, e + 1):
                out = out + np.take(img, np.clip(np.arange(n) + i, 0, n - 1), axis=axis) * k[i + e]
            img = out
    return img


def make(w, h, seed):
    rng = np.random.default_rng([w, h, seed])
    mask = (rng.random((h, w)) < rng.choice([0.02, 0.4, 0.9])).astype(np.uint8)
    rgb = rng.uniform(0, 3, (h, w, 3)).astype(f32)
    return (rgb * mask[..., None] if seed else rgb), mask


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(1, 1), (1, 70), (70, 1), (31, 33), (32, 32), (33, 31), (64, 65), (97, 40), (250, 129)])
@pytest.mark.parametrize("blur", [0.0, 0.5, 1.0, 2.5, 16.0])
def test_finalize_tile_edges(gpu, w, h, blur):
    torch = pytest.importorskip("torch")
    for seed in (0, 1, 2):
        rgb, mask = make(w, h, seed)
        want = finish(rgb, mask, blur)
        src, m = torch.from_numpy(rgb).cuda(), torch.from_numpy(mask).cuda()
        out = torch.full_like(src, float("nan"))
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        for a, b in ((src, out), (src, src)):   # apart, then in place
            assert gpu.ltrg_FinalizeLightmapNoAlloc(a.data_ptr(), m.data_ptr(), b.data_ptr(), w, h, blur,
                                                    stream) == ext.NOALLOC_OK
            torch.cuda.synchronize()
            assert np.array_equal(b.cpu().numpy(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("size,blur", [((33, 50), 0.5), ((64, 31), 0.0), ((40, 95), 17.0)])
def test_bake_finalize(gpu, size, blur):
    """The bake's lightmaps from its own sample colours; blur 17 takes the separate convolutions."""
    d = scenes.cornell(5, lm=32, bounces=0, ao=True)
    d.fixed_lm_size = size
    d.config["blur_size"] = blur
    res = bake(gpu, d)
    for uid, _, _, lm, _ in res.lightmaps:
        h, w, _ = lm.shape
        rgb, mask = np.zeros((h * w, 3), f32), np.zeros(h * w, np.uint8)
        rgb[res.debug[uid]["loc"]] = res.debug[uid]["color"]
        mask[res.debug[uid]["loc"]] = 1
        assert np.array_equal(lm, finish(rgb.reshape(h, w, 3), mask.reshape(h, w), blur))
