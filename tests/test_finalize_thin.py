"""Thin images, which the finalize call finishes pass by pass instead of in tiles: just below and above the rule's 4M
texels of tile regions, in place and out of place, against the numpy restatement (same operations in the same order:
equal bit for bit); and their time, which must not follow the tiles' halos."""
import ctypes as C
import time

import numpy as np
import pytest

from lighter_gb300 import ext
from test_finalize_tiles import finish, make

pytestmark = pytest.mark.gpu


def call(gpu, src, mask, out, w, h, blur):
    torch = pytest.importorskip("torch")
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    return gpu.ltrg_FinalizeLightmapNoAlloc(src.data_ptr(), mask.data_ptr(), out.data_ptr(), w, h, blur, stream)


# regions of (32 + 12 + 2 ext)^2 texels: more than 4M from 2,166 tiles (blur 0), 1,981 (0.5), 726 (16) on
@pytest.mark.parametrize("w,h,blur", [(1, 69313, 0.0), (1, 69312, 0.0), (69313, 1, 0.5), (3, 63392, 0.5), (63400, 2, 0.5),
                                      (1, 23233, 16.0), (23201, 3, 16.0), (5, 23232, 16.0), (17, 25000, 16.0)])
def test_thin_images(gpu, w, h, blur):
    torch = pytest.importorskip("torch")
    for seed in (0, 1):
        rgb, mask = make(w, h, seed)
        want = finish(rgb, mask, blur)
        src, m = torch.from_numpy(rgb).cuda(), torch.from_numpy(mask).cuda()
        out = torch.full_like(src, float("nan"))
        for a, b in ((src, out), (src, src)):
            assert call(gpu, a, m, b, w, h, blur) == ext.NOALLOC_OK
            torch.cuda.synchronize()
            assert np.array_equal(b.cpu().numpy(), want)


def test_overlapping_but_not_in_place(gpu):
    """A thin image whose output begins inside its input keeps to the tiles, which read a copy."""
    torch = pytest.importorskip("torch")
    w, h, blur = 1, 40000, 16.0
    rgb, mask = make(w, h, 0)
    buf = torch.zeros(h * 3 + 30, device="cuda")
    buf[:h * 3] = torch.from_numpy(rgb).cuda().flatten()
    m = torch.from_numpy(mask).cuda()
    assert call(gpu, buf[:h * 3], m, buf[30:], w, h, blur) == ext.NOALLOC_OK
    torch.cuda.synchronize()
    assert np.array_equal(buf[30:].cpu().numpy().reshape(h, w, 3), finish(rgb, mask, blur))


def test_a_thin_image_takes_about_as_long_as_a_square_one(gpu):
    torch = pytest.importorskip("torch")
    took = []
    for w, h in ((1024, 1024), (1, 1 << 20)):
        rgb = torch.rand(w * h * 3, device="cuda")
        mask = (torch.rand(w * h, device="cuda") < 0.6).to(torch.uint8)
        out = torch.empty_like(rgb)
        best = 1e9
        for _ in range(5):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for _ in range(10):
                call(gpu, rgb, mask, out, w, h, 16.0)
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t0)
        took.append(best)
    assert took[1] < 4 * took[0], took   # in tiles: twenty times
