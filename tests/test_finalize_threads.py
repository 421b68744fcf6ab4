"""Finalize calls of several host threads with halos of different sizes: scenes of a batch, and the entry point on
caller-owned buffers (one stream, so the calls follow each other on the GPU while their host sides overlap). Every call
succeeds with the bits of the same call alone."""
import ctypes as C
import threading

import numpy as np
import pytest

from lighter_gb300 import ext, scenes
from lighter_gb300.scene import bake, bake_batch

pytestmark = pytest.mark.gpu
BLURS = (2.5, 5.0, 16.0, 0.5)


def test_batch_of_different_blurs(gpu):
    descs = []
    for k in range(12):
        d = scenes.cornell(5, lm=32, bounces=0, ao=False)
        d.config["blur_size"] = BLURS[k % len(BLURS)]
        descs.append(d)
    alone = [bake(gpu, d, debug=False) for d in descs[:len(BLURS)]]
    for _ in range(6):
        for k, res in enumerate(bake_batch(gpu, descs)[0]):
            for a, b in zip(res.lightmaps, alone[k % len(BLURS)].lightmaps):
                assert np.array_equal(a[3], b[3])


def test_threads_of_different_blurs(gpu):
    torch = pytest.importorskip("torch")
    w = h = 40
    gen = torch.Generator().manual_seed(3)
    rgb = torch.rand(h * w * 3, generator=gen).cuda()
    mask = (torch.rand(h * w, generator=gen) < 0.5).to(torch.uint8).cuda()
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    outs = [torch.empty_like(rgb) for _ in BLURS]
    want = []
    for blur, out in zip(BLURS, outs):
        assert gpu.ltrg_FinalizeLightmapNoAlloc(rgb.data_ptr(), mask.data_ptr(), out.data_ptr(), w, h, blur,
                                                stream) == ext.NOALLOC_OK
        torch.cuda.synchronize()
        want.append(out.clone())
        out.fill_(float("nan"))
    torch.cuda.synchronize()
    codes = [[] for _ in BLURS]
    start = threading.Barrier(len(BLURS))

    def work(k):
        start.wait()
        for _ in range(4000):   # ctypes releases the interpreter lock during the call
            codes[k].append(gpu.ltrg_FinalizeLightmapNoAlloc(rgb.data_ptr(), mask.data_ptr(), outs[k].data_ptr(), w, h,
                                                             BLURS[k], stream))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(BLURS))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for k in range(len(BLURS)):
        assert set(codes[k]) == {ext.NOALLOC_OK}, (BLURS[k], sum(c != ext.NOALLOC_OK for c in codes[k]))
        assert torch.equal(outs[k], want[k])
