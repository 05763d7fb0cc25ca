"""The wavelet calls from several threads at once, at widths whose tiles take
different amounts of shared memory in the same kernel: no launch is refused and
the results are a single thread's."""
import ctypes
import sys
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_widths_in_parallel(built_lib, cuda):
    import torch
    import shearcuda_gb300 as sc
    from shearcuda_gb300._lib import lib
    h = np.ascontiguousarray(sc.MakeONFilter('Symmlet', 4), dtype=np.float64)
    hp = h.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    g = torch.Generator(device='cuda').manual_seed(0)
    refused, wrong = [], []

    def work(x, ref, stream):
        yl, yh, out = torch.empty_like(ref[0]), torch.empty_like(ref[1]), torch.empty_like(x)
        H, W = x.shape
        torch.cuda.synchronize()
        p = [ctypes.c_void_p(t.data_ptr()) for t in (x, yl, yh, out)]
        s = ctypes.c_void_p(stream.cuda_stream)
        for k in range(5000):  # 8 rows of W (lo, hi) pairs per CTA: 49 to 106 KB
            if lib().nsst_mrdwt(p[0], 1, H, W, hp, h.size, 1, p[1], p[2], s):
                refused.append(W)
            if lib().nsst_mirdwt(p[1], p[2], 1, H, W, hp, h.size, 1, p[3], s):
                refused.append(W)
            if k % 200 == 0:
                stream.synchronize()
        stream.synchronize()
        if not (torch.equal(yl, ref[0]) and torch.equal(yh, ref[1]) and torch.equal(out, ref[2])):
            wrong.append(W)
    jobs = []
    for W in (784, 832, 1024, 1280, 1536, 1664, 1700, 900):
        x = torch.randn((2496, W), device='cuda', generator=g)
        yl, yh = sc.mrdwt_cuda(x, h, 1)
        jobs.append(threading.Thread(target=work, args=(x, (yl, yh, sc.mirdwt_cuda(yl, yh, h, 1)), torch.cuda.Stream())))
    torch.cuda.synchronize()
    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-5)
    try:
        for t in jobs:
            t.start()
        for t in jobs:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    assert not refused and not wrong, (len(refused), sorted(set(refused)), wrong)
