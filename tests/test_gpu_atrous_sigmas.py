"""GPU test of the A-trous filter where a sigma's square is infinite (that
term is switched off) in an image with G-buffer misses, which every form of
the filter leaves out. Single iterations against the oracle; the tolerance is
zero (a NaN may carry other bits)."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_atrous_tiles import _images

pytestmark = pytest.mark.gpu
INF, MAX = np.inf, np.finfo(np.float32).max


@pytest.mark.parametrize("tma", [1, 0])
@pytest.mark.parametrize("sig", [(INF, 0.2, 1.0), (1e20, 0.2, 1.0), (MAX, MAX, MAX), (0.25, INF, 1.0),
                                 (0.25, 0.2, INF), (1.8e19, 0.2, 1.0)])
def test_atrous_infinite_sigmas(rr, O, ctx, torch_cuda, sig, tma):
    torch = torch_cuda
    L = rr.lib()
    st = torch.cuda.current_stream().cuda_stream
    ctx.check(L.rr_atrous_set_tma(ctx.handle, tma))
    try:
        for W, H in ((33, 17), (130, 67)):
            for stride in (1, 2, 8, 64):
                for odd in (False, True):
                    rad, pos, nrm = _images(W, H, 5 * W + stride, odd)
                    ref = np.empty_like(rad)
                    O.atrous_iteration(rad, pos, nrm, ref, stride, *sig)
                    t = [torch.from_numpy(a).cuda() for a in (rad, pos, nrm)]
                    out = torch.full_like(t[0], -7.0)
                    p = rr.AtrousParams(W, H, 0, stride, *sig, 0)
                    ctx.check(L.rr_atrous_iteration(ctx.handle, *[a.data_ptr() for a in t], out.data_ptr(),
                                                    C.byref(p), st))
                    got = out.cpu().numpy()
                    same = (got.view(np.uint32) == ref.view(np.uint32)) | (np.isnan(got) & np.isnan(ref))
                    assert same.all(), (W, H, stride, odd, int((~same).any(-1).sum()))
    finally:
        ctx.check(L.rr_atrous_set_tma(ctx.handle, 1))
