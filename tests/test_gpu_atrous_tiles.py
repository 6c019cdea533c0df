"""GPU test of the A-trous lattice tiles: single iterations against the oracle
at the sizes where a tile, its halo or its dispatch can go wrong. The
tolerance is zero (the packed operations round as the scalar ones do); a NaN
may carry other bits."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _images(W, H, seed, odd_values):
    g = np.random.default_rng(seed)
    rad = g.gamma(0.7, 1.5, (H, W, 4)).astype(np.float32)
    pos = g.normal(size=(H, W, 4)).astype(np.float32) * 0.3
    pos[..., 3] = np.where(g.random((H, W)) < 0.15, -1.0, 2.0)      # misses
    nrm = np.zeros((H, W, 4), np.float32)
    nrm[..., :3] = g.normal(size=(H, W, 3)) * 0.3 + np.array([0, 1, 0])
    if odd_values:
        k = g.integers(0, H * W, (6, max(1, H * W // 40)))
        f = lambda a: a.reshape(-1, 4)
        f(rad)[k[0], 0] = np.inf
        f(rad)[k[1], 1] = np.nan
        f(rad)[k[2], :3] = 0.0
        f(pos)[k[3], 0] = 1e20
        f(pos)[k[4], 1] = np.inf
        f(nrm)[k[5], :3] = 0.0
    return rad, pos, nrm


@pytest.mark.parametrize("tma", [1, 0])
@pytest.mark.parametrize("W,H", [(1, 1), (5, 200), (31, 15), (33, 17), (64, 32), (130, 67)])
def test_atrous_tiles_bit_exact(rr, O, ctx, torch_cuda, W, H, tma):
    """Sizes around the 32 x 16 tile; strides on both sides of the dispatch,
    odd ones (rr_atrous_iteration takes any) and zero; sigmas whose squares
    are clamped, ordinary, or outside the range of the reciprocal division;
    values that are not finite."""
    torch = torch_cuda
    L = rr.lib()
    st = torch.cuda.current_stream().cuda_stream
    ctx.check(L.rr_atrous_set_tma(ctx.handle, tma))
    try:
        for stride in (0, 1, 2, 3, 8, 16, 64, 2000):
            for sig, odd in (((0.25, 0.20, 1.0), False), ((1e-5, 0.7, 30.0), False), ((3e6, 0.2, 1e19), False),
                             ((0.25, 0.20, 1.0), True)):
                rad, pos, nrm = _images(W, H, 7 * W + stride, odd)
                ref = np.empty_like(rad)
                O.atrous_iteration(rad, pos, nrm, ref, stride, *sig)
                t = [torch.from_numpy(a).cuda() for a in (rad, pos, nrm)]
                out = torch.full_like(t[0], -7.0)
                p = rr.AtrousParams(W, H, 0, stride, *sig, 0)
                ctx.check(L.rr_atrous_iteration(ctx.handle, *[a.data_ptr() for a in t], out.data_ptr(), C.byref(p),
                                                st))
                got = out.cpu().numpy()
                same = (got.view(np.uint32) == ref.view(np.uint32)) | (np.isnan(got) & np.isnan(ref))
                assert same.all(), (stride, sig, odd, np.argwhere(~same)[:4], got[~same][:4], ref[~same][:4])
    finally:
        ctx.check(L.rr_atrous_set_tma(ctx.handle, 1))
