"""GPU tests of the ray queues' slots at image sizes that do not fill their
8 x 4 tiles or blocks of 256: one path, one tile, one pixel past a tile in
each direction, one row of tiles past a block, and several samples. Bit-exact
against the oracle, with the oracle's ray counts."""
import ctypes as C

import numpy as np
import pytest

import test_gpu_restir_gi as gi
import test_gpu_restir_pt as pt
from test_gpu_parity import cam_for, gpu_pathtrace

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W, H, spp", [(1, 1, 1), (8, 4, 1), (9, 5, 3), (257, 3, 2), (7, 261, 1)])
def test_pathtracer_ragged_tiles(rr, O, ctx, torch_cuda, W, H, spp):
    hs = rr.HostScene.cornell(0)
    scene, oscene = rr.Scene(ctx, hs.arrays), O.OracleScene(hs.arrays)
    cam = cam_for(rr, "cornell", W, H)
    st = rr.PtStats()
    ctx.check(rr.lib().rr_pathtracer_stats(ctx.handle, C.byref(st), 1))
    g = gpu_pathtrace(rr, ctx, scene, cam, torch_cuda, 2, 4, spp)
    ctx.check(rr.lib().rr_pathtracer_stats(ctx.handle, C.byref(st), 1))
    o, (rays, shadow_rays) = O.pathtrace(oscene, cam, 2, 4, spp)
    np.testing.assert_array_equal(g.view(np.uint32), o.view(np.uint32))
    assert (st.extension_rays, st.shadow_rays) == (rays, shadow_rays)


@pytest.mark.parametrize("W, H", [(1, 1), (9, 5), (65, 5)])
@pytest.mark.parametrize("reuse", [gi, pt], ids=["gi", "pt"])
def test_reuse_ragged_tiles(rr, O, ctx, torch_cuda, reuse, W, H):
    hs = rr.HostScene.cornell(0)
    reuse._run(rr, O, ctx, torch_cuda, hs.arrays, W, H, 2, (0.0, 0.0, 3.0), (0.0, 0.0, 0.0), (0.002, 0.0, -0.01))
