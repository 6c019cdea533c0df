"""GPU tests of rays whose hits the quantized boxes do not decide, in scenes
where many are: any-hit rays that meet a surface within a rounding of their
far bound, and rays that leave triangles so large that the triangle test's
rounding reaches the near bound. The queue traversal lists them per warp and
traces them in the full-precision tree. The tolerance is zero: the queues'
images are those of variant 7, which walks that tree alone, and the reuse
passes' are those of their per-pixel form, which keeps no list."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def floor_and_ceiling(rr, height, light_y, intensity, tess=16, emissive=0.0):
    """Two tessellated squares, `height` apart and as wide each way, lit by a
    point light at light_y, or by the ceiling's own emission."""
    g = np.linspace(-height, height, tess + 1, dtype=np.float32)
    x, z = np.meshgrid(g, g, indexing="ij")
    n = (tess + 1) ** 2
    v = np.zeros(2 * n, rr.VERTEX)
    for k, y in enumerate((0.0, height)):
        v["pos"][k * n:(k + 1) * n] = np.stack([x, np.full_like(x, y), z], -1).reshape(-1, 3)
        v["normal"][k * n:(k + 1) * n, 1] = 1.0 - 2.0 * k
    v["tangent"][:, 0] = 1.0
    i, j = np.meshgrid(np.arange(tess), np.arange(tess), indexing="ij")
    a = (i * (tess + 1) + j).reshape(-1)
    quads = np.stack([a, a + tess + 1, a + tess + 2, a, a + tess + 2, a + 1], -1).reshape(-1)
    idx = np.tile(quads, 2).astype(np.uint32)
    m = np.zeros(2, rr.MESH)
    m["vertex_base"], m["vertex_count"] = [0, n], n
    m["index_byte_offset"], m["index_count"] = [0, 4 * len(quads)], len(quads)
    m["material_index"] = [0, 1]
    mt = np.zeros(2, rr.MATERIAL)
    mt["base_color"][:] = 0.8
    mt["roughness"] = 1.0
    mt["emissive"][1] = emissive
    inst = np.zeros(2, rr.INSTANCE)
    inst["transform"] = np.eye(4, dtype=np.float32).reshape(-1)
    inst["mesh_index"] = [0, 1]
    lights = np.zeros(0 if emissive else 1, rr.LIGHT)
    if not emissive:
        lights["position"] = [0.013 * height, light_y, -0.021 * height]
        lights["emission"] = 1.0
        lights["intensity"] = intensity
    return {"vertices": v, "indices": idx, "meshes": m, "materials": mt, "instances": inst, "lights": lights}


# A light 0.01 behind a ceiling 300 up: shadow rays end 0.01 before a light,
# at the ceiling. And a ceiling so far away that 0.01 is lost in the distance,
# with a light on it, or emitting itself (the floor's triangles are 4e4 wide:
# three in a hundred of the rays that leave it hit it again at 1e-3, if
# nothing but their grown boxes keeps them from it).
SCENES = {
    "behind": lambda rr: floor_and_ceiling(rr, 300.0, np.float32(300.01), 1e5),
    "on": lambda rr: floor_and_ceiling(rr, 3e5, 3e5, 1e11),
    "emitting": lambda rr: floor_and_ceiling(rr, 3e5, 0.0, 0.0, emissive=5.0),
}


def _view(rr, height, W, H):
    return rr.camera_data(rr.camera_desc(W, H, eye=(0.0, height / 3, 0.0), center=(0.01 * height, 0.0, 0.02 * height)))


def _height(name):
    return 300.0 if name == "behind" else 3e5


@pytest.mark.parametrize("name", list(SCENES))
def test_shadow_rays_at_their_bound(rr, ctx, torch_cuda, name):
    """Some 160 shadow rays for each resident warp, and 1100 shadow and second
    extension rays in the emitting scene: lists fill, and the rest of the queue
    goes to the loop after them."""
    torch = torch_cuda
    L = rr.lib()
    st = torch.cuda.current_stream().cuda_stream
    scene = rr.Scene(ctx, SCENES[name](rr))
    W, H = 511, 385
    bounces, spp, mode = (2, 28, rr.PT_FLAG_EMITTERS) if name == "emitting" else (1, 4, 0)
    cam = _view(rr, _height(name), W, H)

    def render(variant, flags):
        ctx.check(L.rr_pathtracer_set_variants(ctx.handle, variant, variant))
        out = torch.empty((spp, H, W, 4), device="cuda")
        p = rr.PtParams(3, bounces, spp, flags | mode)
        ctx.check(L.rr_pathtracer_execute(ctx.handle, scene.handle, C.byref(cam), C.byref(p), out.data_ptr(), st))
        return out

    try:
        ref = render(7, 0)
        if name != "behind":
            lit = int((ref[..., :3].amax(-1) > 0).sum())
            assert 0 < lit < ref[..., 0].numel()
        for v in range(rr.PT_VARIANT_COUNT):
            for flags in (0, rr.PT_FLAG_COUNT_TRAVERSAL):
                bad = int((render(v, flags).view(torch.int32) != ref.view(torch.int32)).any(-1).sum())
                assert bad == 0, f"variant {v}, flags {flags}: {bad} paths differ"
    finally:
        ctx.check(L.rr_pathtracer_set_variants(ctx.handle, 4, 4))
        scene.close()


def test_batch_shadow_rays_at_their_bound(rr, ctx, torch_cuda):
    torch = torch_cuda
    L = rr.lib()
    st = torch.cuda.current_stream().cuda_stream
    names = ("behind", "on", "behind", "on")
    scenes = [rr.Scene(ctx, SCENES[n](rr)) for n in names]
    cams = [_view(rr, _height(n), 300 + 7 * k, 221) for k, n in enumerate(names)]
    b = rr.Batch(ctx, scenes)
    b.set_mode(rr.BATCH_WAVEFRONT)
    try:
        images = []
        for v in (4, 0, 7):
            ctx.check(L.rr_pathtracer_set_variants(ctx.handle, v, v))
            outs = [torch.empty((4, c.screen_height, c.screen_width, 4), device="cuda") for c in cams]
            b.execute(cams, rr.PtParams(3, 1, 4, 0), [o.data_ptr() for o in outs], st)
            images.append([o.cpu().numpy().view(np.uint32) for o in outs])
    finally:
        ctx.check(L.rr_pathtracer_set_variants(ctx.handle, 4, 4))
        b.close()
        for s in scenes:
            s.close()
    for got in images[:2]:
        for k, (a, ref) in enumerate(zip(got, images[2])):
            np.testing.assert_array_equal(a, ref, err_msg=f"scene {k}")


@pytest.mark.parametrize("reuse", ["gi", "pt"])
def test_reuse_shadow_rays_at_their_bound(rr, ctx, torch_cuda, reuse):
    """From points on the far ceiling down to the floor, and from there to the
    light on the ceiling."""
    from research_b200 import passes
    torch = torch_cuda
    L = rr.lib()
    W, H, height = 700, 500, 3e5
    scene = rr.Scene(ctx, SCENES["on"](rr))
    g = torch.Generator(device="cuda").manual_seed(5)
    one, zero = torch.ones((H, W), device="cuda"), torch.zeros((H, W), device="cuda")
    x, z = ((torch.rand((H, W), device="cuda", generator=g) - 0.5) * height for _ in range(2))
    bits = torch.zeros((H, W), dtype=torch.int32, device="cuda").view(torch.float32)
    gpos = torch.stack([x, one * height, z, one], -1).contiguous()
    gnrm = torch.stack([zero, -one, zero, bits], -1).contiguous()
    cam = rr.camera_data(rr.camera_desc(W, H, eye=(0.0, height / 3, 0.0), center=(0.01 * height, height, 0.0)))
    got = []
    try:
        for wavefront in (1, 0):
            ctx.check(L.rr_reuse_set_wavefront(ctx.handle, wavefront))
            p = (passes.ReSTIRGIPass if reuse == "gi" else passes.ReSTIRPTPass)(ctx, (W, H))
            p.guiding_enable, p.max_bounces = False, 1
            p.execute(scene, cam, gpos, gnrm, torch.zeros((H, W, 4), device="cuda"))
            got.append([t.cpu().numpy().view(np.uint32) for r in p.reservoirs for t in r] + [p.output.cpu().numpy().view(np.uint32)])
    finally:
        ctx.check(L.rr_reuse_set_wavefront(ctx.handle, 1))
        scene.close()
    assert got[0][-1].reshape(-1, 4)[:, 0].any()
    for k, (a, b) in enumerate(zip(*got)):
        np.testing.assert_array_equal(a, b, err_msg=f"image {k}")


def test_inline_rays_that_leave_large_triangles(rr, ctx, torch_cuda):
    """ReSTIR DI's camera rays (traced in lanes) from just above the floor up
    to the far ceiling: the same hits as in the scene with one instance more,
    so far away that its trees are not quantized."""
    torch = torch_cuda
    L = rr.lib()
    st = torch.cuda.current_stream().cuda_stream
    W, H, height = 300, 200, 3e5
    eye = (-0.943 * height, 1e-4, -0.4416 * height)
    cam = rr.camera_data(rr.camera_desc(W, H, eye=eye, center=(-0.6 * height, height, -0.3 * height)))
    arrays = SCENES["on"](rr)
    far = arrays["instances"][:1].copy()
    far[0]["transform"].reshape(4, 4)[:3, 3] += np.float32(1e13)
    got = []
    for a in (arrays, {**arrays, "instances": np.concatenate([arrays["instances"], far])}):
        scene = rr.Scene(ctx, a)
        z = [torch.zeros((H, W, 4), device="cuda") for _ in range(5)]
        p = rr.DIParams(1, 4, 0, 0, 4, 15, 20, 0)
        ctx.check(L.rr_restir_di_execute(ctx.handle, scene.handle, C.byref(cam), C.byref(p),
                                         *[t.data_ptr() for t in z], st))
        got.append([t.cpu().numpy() for t in z[:2]])
        scene.close()
    assert (got[1][0][..., 3] > 1e4).mean() > 0.9
    for a, b in zip(*got):
        np.testing.assert_array_equal(a.view(np.uint32), b.view(np.uint32))
