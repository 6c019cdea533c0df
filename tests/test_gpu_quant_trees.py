"""GPU tests of the queue traversal over the quantized trees, at the scenes
where its grid and its dispatch can go wrong. The tolerance is zero: a box
only decides which triangles are tested, so the images are the oracle's bits
whichever tree is walked (variant 7 walks the full-precision one)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scaled(arrays, scale, shift):
    """The arrays with every instance scaled per axis, then moved."""
    a = {k: v.copy() for k, v in arrays.items()}
    for inst in a["instances"]:
        m = inst["transform"].reshape(4, 4)
        m[:3] = np.asarray(scale, np.float32)[:, None] * m[:3]
        m[:3, 3] += np.asarray(shift, np.float32)
    a["lights"]["position"] = a["lights"]["position"] * np.asarray(scale, np.float32) + np.asarray(shift, np.float32)
    return a


def _one_mesh(arrays, keep):
    """Only the first `keep` triangles of the first instance's mesh: one leaf for a few."""
    a = {k: v.copy() for k, v in arrays.items()}
    a["instances"] = a["instances"][:1]
    m = int(a["instances"]["mesh_index"][0])
    a["meshes"]["index_count"][m] = 3 * keep
    return a


def _outlier(arrays, distance):
    """One instance more, far away: the grid's step grows with the distance."""
    a = {k: v.copy() for k, v in arrays.items()}
    far = a["instances"][:1].copy()
    far[0]["transform"].reshape(4, 4)[:3, 3] += np.float32(distance)
    a["instances"] = np.concatenate([a["instances"], far])
    return a


CASES = {
    "cornell": lambda c: (c, (1, 1, 1), (0, 0, 0)),
    "root_is_a_leaf": lambda c: (_one_mesh(c, 1), (1, 1, 1), (0, 0, 0)),
    "two_coplanar_triangles": lambda c: (_one_mesh(c, 2), (1, 1, 1), (0, 0, 0)),
    "large_coordinates": lambda c: (_scaled(c, (1, 1, 1), (3e4, -2e4, 5e4)), (1, 1, 1), (3e4, -2e4, 5e4)),
    "tiny": lambda c: (_scaled(c, (1e-3, 1e-3, 1e-3), (0, 0, 0)), (1e-3, 1e-3, 1e-3), (0, 0, 0)),
    "anisotropic": lambda c: (_scaled(c, (50, 0.02, 1), (0, 0, 0)), (50, 0.02, 1), (0, 0, 0)),
    "outlier_near": lambda c: (_outlier(c, 30.0), (1, 1, 1), (0, 0, 0)),
    "outlier_far": lambda c: (_outlier(c, 1e7), (1, 1, 1), (0, 0, 0)),
}


@pytest.mark.parametrize("name", list(CASES))
def test_quantized_traversal_bit_exact(rr, O, ctx, torch_cuda, name):
    torch = torch_cuda
    base = rr.HostScene.cornell(0).arrays
    arrays, scale, shift = CASES[name](base)
    scene = rr.Scene(ctx, arrays)
    oscene = O.OracleScene(arrays, use_bvh=False)
    s, t = np.asarray(scale, np.float64), np.asarray(shift, np.float64)
    # an odd image, and an axis-parallel view: zero direction components
    cam = rr.camera_data(rr.camera_desc(45, 31, eye=tuple(np.array([0.0, 1.0, 3.2]) * s + t),
                                        center=tuple(np.array([0.0, 1.0, 0.0]) * s + t)))
    ref, _ = O.pathtrace(oscene, cam, 5, 4, 2)
    st = torch.cuda.current_stream().cuda_stream
    L = rr.lib()
    try:
        for v in range(rr.PT_VARIANT_COUNT):
            ctx.check(L.rr_pathtracer_set_variants(ctx.handle, v, v))
            for flags in (0, rr.PT_FLAG_COUNT_TRAVERSAL):
                out = torch.empty((2, 31, 45, 4), device="cuda")
                p = rr.PtParams(5, 4, 2, flags)
                ctx.check(L.rr_pathtracer_execute(ctx.handle, scene.handle, C.byref(cam), C.byref(p), out.data_ptr(),
                                                  st))
                got = out.cpu().numpy()
                np.testing.assert_array_equal(got.view(np.uint32), ref.view(np.uint32), err_msg=f"variant {v}")
            stats = rr.PtStats()
            ctx.check(L.rr_pathtracer_stats(ctx.handle, C.byref(stats), 1))
            assert stats.extension_nodes >= stats.extension_rays   # every ray visits the root
    finally:
        ctx.check(L.rr_pathtracer_set_variants(ctx.handle, 0, 0))
        scene.close()


def test_reuse_passes_same_bits_on_both_trees(rr, ctx, torch_cuda):
    """ReSTIR DI, GI and PT over a scene whose trees are quantized and over
    the same scene with an instance so far away that they are not (it is last,
    so the others keep their ids): every image has the same bits. Two frames,
    an odd image (partial warps at its edges), both forms of the initial
    passes, DI with and without emitter candidates."""
    from research_b200 import passes
    torch = torch_cuda
    base = rr.HostScene.cornell(0).arrays
    W, H = 61, 37
    L = rr.lib()
    got = []
    try:
        for arrays in (base, _outlier(base, 1e7)):
            scene = rr.Scene(ctx, arrays)
            images = []
            for wavefront in (1, 0):
                ctx.check(L.rr_reuse_set_wavefront(ctx.handle, wavefront))
                di = passes.ReSTIRDIPass(ctx, (W, H))
                others = [passes.ReSTIRGIPass(ctx, (W, H)), passes.ReSTIRPTPass(ctx, (W, H))]
                for k in range(2):
                    eye = (0.1 * k, 1.0, 3.2)
                    cam = rr.camera_data(rr.camera_desc(W, H, eye=eye, center=(0.0, 1.0, 0.0)),
                                         rr.camera_desc(W, H, eye=(0.0, 1.0, 3.2), center=(0.0, 1.0, 0.0)))
                    di.execute(scene, cam)
                    images += [di.gbuf_pos.clone(), di.gbuf_norm.clone(), di.output.clone()]
                    for p in others:
                        p.execute(scene, cam, di.gbuf_pos, di.gbuf_norm, di.output)
                        images.append(p.output.clone())
                z = [torch.zeros((H, W, 4), device="cuda") for _ in range(5)]
                prm = rr.DIParams(3, 16, 1, 1, 4, 15, 20, rr.DI_FLAG_EMITTERS)
                ctx.check(L.rr_restir_di_execute(ctx.handle, scene.handle, C.byref(cam), C.byref(prm),
                                                 *[t.data_ptr() for t in z], torch.cuda.current_stream().cuda_stream))
                images.append(z[4].clone())
            got.append([i.cpu().numpy().view(np.uint32) for i in images])
            scene.close()
    finally:
        ctx.check(L.rr_reuse_set_wavefront(ctx.handle, 1))
    assert got[0][2].any()
    for k, (a, b) in enumerate(zip(*got)):
        np.testing.assert_array_equal(a, b, err_msg=f"image {k}")


def test_visibility_at_the_far_bound_matches_the_full_tree(rr, ctx, torch_cuda):
    """Shadow rays that meet a surface at their far bound, within a rounding:
    from the floor straight up to samples on the ceiling and on the light
    below it (the ray starts a bias above the floor and ends a bias before the
    sample). Which of them count as blocked follows the full-precision tree's
    rule, so ReSTIR GI's shading agrees with rr_trace_counted ray by ray."""
    torch = torch_cuda
    L = rr.lib()
    st = torch.cuda.current_stream().cuda_stream
    scene = rr.Scene(ctx, rr.HostScene.cornell(0).arrays)
    W = H = 256
    g = torch.Generator(device="cuda").manual_seed(7)
    r = lambda: torch.rand((H, W), device="cuda", generator=g)
    img = lambda *c: torch.stack(list(c), -1).contiguous()
    one, zero = torch.ones((H, W), device="cuda"), torch.zeros((H, W), device="cuda")
    px, pz = (r() - 0.5) * 1.6, (r() - 0.5) * 1.6
    # up to a tenth of the height off the vertical
    tx, tz = px + (r() - 0.5) * 0.1 * r(), pz + (r() - 0.5) * 0.1 * r()
    ty = torch.where((tx.abs() < 0.25) & (tz.abs() < 0.25), torch.tensor(0.999, device="cuda"), one)
    # the floor's material index: any non-emissive one
    mats = rr.HostScene.cornell(0).arrays["materials"]
    mat = int(np.nonzero(mats["emissive"].max(1) == 0)[0][0])
    bits = torch.full((H, W), mat, dtype=torch.int32, device="cuda").view(torch.float32)
    gpos, gnrm = img(px, zero, pz, one), img(zero, one, zero, bits)
    m1 = torch.full((H, W), 1, dtype=torch.int32, device="cuda").view(torch.float32)
    res = [img(tx, ty, tz, one), img(one, one, one, one), img(zero, -one, zero, m1)]
    spare = [torch.zeros((H, W, 4), device="cuda") for _ in range(8)]
    im = rr.GiReuseImages()
    im.gbuf_pos, im.gbuf_norm, im.direct = gpos.data_ptr(), gnrm.data_ptr(), None
    for k in range(3):
        im.reservoir_curr[k], im.reservoir_prev[k] = res[k].data_ptr(), spare[k].data_ptr()
    for k in range(2):
        im.history_curr[k], im.history_prev[k] = spare[3 + k].data_ptr(), spare[5 + k].data_ptr()
    im.output = spare[7].data_ptr()
    bias = 1e-3
    p = rr.gi_reuse_params(1, 8, 0, 0, 0, 12, 0, 1.0, bias)
    cam = rr.camera_data(rr.camera_desc(W, H, eye=(0.0, 0.5, 3.2), center=(0.0, 0.5, 0.0)))
    ctx.check(L.rr_restir_gi_spatial_shade(ctx.handle, scene.handle, C.byref(cam), C.byref(p), C.byref(im), st))
    lit = spare[7][..., :3].amax(-1) > 0
    # the same rays, operation by operation
    dx, dy, dz = tx - px, ty - zero, tz - pz
    xx, yy, zz = dx * dx, dy * dy, dz * dz
    dist = ((xx + yy) + zz).sqrt()
    b = torch.tensor(bias, device="cuda")
    origins = img(px + zero * b, zero + one * b, pz + zero * b, zero).view(-1, 4)
    dirs = img(dx / dist, dy / dist, dz / dist, zero).view(-1, 4)
    tmax = (dist - b).view(-1)
    n = W * H
    hits, prims = torch.empty((n, 4), device="cuda"), torch.empty(n, device="cuda", dtype=torch.int32)
    work = torch.empty((n, 2), device="cuda", dtype=torch.int32)
    blocked = torch.zeros(n, dtype=torch.bool, device="cuda")
    # rr_trace_counted takes one tmax a call: one call per distinct value near the bound, so group by value
    order = tmax.argsort()
    values, counts = torch.unique_consecutive(tmax[order], return_counts=True)
    first = 0
    for v, c in list(zip(values.tolist(), counts.tolist()))[:4000]:
        o, d = origins[order[first:first + c]].contiguous(), dirs[order[first:first + c]].contiguous()
        ctx.check(L.rr_trace_counted(ctx.handle, scene.handle, o.data_ptr(), d.data_ptr(), bias, v, c, rr.TRACE_ANY_HIT,
                                     hits.data_ptr(), prims.data_ptr(), work.data_ptr(), st))
        blocked[order[first:first + c]] = hits[:c, 0] >= 0
        first += c
    done = order[:first]
    got = lit.view(-1)[done]
    want = ~blocked[done]
    assert first > 1000 and 0 < int(want.sum()) < first
    assert int((got != want).sum()) == 0
    scene.close()
