"""GPU test of small dense objects on wide grounds: whether a scene's trees
are quantized or not, a ray tests about as many triangles as in the
full-precision tree (a grid as wide as the ground is too coarse for the
object's boxes), and the images have the same bits."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sphere_on_ground(rr, n, ground):
    """A unit sphere of 4 n^2 triangles, less the poles', on a square of half
    width `ground`."""
    th, ph = np.meshgrid(np.linspace(0, np.pi, n + 1), np.linspace(0, 2 * np.pi, 2 * n + 1), indexing="ij")
    nrm = np.stack([np.sin(th) * np.cos(ph), np.cos(th), np.sin(th) * np.sin(ph)], -1).reshape(-1, 3)
    i, j = np.meshgrid(np.arange(n), np.arange(2 * n), indexing="ij")
    a = (i * (2 * n + 1) + j).reshape(-1)
    b = a + 2 * n + 1
    faces = np.stack([a, b, b + 1, a, b + 1, a + 1], -1).reshape(-1)
    k = len(nrm)
    v = np.zeros(k + 4, rr.VERTEX)
    v["pos"][:k], v["normal"][:k] = nrm + [0, 1, 0], nrm
    v["pos"][k:] = np.array([[-1, 0, -1], [1, 0, -1], [1, 0, 1], [-1, 0, 1]]) * ground
    v["normal"][k:, 1] = 1.0
    v["tangent"][:, 0] = 1.0
    m = np.zeros(2, rr.MESH)
    m["vertex_base"], m["vertex_count"] = [0, k], [k, 4]
    m["index_byte_offset"], m["index_count"] = [0, 4 * len(faces)], [len(faces), 6]
    mt = np.zeros(1, rr.MATERIAL)
    mt["base_color"], mt["roughness"] = 0.8, 0.6
    inst = np.zeros(2, rr.INSTANCE)
    inst["transform"] = np.eye(4, dtype=np.float32).reshape(-1)
    inst["mesh_index"] = [0, 1]
    light = np.zeros(1, rr.LIGHT)
    light["position"], light["emission"], light["intensity"] = [3, 9, 2], 1.0, 200.0
    return {"vertices": v, "indices": np.concatenate([faces, [0, 2, 1, 0, 3, 2]]).astype(np.uint32), "meshes": m,
            "materials": mt, "instances": inst, "lights": light}


@pytest.mark.parametrize("n, ground", [(60, 3.0), (60, 100.0), (60, 300.0), (150, 1e3), (150, 1e4)])
def test_dense_object_on_a_wide_ground(rr, ctx, torch_cuda, n, ground):
    """1.6 times the tests at most: the bound of the rule that refuses to
    quantize. Nodes and triangles counted."""
    torch = torch_cuda
    L = rr.lib()
    st = torch.cuda.current_stream().cuda_stream
    scene = rr.Scene(ctx, sphere_on_ground(rr, n, ground))
    cam = rr.camera_data(rr.camera_desc(97, 61, eye=(0.0, 2.0, 2.6), center=(0.0, 0.9, 0.0)))
    images, tests = [], []
    for v in (7, rr.PT_VARIANT_DEFAULT):
        ctx.check(L.rr_pathtracer_set_variants(ctx.handle, v, v))
        out = torch.empty((2, 61, 97, 4), device="cuda")
        p, s = rr.PtParams(2, 4, 2, rr.PT_FLAG_COUNT_TRAVERSAL), rr.PtStats()
        ctx.check(L.rr_pathtracer_execute(ctx.handle, scene.handle, C.byref(cam), C.byref(p), out.data_ptr(), st))
        ctx.check(L.rr_pathtracer_stats(ctx.handle, C.byref(s), 1))
        images.append(out.cpu().numpy().view(np.uint32))
        tests.append((s.extension_nodes + s.extension_tris, s.shadow_nodes + s.shadow_tris))
    scene.close()
    np.testing.assert_array_equal(images[1], images[0])
    assert tests[1][0] <= 1.6 * tests[0][0] and tests[1][1] <= 1.6 * tests[0][1], tests
