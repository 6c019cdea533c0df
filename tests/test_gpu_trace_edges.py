"""GPU test of ray queries that reach every child slot of a node, the unused
ones of the 4-wide tree included: rays that are not numbers, and rays without
an end towards the point at 1e30 where unused slots lie. Both trees answer
alike, and visit no node twice."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("any_hit", [0, 1])
@pytest.mark.parametrize("triangles", [36, 20_000])
def test_rays_that_meet_unused_slots(rr, ctx, torch_cuda, triangles, any_hit):
    torch = torch_cuda
    L = rr.lib()
    st = torch.cuda.current_stream().cuda_stream
    hs = rr.HostScene.cornell(0) if triangles == 36 else rr.HostScene.procedural(target_triangles=triangles)
    scene = rr.Scene(ctx, hs.arrays)
    nan, inf = np.nan, np.inf
    far = 1.0 / np.sqrt(3.0)
    rays = [((nan, nan, nan), (0, 1, 0)), ((nan, 0, 0), (0, 1, 0)), ((0, 0, 0), (nan, nan, nan)),
            ((0, 0, 0), (0, nan, 1)), ((30, 30, 30), (far, far, far)), ((30, 30, 30), (1, 1, 1)),
            ((0, 0, 0), (far, far, far)), ((0, 0, 0), (0, -1, 0))] * 5
    o = torch.tensor([r[0] + (0,) for r in rays], dtype=torch.float32, device="cuda")
    d = torch.tensor([r[1] + (0,) for r in rays], dtype=torch.float32, device="cuda")
    n = len(rays)
    got = []
    for wide in (0, rr.TRACE_WIDE):
        hits = torch.empty((n, 4), device="cuda")
        prims, work = (torch.empty(s, dtype=torch.int32, device="cuda") for s in ((n,), (n, 2)))
        flags = wide | (rr.TRACE_ANY_HIT if any_hit else 0)
        ctx.check(L.rr_trace_counted(ctx.handle, scene.handle, o.data_ptr(), d.data_ptr(), 1e-3, inf, n, flags,
                                     hits.data_ptr(), prims.data_ptr(), work.data_ptr(), st))
        stats = rr.SceneStats()
        ctx.check(L.rr_scene_get_stats(scene.handle, stats))
        assert int(work[:, 0].max()) <= (stats.bvh4_node_count if wide else stats.bvh_node_count)
        got.append((hits.cpu().numpy(), prims.cpu().numpy()))
    hit = got[0][0][:, 0] >= 0
    np.testing.assert_array_equal(got[1][0][:, 0] >= 0, hit)
    assert not hit[:6].any() and hit[7]
    if not any_hit:
        np.testing.assert_array_equal(got[0][0].view(np.uint32), got[1][0].view(np.uint32))
        np.testing.assert_array_equal(got[0][1][hit], got[1][1][hit])
    scene.close()
