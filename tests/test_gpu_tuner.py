"""GPU tests of the traversal variants: the tuners where there is nothing to
choose, and the default."""
import ctypes as C

import pytest

from test_gpu_quant_trees import _outlier

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [False, True])
def test_tuner_keeps_the_variants_of_a_scene_with_one_kernel(rr, ctx, torch_cuda, batch):
    """A scene that is not quantized (alone, and in a batch with one that is)
    runs the same kernel whatever the variant: it is timed once, and what the
    context had stays, for the scenes that come after it."""
    torch = torch_cuda
    L = rr.lib()
    st = torch.cuda.current_stream().cuda_stream
    base = rr.HostScene.cornell(0).arrays
    scenes = [rr.Scene(ctx, _outlier(base, 1e7)), rr.Scene(ctx, base)]
    cam = rr.camera_data(rr.camera_desc(64, 48))
    outs = [torch.empty((2, 48, 64, 4), device="cuda") for _ in scenes]
    try:
        ctx.check(L.rr_pathtracer_set_variants(ctx.handle, 3, 6))
        if batch:
            b = rr.Batch(ctx, scenes)
            res = b.tune([cam, cam], rr.PtParams(0, 4, 2, 0), [o.data_ptr() for o in outs], st)
            b.close()
        else:
            res = rr.PtTuneResult()
            ctx.check(L.rr_pathtracer_tune(ctx.handle, scenes[0].handle, C.byref(cam), C.byref(rr.PtParams(0, 4, 2, 0)),
                                           outs[0].data_ptr(), st, C.byref(res)))
        assert (res.best_extend, res.best_shadow) == (3, 6)
        assert len(set(res.extend_ms)) == 1 and res.extend_ms[0] > 0
        assert len(set(res.shadow_ms)) == 1 and res.shadow_ms[0] > 0
    finally:
        ctx.check(L.rr_pathtracer_set_variants(ctx.handle, rr.PT_VARIANT_DEFAULT, rr.PT_VARIANT_DEFAULT))
        for s in scenes:
            s.close()


def test_contexts_walk_the_default_tree(rr, ctx, torch_cuda):
    """A new context, and the tests' shared one whatever ran before: as many
    nodes as the default variant visits, which is not what variant 0 does."""
    torch = torch_cuda
    L = rr.lib()
    st = torch.cuda.current_stream().cuda_stream
    cam = rr.camera_data(rr.camera_desc(64, 48))
    arrays = rr.HostScene.cornell(0).arrays

    def nodes(c, scene):
        out = torch.empty((2, 48, 64, 4), device="cuda")
        p, stats = rr.PtParams(0, 4, 2, rr.PT_FLAG_COUNT_TRAVERSAL), rr.PtStats()
        c.check(L.rr_pathtracer_execute(c.handle, scene.handle, C.byref(cam), C.byref(p), out.data_ptr(), st))
        c.check(L.rr_pathtracer_stats(c.handle, C.byref(stats), 1))
        return stats.extension_nodes

    counts = []
    new = rr.Context(0)
    for c in (ctx, new):
        scene = rr.Scene(c, arrays)
        counts.append(nodes(c, scene))
        for v in (rr.PT_VARIANT_DEFAULT, 0):
            c.check(L.rr_pathtracer_set_variants(c.handle, v, v))
            counts.append(nodes(c, scene))
        scene.close()
    new.close()
    assert counts[0] == counts[1] == counts[3] == counts[4]
    assert counts[2] == counts[5] != counts[1]
