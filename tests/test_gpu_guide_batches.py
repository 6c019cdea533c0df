"""GPU test of the learned guide's batch selection and weight normalisation."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_guiding import _direction_samples, _stream, make_guide, set_samples

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, batch", [(1, 128), (147, 256), (149, 128), (3001, 1000), (148 * 256 * 8 + 5, 1 << 20),
                                      (148 * 256 * 8 + 5, 148 * 256 + 1)])
def test_selected_and_clamped_weights(rr, ctx, torch_cuda, n, batch):
    """Batches of one sample, of fewer than and just above one element per
    block, with the selection striding over the samples (twice, the second
    time at another offset), one load per thread and a remainder, and more
    than one round of loads per thread; one weight in fifty is an outlier
    that the clamp at 20 means cuts. Same bounds as the gradient test."""
    import mlp_ref
    torch = torch_cuda
    rng = np.random.default_rng(11)
    g = make_guide(rr, ctx, rr.GUIDE_MLP, batch=batch, max_samples=n, lr=1e-30)
    params = (rng.normal(size=mlp_ref.PARAM_COUNT) * 0.1).astype(np.float32)
    ctx.check(rr.lib().rr_guide_mlp_params(ctx.handle, g, None, None, params.ctypes.data, rr.MLP_PARAM_COUNT, None))
    pos, om, nrm, wo, w = _direction_samples(rng, n, np.array([0.3, 1.0, 0.2]))
    w[::50] *= 1e3
    keep = set_samples(rr, ctx, torch, g, pos, om, w, nrm, wo)
    p16 = torch.from_numpy(params).bfloat16().float().numpy().astype(np.float64)
    k = 0
    for i, o in mlp_ref.LAYERS:
        p16[k + o * i:k + o * i + o] = params[k + o * i:k + o * i + o]
        k += o * i + o
    b = min(n, max(batch, 128))
    for step in range(2):
        ctx.check(rr.lib().rr_guide_update(ctx.handle, g, _stream(torch)))
        grad = np.zeros(mlp_ref.PARAM_COUNT, np.float32)
        ctx.check(rr.lib().rr_guide_mlp_params(ctx.handle, g, None, grad.ctypes.data, None, rr.MLP_PARAM_COUNT, None))
        sel = (np.arange(b, dtype=np.int64) * n // b + (step * 7919) % n) % n
        F = mlp_ref.encode(pos[sel].astype(np.float64), nrm[sel], wo[sel], np.array([-1.0] * 3), np.array([1.0] * 3))
        loss, ref = mlp_ref.loss_and_grad(p16, F, om[sel].astype(np.float64), w[sel].astype(np.float64))
        cos = float(grad @ ref / (np.linalg.norm(grad) * np.linalg.norm(ref)))
        rel = float(np.linalg.norm(grad - ref) / np.linalg.norm(ref))
        assert cos > 0.99 and rel < 0.1, (step, cos, rel)
        st = rr.GuideStats()
        ctx.check(rr.lib().rr_guide_get_stats(ctx.handle, g, C.byref(st)))
        assert st.last_loss == pytest.approx(loss, rel=0.05)
    rr.lib().rr_guide_destroy(g)
