"""The surrogate's GEMMs at the edges of their tiles: widths that are no
multiple of 4, 8, 16 or 64, batches that leave partial row tiles and K chunks,
one output, one sample; against the FP64 oracle with the same roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('widths,batch', [
    ((5, 128, 128, 128, 128, 3), 1), ((5, 128, 128, 128, 128, 3), 4096), ((5, 128, 128, 3), 1003), ((3, 33, 1), 130),
    ((1, 1, 1), 7), ((7, 16, 17, 2), 64), ((4, 64, 65, 63, 5), 257), ((8, 200, 24, 4), 600), ((130, 32, 300), 90)])
def test_gradients(widths, batch):
    import torch
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from oracle import mlp_oracle as MO
    from pypercolate_gb300.surrogate import MLP
    rng = np.random.default_rng(batch)
    x, t, w = (rng.normal(size=(batch, n)).astype(np.float32) for n in (widths[0], widths[-1], widths[-1]))
    w = np.abs(w) + np.float32(0.1)
    model = MLP(widths=widths, seed=2)
    # biases that matter
    model.params.add_(torch.from_numpy(rng.normal(size=model.count).astype(np.float32)).cuda() * 0.02)
    from pypercolate_gb300 import _native as nat
    nat.check(nat.lib_handle().nz_mlp_params_to_bf16(nat.ptr(model.params), model.count, nat.ptr(model.params_bf16),
                                                     nat.stream_handle()), 'nz_mlp_params_to_bf16')
    loss = float(model.loss_and_grads(*(torch.from_numpy(a).cuda() for a in (x, t, w))))
    g = model.grads.cpu().numpy()
    b = model._buffers(batch)
    assert torch.equal(b['z'][-batch * widths[-1]:], b['y'][:batch * widths[-1]])
    loss_ref, g_ref = MO.loss_and_grads(model.params.cpu().numpy(), widths, x, t, w)
    # FP32 accumulation against FP64, and values that round to the other
    # neighbour in BF16 (2^-9 relative, a few of them): well below 5e-3 in norm
    assert abs(loss - loss_ref) <= 2e-3 * abs(loss_ref)
    assert np.linalg.norm(g - g_ref) <= 5e-3 * np.linalg.norm(g_ref)
    assert model.take_errors() == 0
