"""Accuracy of the surrogate's long sums: weight and bias gradients over large
batches of values of one sign, against 64 bits of the same BF16 operands."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('K,N', [(128, 128), (5, 128), (64, 40), (128, 3)])
def test_gradients_over_65536_samples(K, N):
    """The tensor cores' FP32 accumulation rounds toward zero.  A slice of 4,096
    samples in two accumulators is 128 steps of 16 samples each: of the final sum
    0.5 x 2^-23 x 128 / 2 = 3.8e-6 on average (half a last place of a running sum
    that is half the final one on average).  Bias gradients: one rounding of the
    slices' and one of the final sum, at most 2^-24 each, 2^-24 on average."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from pypercolate_gb300 import _native as nat
    B = 65536
    gen = torch.Generator(device='cuda')
    gen.manual_seed(K + N)
    x, dy = (torch.rand(B, n, device='cuda', generator=gen) + 0.5 for n in (K, N))
    weights = torch.zeros(K * N + N, dtype=torch.bfloat16, device='cuda')
    grads, z = torch.zeros(K * N + N, device='cuda'), torch.zeros(B * N, device='cuda')
    scratch = torch.zeros(2 * B * max(K, N), device='cuda')
    widths = np.array([K, N], dtype=np.int32)
    nat.check(nat.lib_handle().nz_mlp_backward(
        widths.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), 1, B, nat.ptr(x), nat.ptr(weights), nat.ptr(z), nat.ptr(z),
        nat.ptr(dy), nat.ptr(grads), nat.ptr(scratch), nat.stream_handle()), 'nz_mlp_backward')
    want = x.bfloat16().double().T @ dy.bfloat16().double()
    assert float((grads[:K * N].double().view(K, N) / want - 1).abs().mean()) < 3.8e-6
    assert float((grads[K * N:].double() / dy.double().sum(0) - 1).abs().mean()) < 2.0 ** -24


@pytest.mark.parametrize('B', [100, 4096, 65536])
@pytest.mark.parametrize('value', [float('inf'), -float('inf'), float('nan'), 3e38])
def test_gradients_of_no_finite_sum(B, value):
    """Two infinite (or not a number, or together out of FP32's range) gradients of one
    output: its bias and positive inputs' weights get the sum that FP32 has, other
    outputs' are not touched."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from pypercolate_gb300 import _native as nat
    K, N = 64, 40
    x, dy = torch.ones(B, K, device='cuda'), torch.ones(B, N, device='cuda')
    dy[3, 5] = dy[B - 2, 5] = value
    weights = torch.zeros(K * N + N, dtype=torch.bfloat16, device='cuda')
    grads, z = torch.zeros(K * N + N, device='cuda'), torch.zeros(B * N, device='cuda')
    scratch = torch.zeros(2 * B * max(K, N), device='cuda')
    widths = np.array([K, N], dtype=np.int32)
    nat.check(nat.lib_handle().nz_mlp_backward(
        widths.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), 1, B, nat.ptr(x), nat.ptr(weights), nat.ptr(z), nat.ptr(z),
        nat.ptr(dy), nat.ptr(grads), nat.ptr(scratch), nat.stream_handle()), 'nz_mlp_backward')
    rows = grads.view(K + 1, N)
    want = torch.full((K + 1, N), float(B), device='cuda')
    want[:, 5] = torch.tensor(value, device='cuda') + torch.tensor(value, device='cuda')
    assert torch.equal(rows.isnan(), want.isnan())
    assert torch.equal(rows.nan_to_num(7.0, 1.0, 2.0), want.nan_to_num(7.0, 1.0, 2.0))
