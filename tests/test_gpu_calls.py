"""What the native host path does with its callers' operands: layouts of dense weights, threads that share a stream, branches of a
captured graph, the layout of quantized results, and autograd features beside the plain backward pass."""
import pytest
import torch

from oracle import blockwise_int8_oracle as O
from tests.gpu_util import DEV, assert_clean_device, randn_bf16, set_config

pytestmark = pytest.mark.gpu


def _tf():
    import triton_functions as tf
    return tf


def _close(got, ref):
    """bf16 results of the same terms in another order of the fp32 sum: one rounding apart."""
    got, ref = got.cpu().float(), ref.float()
    assert ((got - ref).norm() / ref.norm()).item() <= 5e-3
    assert (got - ref).abs().max().item() <= 2.0 ** -7 * ref.abs().max().item()


@pytest.mark.parametrize("m,k,n", [(333, 1000, 1000), (260, 257, 257), (333, 1000, 999), (64, 264, 264)])
def test_dense_weights_of_unaligned_rows(m, k, n):
    """Dense [N, K] int8 weights of the caller's own whose rows are not 16-byte aligned, square ones among them (whose shape does
    not tell the matrix from its transpose), through every function that takes `W.t()`; a square dense [K, N] `b` as well."""
    tf = _tf()
    set_config(64)
    x = randn_bf16((m, k), m + k, std=1.5).to(DEV)
    q, s = O.quantize(randn_bf16((n, k), k + n, std=0.02), 64)
    w, sw = q.to(DEV), s.to(DEV)
    assert w.is_contiguous()
    xq, sx = O.quantize(x.cpu(), 64)
    a, sa = xq.to(DEV), sx.to(DEV)
    ref = O.gemm(xq, q.t(), sx, s, None, 64, torch.bfloat16)
    res = randn_bf16((m, n), 5).to(DEV)
    for b in (w.t(), w.t().contiguous()):
        _close(tf.int8_matmul_block64_rowwise_dequantize(a, b, sa, sw), ref)
        _close(tf.quantize_matmul_block_rowwise_dequantize(x, b, sw), ref)
        _close(tf.pre_quantize_matmul_block_rowwise_dequantize("none", x, b, sw, residual=res), ref + res.cpu())
        parts = tf.int8_matmul_block_partials(a, b, 64).cpu()
        for j in range(parts.shape[0]):
            cols = slice(64 * j, min(k, 64 * (j + 1)))
            assert torch.equal(parts[j].double(), xq[:, cols].double() @ q[:, cols].double().t())
    assert_clean_device()
