"""What the native host path does with its callers' operands: layouts of dense weights, threads that share a stream, branches of a
captured graph, the layout of quantized results, and autograd features beside the plain backward pass."""
import threading

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


@pytest.mark.parametrize("m,k,n", [(20, 1024, 1024), (128, 2048, 1536), (333, 1001, 520)])
def test_threads_that_share_a_stream(m, k, n):
    """Layer calls of several threads on one stream, each on its own activations: a call is a quantizer and a GEMM (with a kernel for
    the divided tiles, and a copy of unaligned weights), which the threads enqueue alternately."""
    from block_linear import BlockInt8Linear
    tf = _tf()
    set_config(64)
    lin = BlockInt8Linear(k, n, bias=False, device=DEV, dtype=torch.bfloat16).eval()
    xs = [randn_bf16((m, k), seed, std=1.0 + seed).to(DEV) for seed in range(4)]
    norm = randn_bf16((k,), 9).to(DEV)
    with torch.no_grad():
        qs = [tf.quantize_block_rowwise(x) for x in xs]
        w, sw = lin._quantized_weight()
        calls = [lambda i: lin(xs[i]), lambda i: lin.infer_pre(xs[i], "rmsnorm", norm_weight=norm),
                 lambda i: tf.int8_matmul_block64_rowwise_dequantize(qs[i][0], w.t(), qs[i][1], sw)]
        want = [[call(i).clone() for call in calls] for i in range(len(xs))]
    torch.cuda.synchronize()
    bad, start = [None] * len(xs), threading.Barrier(len(xs))

    def work(i):
        wrong = 0
        start.wait()
        with torch.no_grad():
            for _ in range(20):
                outs = [[call(i) for _ in range(20)] for call in calls]
                wrong += sum(int((torch.stack(o) != r).any(dim=-1).any(dim=-1).sum()) for o, r in zip(outs, want[i]))
        bad[i] = wrong

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(xs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert bad == [0] * len(xs)
    assert_clean_device()


@pytest.mark.parametrize("m,k,n", [(24, 2048, 4096), (128, 4096, 1536), (333, 1001, 520)])
def test_branches_of_a_captured_graph(m, k, n):
    """Layer calls on two forked streams of one capture: the branches may run at the same time on every replay."""
    from block_linear import BlockInt8Linear
    set_config(64)
    lins = [BlockInt8Linear(k, n, bias=False, device=DEV, dtype=torch.bfloat16).eval() for _ in range(2)]
    xs = [[randn_bf16((m, k), 10 * b + i, std=1.0 + b).to(DEV) for i in range(4)] for b in range(2)]
    with torch.no_grad():
        want = [[lin(x).clone() for x in x_b] for lin, x_b in zip(lins, xs)]
        torch.cuda.synchronize()
        graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        outs = [[], []]
        with torch.cuda.graph(graph):
            main = torch.cuda.current_stream()
            side.wait_stream(main)
            for i in range(4):
                outs[0].append(lins[0](xs[0][i]))
                with torch.cuda.stream(side):
                    outs[1].append(lins[1](xs[1][i]))
            main.wait_stream(side)
        for _ in range(20):
            graph.replay()
            torch.cuda.synchronize()
            for got_b, want_b in zip(outs, want):
                assert all(torch.equal(g, w) for g, w in zip(got_b, want_b))
    del outs, graph
    assert_clean_device()


@pytest.mark.parametrize("m,k,n", [(1, 256, 132), (1, 16384, 260), (16, 1024, 512), (4, 4096, 777), (16, 1040, 512), (17, 512, 128)])
def test_one_launch_calls_without_scratch(m, k, n):
    """Around BI8_ONE_LAUNCH_VALUES (and where that kernel does not take the width, 777): the layer call against quantizer + GEMM."""
    tf = _tf()
    set_config(64)
    x, res, norm = randn_bf16((m, k), m + k).to(DEV), randn_bf16((m, n), 3).to(DEV), randn_bf16((k,), 4).to(DEV)
    bias = randn_bf16((n,), 6).to(DEV)
    w, sw = tf.quantize_block_rowwise(randn_bf16((n, k), n, std=0.02).to(DEV))
    for op, q in (("none", tf.quantize_block_rowwise(x)), ("rmsnorm", tf.rmsnorm_quantize_block_rowwise(x, 1e-5, norm))):
        want = tf.int8_matmul_block64_rowwise_dequantize(q[0], w.t(), q[1], sw)
        for b, r in ((None, None), (None, res), (bias, res)):
            got = tf.pre_quantize_matmul_block_rowwise_dequantize(op, x, w.t(), sw, b, norm_weight=norm, residual=r)
            full = want if b is None else want + b
            assert torch.equal(got, full if r is None else full + r)
    assert_clean_device()


@pytest.mark.parametrize("k", [73, 1001, 64])
def test_residual_and_output_that_overlap(k):
    """Overlap without being the same tensor is an error for every K (with and without aligned rows); the same tensor is updated."""
    from blockwise_int8_linear_b200._lib import Bi8Error
    tf = _tf()
    set_config(64)
    m, n = 40, 64
    x = randn_bf16((m, k), k).to(DEV)
    w, sw = tf.quantize_block_rowwise(randn_bf16((n, k), 1, std=0.02).to(DEV))
    buf = randn_bf16((m + 1, n), 2).to(DEV)
    res, out, before = buf[:m], buf[1:], buf.clone()
    with pytest.raises(Bi8Error, match="overlap"):
        tf.pre_quantize_matmul_block_rowwise_dequantize("none", x, w.t(), sw, residual=res, out=out)
    assert torch.equal(buf, before)
    want = tf.pre_quantize_matmul_block_rowwise_dequantize("none", x, w.t(), sw, residual=res.clone())
    assert tf.pre_quantize_matmul_block_rowwise_dequantize("none", x, w.t(), sw, residual=res, out=res) is not None
    assert torch.equal(buf[:m], want) and torch.equal(buf[m:], before[m:])
    assert_clean_device()


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("r,c", [(1, 1), (1, 1001), (1001, 1), (300, 1001), (257, 264), (250, 20001), (2047, 2047)])
def test_quantized_results_are_dense(r, c, dt):
    """What callers get can be viewed, saved and handed on, whatever the row length, and so can the buffers of a layer."""
    import io
    from block_linear import BlockInt8Linear
    tf = _tf()
    set_config(64, dt)
    x = randn_bf16((r, c), r + c).to(dt).to(DEV)
    q_ref, s_ref = O.quantize(x.cpu(), 64)
    qt_ref, st_ref = O.quantize(x.cpu().t().contiguous(), 64)
    row, col, dual = tf.quantize_block_rowwise(x), tf.quantize_block_colwise(x), tf.quantize_block_dual(x)
    for q, s in (row, dual[:2]):
        assert q.is_contiguous() and torch.equal(q.view(-1).cpu(), q_ref.view(-1)) and torch.equal(s.cpu(), s_ref)
    for q, s in (col, dual[2:]):
        assert q.is_contiguous() and torch.equal(q.view(-1).cpu(), qt_ref.view(-1)) and torch.equal(s.cpu(), st_ref)
    assert tf.rmsnorm_quantize_block_rowwise(x)[0].is_contiguous() and tf.silu_mul_quantize_block_rowwise(x, x)[0].is_contiguous()
    lin = BlockInt8Linear(c, r, bias=False, device=DEV, dtype=dt).eval()
    lin.weight.data = x
    with torch.no_grad():
        y = lin(x[:1])
    assert torch.equal(lin.W_int8.view(-1).cpu(), q_ref.view(-1)) and lin.W_int8.untyped_storage().nbytes() == r * c
    file = io.BytesIO()
    torch.save(lin.state_dict(), file)
    file.seek(0)
    other = BlockInt8Linear(c, r, bias=False, device=DEV, dtype=dt).eval()
    other.load_state_dict(torch.load(file))
    with torch.no_grad():
        assert torch.equal(other(x[:1]), y)
    set_config(64)


@pytest.mark.parametrize("r,c", [(4099, 1031), (1031, 4100)])
def test_large_16_bit_results_are_views_with_a_pitch(r, c):
    """From 4 M elements on rows that are not 16-byte aligned keep the pitch that the GEMM takes without a copy, as `.contiguous()`
    has them; a product of two such matrices quantized on the fly agrees with the one of their dense copies."""
    tf = _tf()
    set_config(64)
    x = randn_bf16((r, c), r).to(DEV)
    q, s = tf.quantize_block_rowwise(x)
    assert q.stride() == (-(-c // 16) * 16, 1)
    q_ref, s_ref = O.quantize(x.cpu(), 64)
    assert torch.equal(q.contiguous().view(-1).cpu(), q_ref.view(-1)) and torch.equal(s.cpu(), s_ref)
    b = randn_bf16((300, c), 3).to(DEV)
    bq, bs = tf.quantize_block_rowwise(b)
    assert bq.is_contiguous()
    want = tf.int8_matmul_block64_rowwise_dequantize(q.contiguous(), bq.t(), s, bs)
    assert torch.equal(tf.fast_matmulT(x, b), want)
    assert torch.equal(tf.int8_matmul_block64_rowwise_dequantize(q, bq.t(), s, bs), want)
    from block_linear import fast_matmul
    assert torch.equal(fast_matmul(x, b.t().contiguous()), want)
    assert torch.equal(tf.fast_matmulT(x[:1], b), tf.int8_matmul_block64_rowwise_dequantize(q[:1].contiguous(), bq.t(), s[:, :1], bs))


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 15), (5, 16), (7, 17), (33, 31), (300, 1000), (1000, 4097)])
@pytest.mark.parametrize("offset,extra", [(0, 0), (1, 0), (7, 3), (13, 9)])
def test_copy_of_rows_of_any_alignment(rows, cols, offset, extra):
    """Every byte of every row, none of what lies around the matrix, nothing written outside the copy."""
    from blockwise_int8_linear_b200 import _lib
    L, lds, ldd = _lib.lib(), cols + extra, -(-cols // 16) * 16
    g = torch.Generator(device=DEV).manual_seed(rows + cols)
    buf = torch.randint(-127, 128, (offset + rows * lds + 32,), generator=g, device=DEV, dtype=torch.int8)
    src = buf[offset:].as_strided((rows, cols), (lds, 1))
    dst = torch.full((rows * ldd + 64,), 99, device=DEV, dtype=torch.int8)
    _lib.check(L.bi8_copy_rows(_lib.ptr(src), lds, _lib.ptr(dst), ldd, rows, cols, _lib.stream_ptr()), "copy_rows")
    assert torch.equal(dst[:rows * ldd].view(rows, ldd)[:, :cols], src)
    assert bool((dst[rows * ldd:] == 99).all())


def _train_case(bias=True):
    from block_linear import BlockInt8Linear
    set_config(64)
    lin = BlockInt8Linear(208, 144, bias, device=DEV, dtype=torch.bfloat16).train()
    x = randn_bf16((2, 56, 208), 1).to(DEV).requires_grad_(True)
    return lin, x, randn_bf16((2, 56, 144), 2, outliers=0).to(DEV)


@pytest.mark.parametrize("fuse", [True, False])
@pytest.mark.parametrize("frozen", ["", "x", "w"])
def test_python_form_of_the_layer_equals_the_native_one(fuse, frozen):
    """A class derived from the autograd function runs its `forward` and `backward`: bit for bit the native passes (whose
    operands have aligned rows for every length, as these do for multiples of 16)."""
    import block_linear_config as cfg
    from block_linear import blockwise_int8_linear

    class Derived(blockwise_int8_linear):
        pass

    lin, x, g = _train_case()
    x.requires_grad_(frozen != "x")
    lin.weight.requires_grad_(frozen != "w")
    of = [t for t in (x, lin.weight, lin.bias) if t.requires_grad]
    results = []
    try:
        cfg.FUSE_DUAL_QUANTIZE = fuse
        for fn in (blockwise_int8_linear, Derived):
            y = fn.apply(x, lin.weight, lin.bias)
            results.append((y.detach(), *torch.autograd.grad(y, of, g)))
    finally:
        cfg.FUSE_DUAL_QUANTIZE = True
    *native, native_b = results[0]
    *python, python_b = results[1]
    assert all(torch.equal(a, b) for a, b in zip(native, python)) and len(native) == len(python)
    # the bias gradients are sums of bf16 values in fp32 in two orders: one rounding apart at most
    assert ((native_b.float() - python_b.float()).abs() <= 2.0 ** -7 * native_b.float().abs() + 112 * 2.0 ** -23 * g.float().abs().sum((0, 1))).all()


def test_forward_mode_differentiation_is_refused():
    import torch.autograd.forward_ad as forward_ad
    lin, x, _ = _train_case()
    with forward_ad.dual_level():
        assert lin(x).shape == (2, 56, 144)                   # nothing dual about it
        with pytest.raises(RuntimeError, match="jvp"):
            lin(forward_ad.make_dual(x.detach(), torch.ones_like(x)))
        with pytest.raises(RuntimeError, match="jvp"):
            torch.func.functional_call(lin, {"weight": forward_ad.make_dual(lin.weight.detach(), torch.ones_like(lin.weight))}, (x.detach(),))


def test_recorded_backward_pass_keeps_the_bias_gradient_differentiable():
    lin, x, _ = _train_case()
    y = lin(x)
    gx, gw, gb = torch.autograd.grad((y.float() ** 2).sum(), (x, lin.weight, lin.bias), create_graph=True)
    assert gb.requires_grad and not gx.requires_grad and not gw.requires_grad
    # d sum(gb) / d bias = 2 per row of y
    again = torch.autograd.grad(gb.float().sum(), lin.bias)[0]
    assert torch.equal(again.float(), torch.full((144,), 2.0 * 112, device=DEV))
    plain = torch.autograd.grad((lin(x).float() ** 2).sum(), lin.bias)[0]
    assert ((plain.float() - gb.detach().float()).abs() <= 2.0 ** -7 * plain.float().abs() + 1e-2).all()


@pytest.mark.parametrize("block", [32, 64, 128])
@pytest.mark.parametrize("m,k,n", [(1, 255, 64), (1, 257, 64), (8, 1001, 1000), (64, 257, 36), (65, 1001, 40), (16, 1001, 777), (40, 2049, 132),
                                   (300, 17, 5600), (2048, 65, 500), (2048, 65, 520)])
def test_dense_layers_with_unaligned_rows(m, k, n, block):
    """A layer's dense weights around the K and the outputs from which they are copied to aligned rows, widths that the decode kernel
    takes and does not take: against the oracle, plain and with a residual."""
    from block_linear import BlockInt8Linear
    set_config(block)
    lin = BlockInt8Linear(k, n, bias=True, device=DEV, dtype=torch.bfloat16).eval()
    lin.weight.data = randn_bf16((n, k), n, std=0.02).to(DEV)
    lin.bias.data = randn_bf16((n,), 2).to(DEV)
    x, res = randn_bf16((m, k), m + k, std=1.5), randn_bf16((m, n), 4)
    ref = O.linear_forward(x, lin.weight.detach().cpu(), lin.bias.detach().cpu(), block)
    with torch.no_grad():
        _close(lin(x.to(DEV)), ref)
        _close(lin.infer_pre(x.to(DEV), residual=res.to(DEV)), ref + res)
    assert lin.W_int8.is_contiguous()
    assert_clean_device()
    set_config(64)


@pytest.mark.parametrize("k", [4096, 4095])
def test_layer_call_without_seeds_has_the_workspace_of_its_plan(k):
    """BI8_GEMM_NO_SEED takes no clusters, so K is divided through a workspace: the layer's call as the two-step one, bit for bit (undivided
    sums would differ in their last bits), for weights on 16-byte rows and off them."""
    from blockwise_int8_linear_b200 import _lib
    tf = _tf()
    set_config(64, torch.float32)
    m, n = 128, 11008
    assert _lib.lib().bi8_gemm_workspace_bytes(m, n, k, 64) > 0 == _lib.lib().bi8_gemm_workspace_used(m, n, k, 64)
    x = randn_bf16((m, k), 1, std=1.5).to(DEV)
    q, s = O.quantize(randn_bf16((n, k), 2, std=0.02), 64)
    w, sw = q.to(DEV), s.to(DEV)
    xq, sx = tf.quantize_block_rowwise(x)
    two = tf.int8_matmul_block64_rowwise_dequantize(xq, w.t(), sx, sw, flags=_lib.GEMM_NO_SEED)
    assert torch.equal(tf.quantize_matmul_block_rowwise_dequantize(x, w.t(), sw, flags=_lib.GEMM_NO_SEED), two)
    assert torch.equal(tf.pre_quantize_matmul_block_rowwise_dequantize("none", x, w.t(), sw, flags=_lib.GEMM_NO_SEED), two)
    assert_clean_device()
    set_config(64)
