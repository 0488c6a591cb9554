"""Kernel variants at the sizes where they can go wrong: rows of any alignment, every 16-bit gate value, the cluster sizes and
tile edges of the decode GEMM with its quantization inside, and the additions behind the general GEMM."""
import pytest
import torch
import torch.nn.functional as F

from oracle import blockwise_int8_oracle as O
from tests.gpu_util import DEV, assert_clean_device, randn_bf16, set_config

pytestmark = pytest.mark.gpu


def _tf():
    import triton_functions as tf
    return tf


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("block", [32, 64, 128])
@pytest.mark.parametrize("shape,offset", [((1, 1), 0), ((3, 7), 1), ((129, 131), 0), ((257, 1001), 3), ((128, 136), 5), ((70, 4101), 0)])
def test_quantizers_take_rows_of_any_alignment(shape, offset, block, dt):
    tf = _tf()
    set_config(block, dt)
    r, c = shape
    x = randn_bf16((r, c), r + c, std=2.0).to(dt)
    if dt == torch.float32:
        x = x + torch.randn((r, c), generator=torch.Generator().manual_seed(c)) * 1e-3
    buf = torch.full((r * c + 16,), float("inf"), dtype=dt, device=DEV)         # what lies around the matrix must not be taken in
    view = buf[offset:offset + r * c].view(r, c)
    view.copy_(x)
    q_ref, s_ref = O.quantize(x, block)
    qt_ref, st_ref = O.quantize(x.t().contiguous(), block)
    for q, s in (tf.quantize_block_rowwise(view), tf.quantize_block_dual(view)[:2]):
        assert torch.equal(q.cpu(), q_ref) and torch.equal(s.cpu(), s_ref)
    for q, s in (tf.quantize_block_colwise(view), tf.quantize_block_dual(view)[2:]):
        assert torch.equal(q.cpu(), qt_ref) and torch.equal(s.cpu(), st_ref)
    q, s = tf.quantize_block_rowwise(view)
    for pitched in (q, q.contiguous()):
        assert torch.equal(tf.dequantize_block_rowwise(pitched, s).cpu(), O.dequantize(q_ref, s_ref, block, dt))
    assert_clean_device()
    set_config(64)


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_gated_activation_of_every_gate_value(dt):
    """Every finite 16-bit value as the gate: the approximate evaluation with its exact fallback is bit-identical to
    F.silu(gate) * up, quantized."""
    tf = _tf()
    set_config(64, dt)
    bits = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(dt)
    gate = torch.where(bits.isfinite(), bits, torch.zeros_like(bits)).view(256, 256).to(DEV)
    up = randn_bf16((256, 256), 3).to(dt).to(DEV)
    for u in (up, torch.ones_like(up)):
        q, s = tf.silu_mul_quantize_block_rowwise(gate, u)
        q_ref, s_ref = tf.quantize_block_rowwise(F.silu(gate) * u)
        fine = s_ref.isfinite()
        assert torch.equal(s[fine], s_ref[fine])
        assert torch.equal(q.view(256, 4, 64)[fine.t()], q_ref.view(256, 4, 64)[fine.t()])
    assert_clean_device()


@pytest.mark.parametrize("block", [32, 64, 128])
@pytest.mark.parametrize("m,k,n", [(1, 16, 4), (1, 128, 128), (7, 272, 132), (8, 1024, 4096), (9, 4096, 260), (16, 2064, 1028), (17, 528, 388),
                                   (32, 4096, 512), (2, 8192, 22016), (5, 640, 20000)])
def test_decode_layer_quantized_inside_the_gemm(m, k, n, block):
    """One launch against quantizer + GEMM: bit-identical, for clusters of 1 to 8 CTAs, one and several tiles per cluster, K that
    ends inside a block, a 128-byte step and a stage; plain, behind RMSNorm and SiLU * up, with a residual in place."""
    tf = _tf()
    set_config(block)
    x = randn_bf16((m, 2 * k), 5 * m + k, std=1.5).to(DEV)
    a, b = x[:, :k], x[:, k:]
    wq, sw = tf.quantize_block_rowwise(randn_bf16((n, k), k + n, std=0.02).to(DEV))
    norm = randn_bf16((k,), 9).to(DEV)
    res = randn_bf16((m, n), 14).to(DEV)
    steps = {"none": tf.quantize_block_rowwise(a), "rmsnorm": tf.rmsnorm_quantize_block_rowwise(a, 1e-5, norm),
             "silu_mul": tf.silu_mul_quantize_block_rowwise(a, b)}
    for op, (xq, sx) in steps.items():
        want = tf.int8_matmul_block64_rowwise_dequantize(xq, wq.t(), sx, sw)
        kw = dict(x2=b if op == "silu_mul" else None, norm_weight=norm if op == "rmsnorm" else None)
        got = tf.pre_quantize_matmul_block_rowwise_dequantize(op, a, wq.t(), sw, flags=32, **kw)
        assert torch.equal(got, want), op
        out = res.clone()
        tf.pre_quantize_matmul_block_rowwise_dequantize(op, a, wq.t(), sw, residual=out, out=out, flags=32, **kw)
        assert torch.equal(out, want + res), op
    q, s = (t.cpu() for t in steps["none"])
    ref = O.gemm(q, wq.cpu().t(), s, sw.cpu(), None, block, torch.bfloat16).float()
    got = tf.quantize_matmul_block_rowwise_dequantize(a, wq.t(), sw).cpu().float()
    assert (got - ref).abs().max().item() <= 2.0 ** -7 * ref.abs().max().item()
    assert_clean_device()
    set_config(64)


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("m,k,n", [(65, 512, 160), (129, 128, 161), (100, 2048, 777), (300, 1000, 328), (2500, 256, 1000)])
def test_bias_and_residual_behind_the_general_gemm(m, k, n, dt):
    """Whole and divided tiles, outputs with and without aligned rows, a strided residual: each addition in the output type."""
    tf = _tf()
    set_config(64, dt)
    x = randn_bf16((m, k), m + k).to(dt).to(DEV)
    wq, sw = tf.quantize_block_rowwise(randn_bf16((n, k), k + n, std=0.02).to(DEV))
    bias = randn_bf16((n,), 7).to(DEV)
    wide = randn_bf16((m, n + 3), 8).to(dt).to(DEV)
    plain = tf.quantize_matmul_block_rowwise_dequantize(x, wq.t(), sw)
    xq, sx = tf.quantize_block_rowwise(x)
    assert torch.equal(plain, tf.int8_matmul_block64_rowwise_dequantize(xq, wq.t(), sx, sw))
    # 12 * 2^-24 of the terms' absolute sum and half a step of the output type
    acc = O.gemm_acc(xq.cpu(), wq.cpu().t(), sx.cpu(), sw.cpu(), 64)
    mag = O.gemm_term_abs_sum(xq.cpu(), wq.cpu().t(), sx.cpu(), sw.cpu(), 64)
    step = {torch.bfloat16: 2.0 ** -9, torch.float16: 2.0 ** -12, torch.float32: 0.0}[dt]
    assert ((plain.cpu().float() - acc).abs() <= 12 * 2.0 ** -24 * mag + 2 * step * acc.abs() + (6e-8 if dt == torch.float16 else 0.0)).all()
    for b in (None, bias):
        base = plain if b is None else plain + b.to(dt)
        assert torch.equal(tf.quantize_matmul_block_rowwise_dequantize(x, wq.t(), sw, b), base)
        for res in (wide[:, :n].contiguous(), wide[:, :n]):
            got = tf.pre_quantize_matmul_block_rowwise_dequantize("none", x, wq.t(), sw, b, residual=res)
            assert torch.equal(got, base + res)
    assert_clean_device()
    set_config(64)


@pytest.mark.parametrize("m", [2, 20, 40, 64])
def test_decode_gemm_with_weights_arriving_late(m):
    """Weights that no cache or address translation holds yet arrive out of order: the first product with them equals the later ones."""
    tf = _tf()
    set_config(64)
    xq, sx = tf.quantize_block_rowwise(randn_bf16((m, 11008), m).to(DEV))
    gen = torch.Generator(device=DEV).manual_seed(m)
    for _ in range(12):
        wq, sw = tf.quantize_block_rowwise(torch.randn((4096, 11008), generator=gen, device=DEV, dtype=torch.bfloat16))
        torch.randn((1 << 26,), device=DEV)
        first = tf.int8_matmul_block64_rowwise_dequantize(xq, wq.t(), sx, sw)
        assert torch.equal(first, tf.int8_matmul_block64_rowwise_dequantize(xq, wq.t(), sx, sw))
    assert_clean_device()


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,n", [(1, 1), (127, 129), (128, 128), (129, 1001), (4000, 7), (2049, 520)])
def test_bias_gradient_is_the_column_sum(rows, n, dt):
    """Batches of loads and the rows behind them, columns of a last tile, rows of any alignment; the same bits each time."""
    from block_linear import BlockInt8Linear
    set_config(64, dt)
    lin = BlockInt8Linear(64, n, True, device=DEV, dtype=dt).train()
    x, g = randn_bf16((1, rows, 64), rows).to(dt).to(DEV), randn_bf16((1, rows, n), n, outliers=0).to(dt).to(DEV)
    lin(x).backward(g)
    want = g[0].double().sum(0)
    eps = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -23}[dt]
    bound = eps * want.abs() + rows * 2.0 ** -23 * g[0].double().abs().sum(0) + 1e-12
    assert ((lin.bias.grad.double() - want).abs() <= bound).all()
    first = lin.bias.grad.clone()
    lin.bias.grad = None
    lin(x).backward(g)
    assert torch.equal(first, lin.bias.grad)
    set_config(64)


@pytest.mark.parametrize("block", [32, 64, 128])
@pytest.mark.parametrize("m,k,n", [(1024, 11008, 4096), (2000, 8200, 2001), (8192, 20000, 768)])
def test_outputs_of_a_few_rounds_are_divided_over_k(m, k, n, block):
    """More tiles than half the SMs, a last range of K that is shorter, more parts than one batch of loads: against the undivided
    kernel, which is what a caller with the small built-in workspace still gets, and sampled rows against the oracle."""
    from tests.test_zz_no_alloc import _lib
    lib, L = _lib()
    gen = torch.Generator(device=DEV).manual_seed(k)
    ld, nb = (k + 15) // 16 * 16, -(-k // block)
    a, bt = (torch.randint(-127, 128, (r, ld), generator=gen, device=DEV, dtype=torch.int8)[:, :k] for r in (m, n))
    sa, sb = (torch.rand((nb, r), generator=gen, device=DEV) + 0.1 for r in (m, n))
    tf = _tf()
    set_config(block)
    assert L.bi8_gemm_workspace_bytes(m, n, k, block) > 8 << 20
    got = tf.int8_matmul_block64_rowwise_dequantize(a, bt.t(), sa, sb).float()
    c = torch.empty((m, n), dtype=torch.bfloat16, device=DEV)
    p = lib.ptr
    lib.check(L.bi8_gemm_dequant_static(p(a), ld, p(bt), ld, p(sa), p(sb), None, 0, p(c), n, 0, m, n, k, block, 0, lib.stream_ptr()), "static")
    want = c.float()
    assert ((got - want).norm() / want.norm()).item() <= 5e-3
    assert (got - want).abs().max().item() <= 2.0 ** -7 * want.abs().max().item()
    rows = torch.arange(0, m, m // 5)
    ref = O.gemm(a[rows].cpu(), bt.cpu().t(), sa[:, rows].cpu(), sb.cpu(), None, block, torch.bfloat16).float()
    assert (got[rows].cpu() - ref).abs().max().item() <= 2.0 ** -7 * ref.abs().max().item()
    assert_clean_device()
    set_config(64)


@pytest.mark.parametrize("m,k,n,divided", [(512, 768, 768, {32}), (300, 3072, 768, {32, 64, 128}), (333, 1008, 776, {32, 64}), (768, 8192, 3072, set())])
@pytest.mark.parametrize("block", [32, 64, 128])
def test_division_over_k_knows_the_block(m, k, n, divided, block):
    """A stage of block 32 takes three times one of block 128, so dividing pays earlier: which blocks divide a shape, and the result
    against the undivided kernel (no workspace; without seeds no clusters either), as far apart as two orders of an fp32 sum and another
    conversion are, and against the oracle."""
    from tests.test_zz_no_alloc import _lib
    lib, L = _lib()
    set_config(block)
    assert (L.bi8_gemm_workspace_bytes(m, n, k, block) > 0) == (block in divided)
    xq, sx = O.quantize(randn_bf16((m, k), m, std=1.5), block)
    wq, sw = O.quantize(randn_bf16((n, k), n, std=0.02), block)
    a, bt, sa, sb = (t.to(DEV) for t in (xq, wq, sx, sw))
    got = _tf().int8_matmul_block64_rowwise_dequantize(a, bt.t(), sa, sb).float()
    c = torch.empty((m, n), dtype=torch.bfloat16, device=DEV)
    p = lib.ptr
    lib.check(L.bi8_gemm_dequant(p(a), k, p(bt), k, p(sa), p(sb), None, 0, p(c), n, 0, m, n, k, block, None, 0, lib.GEMM_NO_SEED, lib.stream_ptr()), "undivided")
    rows = torch.arange(0, m, 37)
    ref = O.gemm(xq[rows], wq.t(), sx[:, rows], sw, None, block, torch.bfloat16).float()
    for want in (c.float()[rows.to(DEV)].cpu(), ref):
        assert (got[rows.to(DEV)].cpu() - want).abs().max().item() <= 2.0 ** -7 * want.abs().max().item()
    assert ((got - c.float()).norm() / c.float().norm()).item() <= 5e-3
    assert_clean_device()
    set_config(64)


@pytest.mark.parametrize("flags", [2, 2 | 4])
@pytest.mark.parametrize("m,k,n,block", [(300, 3072, 768, 64), (128, 4096, 4096, 32), (96, 5120, 640, 128), (1000, 40960, 1600, 64)])
def test_smaller_workspace_takes_a_smaller_plan(m, k, n, block, flags):
    """What a call's plan needs, a byte less, two parts, a byte less, none: divided through whatever workspace holds a plan that pays (few
    tiles without clusters: two parts), written only there, and within the tolerance of the oracle on sampled rows."""
    from blockwise_int8_linear_b200 import _lib as lib
    L = lib.lib()
    need = L.bi8_gemm_workspace_bytes(m, n, k, block)
    tiles = -(-m // 128) * -(-n // 160)
    part = tiles * min(128, -(-m // 32) * 32) * 160 * 4
    assert need >= 3 * part, "the plan has three parts or more"
    gen = torch.Generator(device=DEV).manual_seed(k)
    nb = -(-k // block)
    a, bt = (torch.randint(-127, 128, (r, k), generator=gen, device=DEV, dtype=torch.int8) for r in (m, n))
    sa, sb = (torch.rand((nb, r), generator=gen, device=DEV) + 0.1 for r in (m, n))
    rows = torch.tensor([0, 31, m // 2, m - 1])
    host = (a[rows].cpu(), bt.cpu().t(), sa[:, rows].cpu(), sb.cpu(), block)
    acc, mag = O.gemm_acc(*host), O.gemm_term_abs_sum(*host)
    p = lib.ptr
    few = tiles * 2 <= torch.cuda.get_device_properties(0).multi_processor_count
    for given in (need, need - 1, 2 * part, 2 * part - 1, 0):
        ws = torch.full((need + 4096,), 0x5A, dtype=torch.uint8, device=DEV)
        c = torch.empty((m, n), dtype=torch.float32, device=DEV)
        lib.check(L.bi8_gemm_dequant(p(a), k, p(bt), k, p(sa), p(sb), None, 0, p(c), n, lib.BI8_F32, m, n, k, block, p(ws), given, flags,
                                     lib.stream_ptr()), "bi8_gemm_dequant")
        written = bool((ws[:given] != 0x5A).any())
        assert bool((ws[given:] == 0x5A).all())
        if given >= need - 1 or given < 2 * part or (few and flags & lib.GEMM_NO_SEED):
            assert written == (given >= 2 * part)
        assert bool(((c[rows].cpu() - acc).abs() <= 12 * 2.0 ** -24 * mag).all())
    assert_clean_device()


@pytest.mark.parametrize("block", [32, 64, 128])
@pytest.mark.parametrize("m,k,n", [(33, 512, 12288), (64, 4096, 12288), (40, 768, 2304), (64, 2048, 264)])
def test_either_side_of_the_choice_at_33_to_64_rows(m, k, n, block):
    """Where the line between the decode and the general kernel depends on the block: both, and the choice, against the oracle."""
    tf = _tf()
    set_config(block)
    xq, sx = O.quantize(randn_bf16((m, k), m, std=1.5), block)
    wq, sw = O.quantize(randn_bf16((n, k), n, std=0.02), block)
    ref = O.gemm(xq, wq.t(), sx, sw, None, block, torch.bfloat16).float()
    a, b, sa, sb = xq.to(DEV), wq.to(DEV).t(), sx.to(DEV), sw.to(DEV)
    outs = [tf.int8_matmul_block64_rowwise_dequantize(a, b, sa, sb, flags=f) for f in (0, 2, 16)]
    for got in outs:
        assert (got.cpu().float() - ref).abs().max().item() <= 2.0 ** -7 * ref.abs().max().item()
    assert torch.equal(outs[0], outs[1]) or torch.equal(outs[0], outs[2])
    assert_clean_device()
    set_config(64)
