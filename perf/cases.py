"""The work that a program using this framework has it do, as cases that can be timed and compared.

A case is a dict of plain values.  ``kind`` says which path it takes, always through the public modules:

  linear        ``BlockInt8Linear`` in eval mode: quantize the activations, block GEMM with fused dequantize, bias
  mlp           the MLP half of a transformer layer in inference: RMSNorm -> gate/up -> SiLU * up -> down -> residual sum,
                the elementwise steps inside the layer's own calls (``BlockInt8Linear.infer_pre``)
  decode_layer  one new token per sequence through everything of a transformer layer that this framework does: RMSNorm and
                q/k/v projection, rotary embedding with the append to the key/value caches, output projection with its
                residual sum, then the MLP half.  The attention call between them is not the framework's; its result
                stands ready among the inputs
  train         ``BlockInt8Linear`` in train mode, forward and backward: y, dX, dW and, with a bias, dbias
  matmul        ``fast_matmulT``: both operands quantized on the fly (the reference's own K = 512 benchmark)
  round_trip    block quantize and block dequantize of a matrix, as for storing and restoring weights

Sizes: M tokens (or sequences), K and N the features in and out; for mlp and decode_layer, K the hidden and N the
intermediate size.  Sizes are those of the Llama-7B and GPT-2 small projections in the examples, of the reference's sweep, and
generic ones.  ``block`` is the quantisation block, ``dtype`` that of activations, weights and results.
"""
import math

import torch

import block_linear_config
from block_linear import BlockInt8Linear
from blockwise_int8_linear_b200.decode_ops import rope_cache_append
from triton_functions import dequantize_block_rowwise, fast_matmulT, quantize_block_rowwise

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
SIZE = {"bf16": 2, "fp16": 2, "fp32": 4}
HEAD_DIM, CACHE_ROWS = 128, 256


def _case(name, kind, M, K, N, block=64, dtype="bf16", bias=False):
    return {"name": name, "kind": kind, "M": M, "K": K, "N": N, "block": block, "dtype": dtype, "bias": bias}


def listed():
    return [
        # generating text for one user: one token through an attention projection; latency is all
        _case("token_projection", "linear", 1, 4096, 4096),
        # a decode step of a small serving batch, one layer of it
        _case("decode_layer_batch8", "decode_layer", 8, 4096, 11008),
        # a decode step of a large serving batch, or a short prompt
        _case("linear_m128", "linear", 128, 4096, 11008),
        # prompts being read in (prefill) with the elementwise steps inside the calls, at the default block of 128
        _case("prefill_mlp", "mlp", 2048, 4096, 11008, block=128),
        # the benchmark workload of the repository: a long prefill through the up projection
        _case("prefill_m8192", "linear", 8192, 4096, 11008),
        # a model whose sizes nobody rounded: unaligned rows in and out, half precision, bias
        _case("ragged_fp16", "linear", 333, 1000, 777, dtype="fp16", bias=True),
        # a small encoder kept in single precision outside its GEMMs
        _case("encoder_fp32", "linear", 512, 768, 2304, block=128, dtype="fp32", bias=True),
        # training GPT-2 small: the widening MLP projection of 8 x 1024 tokens
        _case("train_mlp", "train", 8192, 768, 3072, bias=True),
        # training GPT-2 small: the head over the 50257 words of its vocabulary
        _case("train_lm_head", "train", 8192, 768, 50257),
        # fine-tuning a small layer in single precision on a ragged batch
        _case("train_small_fp32", "train", 300, 256, 384, block=32, dtype="fp32", bias=True),
        # a product of two plain matrices, at a size of the reference's sweep
        _case("matmul_k512", "matmul", 4096, 512, 4096),
        # storing a weight matrix as int8 and restoring it
        _case("weight_round_trip", "round_trip", 11008, 4096, 0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _features(rng, lo, hi, ragged):
    n = _log(rng, lo, hi)
    return n if ragged else max(lo, n // 64 * 64)


def draw(rng):
    """One more case of the same ranges: any number of tokens from one up, feature sizes from 256 to 11008 (to a vocabulary's
    width in training), a quarter of them ragged, every block size and type; never more arithmetic than the largest of its kind."""
    kind = rng.choice(["linear", "linear", "linear", "mlp", "decode_layer", "train", "train", "matmul", "round_trip"])
    block = rng.choice([64, 64, 64, 128, 128, 32])
    dtype = rng.choice(["bf16", "bf16", "bf16", "bf16", "fp16", "fp32"])
    ragged, bias = rng.random() < 0.25, rng.random() < 0.4
    if kind == "linear":
        most = 8192 * 4096 * 11008
        M, K, N = _log(rng, 1, 8192), _features(rng, 256, 11008, ragged), _features(rng, 256, 11008, ragged)
    elif kind == "mlp":
        most, bias = 2048 * 4096 * 11008, False
        M, K, N = _log(rng, 1, 4096), _features(rng, 256, 4096, ragged), _features(rng, 512, 11008, ragged)
    elif kind == "decode_layer":
        most, bias = 64 * 4096 * 11008, False
        dtype = "fp16" if dtype == "fp32" else dtype
        M, K, N = _log(rng, 1, 64), HEAD_DIM * rng.randint(4, 32), _features(rng, 1024, 11008, False)
    elif kind == "train":
        most = 8192 * 768 * 50257
        M, K, N = _log(rng, 64, 8192), _features(rng, 256, 4096, ragged), _features(rng, 256, 50257, ragged)
    elif kind == "matmul":
        most, bias = 8192 * 1024 * 8192, False
        M, K, N = _log(rng, 128, 8192), _features(rng, 256, 1024, ragged), _features(rng, 128, 8192, ragged)
    else:
        most, bias = 1 << 60, False
        M, K, N = _log(rng, 64, 11008), _features(rng, 256, 11008, ragged), 0
    if dtype == "fp32":
        most //= 4                                       # four-byte activations and gradients: keep the memory in bounds
    if M * K * max(N, 1) > most:
        M = max(1, most // (K * max(N, 1)))
    c = _case("", kind, M, K, N, block, dtype, bias)
    del c["name"]
    return c


def _activations(g, shape, dtype, std=1.0):
    """Hidden states: normal, with a few feature channels an order of magnitude above the rest."""
    t = torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).mul_(std)
    k = shape[-1]
    loud = torch.randint(0, k, (max(1, k // 512),), generator=g, device="cuda")
    t[..., loud] *= 12.0
    return t.to(dtype)


def _layer(g, n, k, case, train=False):
    dtype = DTYPES[case["dtype"]]
    lin = BlockInt8Linear(k, n, case["bias"], device="cuda", dtype=dtype)
    lin.weight.data = torch.randn((n, k), generator=g, device="cuda", dtype=dtype).mul_(0.02)
    if case["bias"]:
        lin.bias.data = torch.randn((n,), generator=g, device="cuda", dtype=dtype).mul_(0.1)
    lin.train(train)
    if not train:
        lin.prepare_for_eval(drop_weight=True)           # int8-resident inference
    return lin


def prepare(case, seed):
    torch.cuda.set_device(0)
    block_linear_config.GROUP_SIZE = case["block"]
    block_linear_config.INPUT_OUTPUT_TORCH_TYPE = dtype = DTYPES[case["dtype"]]
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    M, K, N = case["M"], case["K"], case["N"]
    s = {"kind": case["kind"]}
    with torch.no_grad():
        if case["kind"] == "linear":
            s["lin"] = _layer(g, N, K, case)
            s["x"] = _activations(g, (1, M, K), dtype)
        elif case["kind"] in ("mlp", "decode_layer"):
            s["x"] = _activations(g, (M, K), dtype)
            s["norm2"] = torch.randn((K,), generator=g, device="cuda", dtype=dtype).mul_(0.1).add_(1.0)
            s["gate_up"], s["down"], s["N"] = _layer(g, 2 * N, K, case), _layer(g, K, N, case), N
            if case["kind"] == "decode_layer":
                heads = K // HEAD_DIM
                s["norm1"] = torch.randn((K,), generator=g, device="cuda", dtype=dtype).mul_(0.1).add_(1.0)
                s["qkv"], s["out"] = _layer(g, 3 * K, K, case), _layer(g, K, K, case)
                s["shape"] = (M, 3, heads, HEAD_DIM)
                s["kcache"], s["vcache"] = (torch.randn((M, heads, CACHE_ROWS, HEAD_DIM), generator=g, device="cuda",
                                                        dtype=torch.float32).to(dtype) for _ in range(2))
                s["pos"] = torch.randint(0, CACHE_ROWS, (1,), generator=g, device="cuda")
                angle = s["pos"] * torch.pow(10000.0, -torch.arange(0, HEAD_DIM, 2, device="cuda") / HEAD_DIM)
                s["cis"] = torch.polar(torch.ones_like(angle), angle)
                s["attention"] = _activations(g, (M, K), dtype, 0.5)
        elif case["kind"] == "train":
            s["lin"] = _layer(g, N, K, case, train=True)
            s["x"] = _activations(g, (1, M, K), dtype).requires_grad_(True)
            s["gy"] = torch.randn((1, M, N), generator=g, device="cuda", dtype=dtype).mul_(1e-3)
        elif case["kind"] == "matmul":
            s["a"] = _activations(g, (M, K), dtype)
            s["b"] = torch.randn((N, K), generator=g, device="cuda", dtype=dtype).mul_(0.02)
        else:
            s["w"] = torch.randn((M, K), generator=g, device="cuda", dtype=dtype).mul_(0.02)
    return s


def _mlp(s, x):
    h = s["gate_up"].infer_pre(x, "rmsnorm", norm_weight=s["norm2"], eps=1e-5)
    return s["down"].infer_pre(h[:, :s["N"]], "silu_mul", x2=h[:, s["N"]:], residual=x)


def run(s):
    kind = s["kind"]
    if kind == "train":
        lin = s["lin"]
        y = lin(s["x"])
        of = (s["x"], lin.weight) if lin.bias is None else (s["x"], lin.weight, lin.bias)
        return (y.detach(), *torch.autograd.grad(y, of, s["gy"]))
    with torch.no_grad():
        if kind == "linear":
            return s["lin"](s["x"])
        if kind == "mlp":
            return _mlp(s, s["x"])
        if kind == "decode_layer":
            qkv = s["qkv"].infer_pre(s["x"], "rmsnorm", norm_weight=s["norm1"], eps=1e-5)
            q = rope_cache_append(qkv.view(s["shape"]), s["cis"], s["pos"], s["kcache"], s["vcache"])
            x = s["out"].infer_pre(s["attention"], residual=s["x"])
            return _mlp(s, x), q, s["kcache"], s["vcache"]
        if kind == "matmul":
            return fast_matmulT(s["a"], s["b"])
        q, state = quantize_block_rowwise(s["w"])
        return q, state, dequantize_block_rowwise(q, state)


def _quantized(n, k, block):
    """Bytes of a quantized [n, k] matrix: int8 values and fp32 block scales."""
    return n * k + 4 * n * -(-k // block)


def work(case):
    M, K, N, b, e = case["M"], case["K"], case["N"], case["block"], SIZE[case["dtype"]]
    bias = N * e if case["bias"] else 0
    if case["kind"] == "linear":
        return {"bytes": M * K * e + _quantized(N, K, b) + M * N * e + bias, "flops": 2 * M * K * N}
    mlp = {"bytes": 2 * M * K * e + K * e + _quantized(2 * N, K, b) + _quantized(K, N, b), "flops": 6 * M * K * N}
    if case["kind"] == "mlp":
        return mlp
    if case["kind"] == "decode_layer":
        # q is returned, one row of k and one of v written per sequence
        more = K * e + _quantized(3 * K, K, b) + _quantized(K, K, b) + M * K * e + 3 * M * K * e + HEAD_DIM * 4
        return {"bytes": mlp["bytes"] + more, "flops": mlp["flops"] + 8 * M * K * K}
    if case["kind"] == "train":
        # x, W, dY (and the bias) in; y, dX, dW (and dbias) out
        return {"bytes": e * 2 * (M * K + N * K + M * N) + 2 * bias, "flops": 6 * M * K * N}
    if case["kind"] == "matmul":
        return {"bytes": e * (M * K + N * K + M * N), "flops": 2 * M * K * N}
    return {"bytes": M * K * e + _quantized(M, K, b) + M * K * e, "flops": 0}


def tolerance(case):
    """Quantized values, scales and dequantized results are defined to the bit.  A GEMM's block partial sums are exact integers,
    what may differ is the order of the fp32 sum over blocks and the rounding of the result: 32-bit sums in single
    precision, one rounding of 16-bit results.  In mlp and decode_layer such a rounding, or the order of the
    normalisation's sum, moves a value of the next quantizer's input by one step of its type, and some int8 values with it."""
    if case["kind"] == "round_trip":
        return "exact"
    if case["kind"] in ("mlp", "decode_layer"):
        return {"rel": 1e-2}
    return {"rel": {"bf16": 5e-3, "fp16": 1e-3, "fp32": 1e-5}[case["dtype"]]}
