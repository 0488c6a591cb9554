"""Several small quantizations in one launch (bi8_quantize_many) against the single-purpose functions: the same bits, whatever runs beside
them; column sums against fp64 (fp32 accumulation of R terms: R * 2^-24 * sum |x|, plus the rounding to the result's type)."""
import ctypes

import pytest
import torch

from tests.gpu_util import DEV, assert_clean_device, randn_bf16

pytestmark = pytest.mark.gpu


class Task(ctypes.Structure):
    _fields_ = [("x", ctypes.c_void_p), ("ldx", ctypes.c_int64), ("rows", ctypes.c_int64), ("cols", ctypes.c_int64), ("q_row", ctypes.c_void_p),
                ("ldq_row", ctypes.c_int64), ("s_row", ctypes.c_void_p), ("q_col", ctypes.c_void_p), ("ldq_col", ctypes.c_int64),
                ("s_col", ctypes.c_void_p), ("sum", ctypes.c_void_p), ("x_dtype", ctypes.c_int)]


def _pitch(n):
    return (n + 15) // 16 * 16


def _task(x, code, block, row, col, sums):
    r, c = x.shape
    out = {}
    if row:
        out["q_row"] = torch.zeros((r, _pitch(c)), dtype=torch.int8, device=DEV)
        out["s_row"] = torch.zeros((-(-c // block), r), device=DEV)
    if col:
        out["q_col"] = torch.zeros((c, _pitch(r)), dtype=torch.int8, device=DEV)
        out["s_col"] = torch.zeros((-(-r // block), c), device=DEV)
    if sums:
        out["sum"] = torch.zeros(c, dtype=x.dtype, device=DEV)
    p = {k: v.data_ptr() for k, v in out.items()}
    return Task(x.data_ptr(), x.stride(0), r, c, p.get("q_row"), _pitch(c), p.get("s_row"), p.get("q_col"), _pitch(r), p.get("s_col"), p.get("sum"), code), out


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("block", [32, 64, 128])
@pytest.mark.parametrize("shapes", [((300, 256), (384, 256)), ((1, 1), (7, 9)), ((129, 65), (33, 257)), ((511, 130), (64, 1000)), ((512, 512), (1024, 257))])
def test_jobs_share_a_launch(shapes, block, dtype):
    from blockwise_int8_linear_b200 import _lib
    from triton_functions import quantize_block_colwise, quantize_block_rowwise
    L = _lib.lib()
    code = {torch.bfloat16: _lib.BI8_BF16, torch.float16: _lib.BI8_F16, torch.float32: _lib.BI8_F32}[dtype]
    a, b = (randn_bf16(s, s[0] + s[1], outliers=0.01).to(dtype).to(DEV) for s in shapes)
    w = torch.randint(-127, 128, (37, 101), dtype=torch.int8, device=DEV)
    wc = torch.zeros((37, _pitch(101)), dtype=torch.int8, device=DEV)
    ta, oa = _task(a, code, block, True, True, True)
    tb, ob = _task(b, code, block, True, False, False)
    tw = Task(w.data_ptr(), 101, 37, 101, wc.data_ptr(), _pitch(101), None, None, 0, None, None, 3)
    tasks = (Task * 3)(ta, tb, tw)
    assert L.bi8_quantize_many_fits(tasks, 3, block) == 1
    _lib.check(L.bi8_quantize_many(tasks, 3, block, _lib.stream_ptr()), "bi8_quantize_many")
    for x, o in ((a, oa), (b, ob)):
        q, s = quantize_block_rowwise(x, block)
        assert torch.equal(o["q_row"][:, :x.shape[1]], q) and torch.equal(o["s_row"], s)
    q, s = quantize_block_colwise(a, block)
    assert torch.equal(oa["q_col"][:, :a.shape[0]], q) and torch.equal(oa["s_col"], s)
    assert torch.equal(wc[:, :101], w)
    exact, mag = a.double().sum(0), a.double().abs().sum(0)
    step = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -24}[dtype]
    assert bool(((oa["sum"].double() - exact).abs() <= a.shape[0] * 2.0 ** -24 * mag + step * exact.abs()).all())
    assert_clean_device()


def test_tasks_that_do_not_share_a_launch():
    """Large tasks run one after another with the same results, and refuse column sums."""
    from blockwise_int8_linear_b200 import _lib
    from triton_functions import quantize_block_colwise, quantize_block_rowwise
    L = _lib.lib()
    x = randn_bf16((4096, 1024), 3).to(DEV)
    t, o = _task(x, _lib.BI8_BF16, 64, True, True, False)
    tasks = (Task * 1)(t)
    assert L.bi8_quantize_many_fits(tasks, 1, 64) == 0
    _lib.check(L.bi8_quantize_many(tasks, 1, 64, _lib.stream_ptr()), "bi8_quantize_many")
    q, s = quantize_block_rowwise(x, 64)
    assert torch.equal(o["q_row"], q) and torch.equal(o["s_row"], s)
    q, s = quantize_block_colwise(x, 64)
    assert torch.equal(o["q_col"], q) and torch.equal(o["s_col"], s)
    t, o = _task(x, _lib.BI8_BF16, 64, True, True, True)
    assert L.bi8_quantize_many((Task * 1)(t), 1, 64, _lib.stream_ptr()) == -9
    assert_clean_device()
