"""The native host path and the Python code behind it give the same results for the same call, and the
calls that the native path leaves alone still end in the Python code's errors."""
import threading
import time

import pytest
import torch

import flag_gems
from flaggems_b200 import _cabi

pytestmark = pytest.mark.gpu
FP8 = torch.float8_e4m3fn


class _Off:
    def __getattr__(self, name):
        return lambda *args: None


def _rand(*shape, dtype=torch.bfloat16, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).cuda().to(dtype)


def _mm_operands(m, n, k):
    return _rand(m, k, dtype=FP8), _rand(n, k, dtype=FP8, seed=1), _rand(m, 1, dtype=torch.float32, seed=2).abs(), \
        _rand(n, dtype=torch.float32, seed=3).abs()


def _cutlass(m, n, k, bias):
    a, b, sa, sb = _mm_operands(m, n, k)
    c = torch.zeros(m, n, dtype=torch.bfloat16, device="cuda")
    flag_gems.cutlass_scaled_mm(c, a, b.t(), sa, sb, bias)
    return c


def _aten(m, n, k, out_dtype, bias=None):
    a, b, sa, sb = _mm_operands(m, n, k)
    return flag_gems.scaled_mm(a, b.t(), sa, sb.view(1, n), bias, None, out_dtype)


def _block(m, k, n=256):
    a, b = _rand(m, k, dtype=FP8), _rand(n, k, dtype=FP8, seed=1)
    s, bs = _rand(m, k // 128, dtype=torch.float32, seed=2).abs(), _rand(n // 128, k // 128, dtype=torch.float32, seed=3).abs()
    return flag_gems.w8a8_block_fp8_matmul(a, b, s, bs, [128, 128], torch.float16)


def _topk(dtype):
    w = torch.empty(5, 2, device="cuda")
    i, s = torch.empty(5, 2, dtype=dtype, device="cuda"), torch.empty(5, 2, dtype=torch.int32, device="cuda")
    flag_gems.topk_softmax(w, i, s, _rand(5, 16), True)
    return w, i, s


def _grouped(offs):
    a, b = _rand(37, 64, dtype=FP8), _rand(3, 32, 64, dtype=FP8, seed=1)
    return flag_gems.scaled_grouped_mm(a, b.transpose(1, 2), torch.full((37,), 0.5, device="cuda"),
                                       torch.full((3, 32), 0.25, device="cuda"), torch.tensor(offs, dtype=torch.int32, device="cuda"))


CALLS = [
    lambda: flag_gems.act_quant_triton(_rand(3, 256), 128, "ue8m0"),
    lambda: flag_gems.per_token_group_quant_fp8(_rand(2, 3, 256), 128),
    lambda: flag_gems.per_token_group_quant_fp8(_rand(7, 512)[:, :256], 64, column_major_scales=True),
    lambda: flag_gems.per_token_group_quant_fp8(_rand(1, 256, dtype=torch.float32), 128, 1e-6, None, False, True),
    lambda: flag_gems.moe_kernel_quantize_input(_rand(5, 264), None, FP8, True),
    lambda: flag_gems.moe_kernel_quantize_input(_rand(5, 264), torch.full((1,), 0.01, device="cuda"), FP8, False),
    lambda: _cutlass(1, 128, 256, None),
    lambda: _cutlass(33, 128, 256, _rand(128)),
    lambda: _aten(33, 128, 256, torch.float32),
    lambda: _aten(2, 128, 256, None, _rand(128, dtype=torch.float32)),
    lambda: _block(1, 256),
    lambda: _block(130, 384),
    lambda: _grouped([5, 5, 37]),
    lambda: _topk(torch.int32),
    lambda: _topk(torch.int64),
    lambda: flag_gems.grouped_topk(_rand(9, 32), 4, 2, 4, True, 2.5, _rand(32), 1),
    lambda: flag_gems.moe_align_block_size(torch.arange(24, device="cuda", dtype=torch.int64).view(12, 2) % 5, 16, 5, None, True),
    lambda: flag_gems.silu_and_mul(_rand(4, 64)[:, :32], _rand(4, 32, seed=1)),
    lambda: flag_gems.moe_sum(_rand(3, 2, 64), torch.empty(3, 64, dtype=torch.bfloat16, device="cuda")),
]


@pytest.mark.parametrize("call", CALLS)
def test_native_and_python_host_paths_agree(call, monkeypatch):
    native = call()
    monkeypatch.setattr(_cabi, "host", _Off())
    python = call()
    for x, y in zip(native if isinstance(native, tuple) else (native,), python if isinstance(python, tuple) else (python,)):
        assert x.shape == y.shape and x.dtype == y.dtype and x.stride() == y.stride()
        assert torch.equal(x.contiguous().view(torch.uint8), y.contiguous().view(torch.uint8))


def test_refused_calls_still_raise():
    a, b, sa, sb = _mm_operands(4, 128, 256)
    with pytest.raises(AssertionError, match="16-byte aligned"):
        flag_gems.cutlass_scaled_mm(torch.empty(4, 136, dtype=torch.bfloat16, device="cuda")[:, :128], a, b.t(), sa, sb)
    with pytest.raises(RuntimeError, match="scale_a must be a scalar tensor"):
        flag_gems.scaled_mm(a, b.t(), sa.view(1, 4), sb)
    with pytest.raises(NotImplementedError, match="16-byte aligned"):
        flag_gems.per_token_group_quant_fp8(_rand(1, 1025)[:, 1:], 128)
    with pytest.raises(AssertionError, match="must be divisible"):
        flag_gems.per_token_group_quant_fp8(_rand(1, 100), 128)


def test_other_threads_run_while_a_call_blocks():
    # A kernel of about 0.6 s in front of more launches than the queue holds: the calls block, other Python threads do not.
    x = _rand(1, 256)
    flag_gems.act_quant_triton(x, 128)
    torch.cuda.synchronize()
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.monotonic())
            time.sleep(0.002)

    thread = threading.Thread(target=tick)
    thread.start()
    try:
        torch.cuda._sleep(1_200_000_000)  # GPU clocks, below 2 GHz
        begin = time.monotonic()
        for _ in range(6000):
            flag_gems.act_quant_triton(x, 128)
        blocked = time.monotonic() - begin
    finally:
        stop.set()
        thread.join()
    torch.cuda.synchronize()
    assert blocked > 0.3, "the launch queue never filled: nothing was tested"
    assert max(b - a for a, b in zip(ticks, ticks[1:])) < 0.15


def test_a_flag_without_a_truth_value_raises_its_own_error():
    both = torch.ones(2, dtype=torch.bool)
    x = _rand(9, 256)
    for call in (lambda: flag_gems.per_token_group_quant_fp8(x, 128, scale_ue8m0=both),
                 lambda: flag_gems.per_token_group_quant_fp8(x, 128, column_major_scales=both),
                 lambda: flag_gems.grouped_topk(x, 4, 2, 4, both, 2.5, x[0], 1),
                 lambda: flag_gems.topk_softmax(*_topk(torch.int32), x[:5, :16].contiguous(), both)):
        with pytest.raises(RuntimeError, match="ambiguous"):
            call()
