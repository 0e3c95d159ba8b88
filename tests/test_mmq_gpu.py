"""Prefill tcgen05 dequant-GEMM vs the oracle's EXACT product (f64 sum of deq(w)*x) — the
known-answer structure of the reference's own GEMM test (packed_affine.rs:967-1000:
quantized product == dequantize() . x, max abs <= 0.08, mean <= 0.01 on patterned inputs)."""
import os

import numpy as np
import pytest
import torch

import oracle
from mistralrs_b200 import mmq, quant
from util import ALL_TYPES, make_acts, make_weight, to_dev

pytestmark = pytest.mark.gpu


def _check(dtype, M, N, K, dt, seed=0):
    cuda = torch.device("cuda:0")
    wb = make_weight(dtype, N, K, seed)
    x = make_acts(M, K, seed + 1, dt)
    w = quant.QTensor(to_dev(wb.reshape(-1), cuda), dtype, (N, K))
    y = mmq.forward(w, to_dev(x, cuda, dt)).float().cpu().numpy()
    ref = oracle.matmul_exact(dtype, wb, x, K, N)
    mag = np.abs(oracle.dequantize(dtype, wb).reshape(N, K)).astype(np.float64) @ np.abs(x).astype(np.float64).T  # sum |w||x|
    ulp = {"bf16": 2.0 ** -8, "f16": 2.0 ** -11}[dt]
    # one output rounding + weight rounding to the operand format (2^-9 bf16 / 2^-12 f16 per
    # term, random sign -> well inside ulp * sum|w||x|) + f32 accumulation
    tol = ulp * np.abs(ref) * 1.01 + ulp * mag.T + 1e-6
    err = np.abs(y - ref)
    assert (err <= tol).all(), (dtype, M, N, K, float((err / tol).max()))


@pytest.mark.parametrize("dtype", ["q8_0", "q4_k", "q6_k"])
@pytest.mark.parametrize("dt", ["bf16", "f16"])
def test_main_types(cuda, dtype, dt):
    _check(dtype, 300, 520, 512, dt)      # ragged M and N (partial tiles)
    _check(dtype, 256, 256, 1024, dt, 3)  # exactly one tile, several ring wraps


@pytest.mark.parametrize("dtype", [t for t in ALL_TYPES if t not in ("q8_0", "q4_k", "q6_k")])
def test_other_types(cuda, dtype):
    _check(dtype, 130, 260, 256, "bf16", 5)


def test_reference_known_answer_shapes(cuda):
    # shapes of the reference's marlin_matches_dequantized_* tests, patterned inputs
    def patterned(shape, seed, scale):
        i = np.arange(int(np.prod(shape)))
        return (np.sin(((i * 37 + seed * 17) % 251) * 0.071) * scale).astype(np.float32).reshape(shape)
    for (m, n, k) in [(9, 64, 256), (64, 128, 512), (127, 192, 512)]:
        for dtype in ("q4_k", "q8_0", "q6_k"):
            wb = make_weight(dtype, n, k, 11)
            x = oracle.round_dtype(patterned((m, k), 3, 0.5), "bf16")
            w = quant.QTensor(to_dev(wb.reshape(-1), cuda), dtype, (n, k))
            y = mmq.forward(w, to_dev(x, cuda, "bf16")).float().cpu().numpy()
            ref = oracle.matmul_exact(dtype, wb, x, k, n)
            scale = np.abs(ref).max()
            assert np.abs(y - ref).max() <= 0.08 * max(scale, 1.0) / 8 and np.abs(y - ref).mean() <= 0.01 * max(scale, 1.0) / 8


def test_matches_decode_path_semantics(cuda):
    # GgufMatMul dispatch: batch 8 -> MMVQ (Q8_1 activations), batch 9 -> tcgen05 GEMM; both
    # must agree with the exact product within the reference's MMVQ-vs-dequant envelope
    K, N = 1024, 256
    wb = make_weight("q4_k", N, K, 2)
    w = quant.QTensor(to_dev(wb.reshape(-1), cuda), "q4_k", (N, K))
    lin = quant.GgufMatMul(w)
    x = make_acts(9, K, 4, "bf16")
    y9 = lin.forward(to_dev(x, cuda, "bf16")).float().cpu().numpy()
    y8 = lin.forward(to_dev(x[:8], cuda, "bf16")).float().cpu().numpy()
    ref = oracle.matmul_exact("q4_k", wb, x, K, N)
    scale = np.abs(ref).max()
    assert np.abs(y9 - ref).max() <= 2.0 ** -7 * scale
    assert np.abs(y8 - ref[:8]).max() <= 2e-2 * scale   # int8 activations: ~1/127 per-block noise


@pytest.mark.parametrize("dtype", ["q8_0", "q4_k", "q6_k"])
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("M,N,K", [(300, 520, 2048), (64, 136, 4096), (129, 128, 2048)])
def test_second_generation_kernel(cuda, dtype, dt, M, N, K):
    """csrc/mmq_ts.cu (swap-AB, dequantised weights as the A operand in tensor memory, raw blocks through the TMA) —
    shapes it takes for all three types (K % 2048 == 0 keeps Q6_K rows a multiple of 16 bytes): ragged token and row
    tiles, both token-tile widths (M <= 128 -> 128, else 256).  Against the exact product, and bit for bit against
    csrc/mmq_tc.cu: same weight rounding, same k order of the f32 accumulation."""
    _check(dtype, M, N, K, dt, 7)
    wb = make_weight(dtype, N, K, 7)
    x = to_dev(make_acts(M, K, 8, dt), cuda, dt)
    w = quant.QTensor(to_dev(wb.reshape(-1), cuda), dtype, (N, K))
    try:
        mmq.set_path("tc")
        y_tc = mmq.forward(w, x).clone()
    finally:
        mmq.set_path("auto")
    y_ts = mmq.forward(w, x)
    assert torch.equal(y_tc, y_ts), float((y_tc.float() - y_ts.float()).abs().max())


@pytest.mark.parametrize("dtype", ALL_TYPES)
@pytest.mark.parametrize("dt,M,N,K", [("f16", 9, 129, 768), ("bf16", 130, 1029, 1280), ("bf16", 17, 1024, 2048), ("f16", 257, 1030, 2304)])
def test_every_type_at_tile_edges(cuda, dtype, dt, M, N, K):
    """csrc/mmq_ts.cuh: rows that are multiples of 16 bytes and rows that are not (768, 1280, 2304), K whole and K split over a cluster
    (from 1024 rows on), ragged token and row tiles, one token past a tile."""
    from mistralrs_b200 import lib
    _check(dtype, M, N, K, dt, 11)
    assert lib().mrs_mmq_timeouts() == 0


@pytest.mark.parametrize("dtype", ["q4_0", "q4_1", "q5_0", "q5_1", "q8_0"])
@pytest.mark.parametrize("K", [64, 320, 2880])
def test_ragged_last_span(cuda, dtype, K):
    """32-wide types take any multiple of 64 columns: the last 256 are partly past the row."""
    _check(dtype, 33, 1100, K, "bf16", 13)


def test_calls_are_refused_once_a_wait_has_run_out(cuda):
    """The word that a kernel sets when a wait runs out, set here by the host: ggml and int4 calls and the runners' check report it."""
    import ctypes
    from mistralrs_b200 import gptq, lib
    K, N = 256, 64
    w = quant.QTensor(to_dev(make_weight("q4_k", N, K, 1).reshape(-1), cuda), "q4_k", (N, K))
    int4 = gptq.GptqMarlinLayer(torch.zeros(K // 8, N, dtype=torch.int32, device=cuda), torch.ones(K // 64, N, dtype=torch.float16, device=cuda), group_size=64)
    x = torch.ones(9, K, dtype=torch.float16, device=cuda)
    want = [mmq.forward(w, x), int4.forward_raw(x)]
    assert lib().mrs_mmq_timeouts() == 0
    fn = lib().mrs_mmq_timeout_flag
    fn.restype = ctypes.POINTER(ctypes.c_int32)
    flag = fn()
    try:
        flag[0] = 1
        for call in (lambda: mmq.forward(w, x), lambda: int4.forward_raw(x)):
            with pytest.raises(RuntimeError, match="702"):
                call()
        with pytest.raises(RuntimeError, match="ran out"):
            mmq.check_timeouts(cuda)
        assert lib().mrs_mmq_timeouts() == 1
    finally:
        flag[0] = 0
    mmq.check_timeouts(cuda)
    assert torch.equal(mmq.forward(w, x), want[0]) and torch.equal(int4.forward_raw(x), want[1])


def test_first_call_of_a_process_inside_a_capture(cuda):
    """The first call sets up what calls on a device share; a capture does not forbid it."""
    import subprocess
    import sys
    code = """
import torch
from __graft_entry__ import load_package
load_package()
from mistralrs_b200 import mmq, quant
w = quant.QTensor(torch.randint(0, 64, (64 * 144,), dtype=torch.uint8, device='cuda'), 'q4_k', (64, 256))
x = torch.ones(9, 256, dtype=torch.bfloat16, device='cuda')
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    y = mmq.forward(w, x)
g.replay()
torch.cuda.synchronize()
assert torch.equal(y, mmq.forward(w, x))
mmq.check_timeouts(x.device)
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
