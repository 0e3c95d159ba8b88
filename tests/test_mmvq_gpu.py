"""Decode GEMV parity: CUDA (through the reference-shaped C ABI) vs the CPU oracle's Q8_1
arithmetic on the same seeded inputs.  Tolerances: the oracle value is the infinitely-precise
result of the reference's integer-dot arithmetic; the kernel may differ by f32 accumulation
order (<= 2e-6 of the output scale) plus one rounding to the output dtype."""
import numpy as np
import pytest
import torch

import oracle
from mistralrs_b200 import quant
from util import ALL_TYPES, make_acts, make_weight, to_dev, ulp_report

pytestmark = pytest.mark.gpu


def _oracle_gemv(dtype, wb, x_np, K, N):
    xq, stride = oracle.quantize_q8_1(x_np)
    return oracle.mmvq_q8_1(dtype, wb, xq, K, N, stride, x_np.shape[0])


@pytest.mark.parametrize("dtype", ALL_TYPES)
@pytest.mark.parametrize("dt", ["bf16", "f32", "f16"])
def test_plain_batch1(cuda, dtype, dt):
    K, N = 2048, 70  # ragged N: not a multiple of the 16-row pass
    wb = make_weight(dtype, N, K, 1)
    x = make_acts(1, K, 2, dt)
    w = quant.QTensor(to_dev(wb.reshape(-1), cuda), dtype, (N, K))
    y = quant.plain(w, to_dev(x, cuda, dt)).float().cpu().numpy()
    ref = _oracle_gemv(dtype, wb, x, K, N)
    rel, frac = ulp_report(y, ref, dt)
    assert frac >= 0.995 and rel < 4e-3, (dtype, dt, rel, frac)


@pytest.mark.parametrize("dtype", ["q4_k", "q6_k", "q8_0", "q5_k", "q2_k", "q3_k", "q4_0", "q5_1"])
@pytest.mark.parametrize("batch", [2, 3, 4, 5, 8])
def test_plain_batched(cuda, dtype, batch):
    K, N = 1536, 33  # K = 1.5 segments (ragged K), odd N
    wb = make_weight(dtype, N, K, 3)
    x = make_acts(batch, K, 4, "f32")
    w = quant.QTensor(to_dev(wb.reshape(-1), cuda), dtype, (N, K))
    y = quant.plain(w, to_dev(x, cuda, "f32")).cpu().numpy()
    ref = _oracle_gemv(dtype, wb, x, K, N)
    rel, frac = ulp_report(y, ref, "f32")
    assert rel < 5e-6, (dtype, batch, rel, frac)


@pytest.mark.parametrize("dtype", ["q4_k", "q6_k", "q8_0", "q5_0"])
def test_llama_shapes_f32(cuda, dtype):
    # the real Llama-3-8B projection shapes, f32 output so the check is tight
    for (N, K) in [(4096, 4096), (1024, 4096), (256, 14336)]:
        wb = make_weight(dtype, N, K, 5)
        x = make_acts(1, K, 6, "f32")
        w = quant.QTensor(to_dev(wb.reshape(-1), cuda), dtype, (N, K))
        y = quant.plain(w, to_dev(x, cuda, "f32")).cpu().numpy()
        ref = _oracle_gemv(dtype, wb, x, K, N)
        rel, _ = ulp_report(y, ref, "f32")
        assert rel < 5e-6, (dtype, N, K, rel)


@pytest.mark.parametrize("dtype", ALL_TYPES)
@pytest.mark.parametrize("batch", [1, 3])
def test_fused_qkv_matches_plain(cuda, dtype, batch):
    # the reference's own self-consistency test (fast_mmq.rs:1583-1703): fused == unfused
    K = 1024
    nq, nk, nv = 96, 24, 24
    ws = [quant.QTensor(to_dev(make_weight(dtype, n, K, 10 + i).reshape(-1), cuda), dtype, (n, K))
          for i, n in enumerate((nq, nk, nv))]
    x = to_dev(make_acts(batch, K, 7, "bf16"), cuda, "bf16")
    q, k, v = quant.fused_qkv(ws[0], ws[1], ws[2], x)
    for got, w in zip((q, k, v), ws):
        assert torch.equal(got, quant.plain(w, x))


@pytest.mark.parametrize("dtype", ["q4_k", "q6_k", "q8_0", "q4_1", "q3_k"])
@pytest.mark.parametrize("act", [0, 1, 2, 3, 4])
def test_fused_glu(cuda, dtype, act):
    K, N = 1024, 41
    g = quant.QTensor(to_dev(make_weight(dtype, N, K, 20).reshape(-1), cuda), dtype, (N, K))
    u = quant.QTensor(to_dev(make_weight(dtype, N, K, 21).reshape(-1), cuda), dtype, (N, K))
    x = to_dev(make_acts(2, K, 8, "bf16"), cuda, "bf16")
    got = quant.fused_glu(g, u, x, quant.GluActivationType(act)).float().cpu().numpy()
    gate = quant.plain(g, x).float().cpu().numpy()
    up = quant.plain(u, x).float().cpu().numpy()
    want = oracle.fused_glu(gate, up, act, "bf16")
    # activation uses the GPU's fast exp/div/tanh (the reference builds with --use_fast_math): one
    # bf16 ulp on the activated value, plus tanh.approx's 2^-10.99 absolute error carried through
    # 0.5*gate*(1+tanh)*up where 1+tanh cancels
    tol = 2.0 ** -7 * np.abs(want) + 2.0 ** -10 * np.abs(gate * up) + 1e-6
    assert (np.abs(got - want) <= tol).all(), (dtype, act, np.abs(got - want).max())


def test_quantize_q8_1_vs_oracle(cuda):
    # bit-level: d, sum and the int8 quants (approximate GPU division may move a tie by 1)
    for dt in ("bf16", "f16", "f32"):
        x = make_acts(3, 1000, 9, dt)  # ragged K -> zero padding to 1024
        got = quant.quantize_q8_1(to_dev(x, cuda, dt)).cpu().numpy().reshape(3, -1, 36)
        want, stride = oracle.quantize_q8_1(x)
        want = want.reshape(3, -1, 36)
        assert got.shape == want.shape
        dq = np.abs(got[..., 4:].view(np.int8).astype(int) - want[..., 4:].view(np.int8).astype(int))
        assert dq.max() <= 1 and (dq != 0).mean() < 2e-3, (dt, dq.max(), (dq != 0).mean())
        dd = np.abs(got[..., :4].view(np.float16).astype(np.float32) - want[..., :4].view(np.float16).astype(np.float32))
        assert (dd <= 2e-3 * np.abs(want[..., :4].view(np.float16).astype(np.float32)) + 1e-7).all()


def test_fused_prologue_matches_two_step(cuda):
    # mrs_mmvq_fused (RMSNorm + Q8_1 + GEMV + residual in one launch) == unfused chain
    K, N = 2048, 64
    for dtype in ("q4_k", "q6_k"):
        w = quant.QTensor(to_dev(make_weight(dtype, N, K, 30).reshape(-1), cuda), dtype, (N, K))
        x = to_dev(make_acts(1, K, 31, "bf16"), cuda, "bf16")
        nw = to_dev(1.0 + 0.1 * make_acts(1, K, 32, "bf16")[0], cuda, "bf16")
        res = to_dev(make_acts(1, N, 33, "bf16"), cuda, "bf16")
        normed = oracle.rms_norm(x.float().cpu().numpy(), nw.float().cpu().numpy(), 1e-5, "bf16")
        want = quant.plain(w, to_dev(normed, cuda, "bf16"))
        want = (want.float() + res.float()).to(torch.bfloat16)
        got = quant.mmvq_fused(w, x, norm_w=nw, eps=1e-5, residual=res)
        diff = (got.float() - want.float()).abs().max().item()
        assert diff <= 2.0 ** -6 * want.float().abs().max().item(), (dtype, diff)


@pytest.mark.parametrize("dtype", ["q4_k", "q6_k"])
def test_long_segment_variant_agrees(cuda, dtype):
    # lm_head-sized streams take K segments twice as long (UPL x2): same arithmetic in a different
    # consumption order of the activation image -> results must agree bit for bit with the short
    # segments, with pre-quantised activations and with the fused RMSNorm prologue
    import ctypes
    from mistralrs_b200 import lib
    K, N = 4096, 700
    w = quant.QTensor(to_dev(make_weight(dtype, N, K, 40).reshape(-1), cuda), dtype, (N, K))
    nw = to_dev(1.0 + 0.1 * make_acts(1, K, 42, "bf16")[0], cuda, "bf16")
    x = to_dev(make_acts(1, K, 44, "bf16"), cuda, "bf16")
    outs = []
    try:
        for flags in (8 | (1 << 8), 1 << 8):      # long variant off / on from 1 MiB of weights
            lib().mrs_set_mmvq_flags(ctypes.c_int(flags))
            outs.append([quant.plain(w, x), quant.mmvq_fused(w, x, norm_w=nw, eps=1e-5)])
    finally:
        lib().mrs_set_mmvq_flags(ctypes.c_int(128 << 8))
    for a, b in zip(*outs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("pair", [("q4_k", "q6_k"), ("q5_k", "q6_k"), ("q4_k", "q5_k"), ("q4_0", "q8_0")])
@pytest.mark.parametrize("batch", [1, 3])
def test_fused_qkv_mixed_matches_separate_launches(cuda, pair, batch):
    # two-type QKV grid (attn_v in its own ggml type) == mode-2 q||k launch + plain v launch, bit for
    # bit; unsupported pairs / batch > 1 take the two-launch fallback inside the same entry point
    tq, tv = pair
    K, nq, nk, nv = 2048, 320, 64, 64
    wq, wk = (quant.QTensor(to_dev(make_weight(tq, n, K, 50 + i).reshape(-1), cuda), tq, (n, K)) for i, n in enumerate((nq, nk)))
    wv = quant.QTensor(to_dev(make_weight(tv, nv, K, 52).reshape(-1), cuda), tv, (nv, K))
    x = to_dev(make_acts(batch, K, 53, "bf16"), cuda, "bf16")
    nw = to_dev(1.0 + 0.1 * make_acts(1, K, 54, "bf16")[0], cuda, "bf16")
    q, k, v = quant.fused_qkv_mixed(wq, wk, wv, x, norm_w=nw, eps=1e-5)
    q2, k2 = quant.mmvq_fused(wq, x, mode=2, w1=wk, norm_w=nw, eps=1e-5)[:2]
    v2 = quant.mmvq_fused(wv, x, norm_w=nw, eps=1e-5)
    assert torch.equal(q, q2) and torch.equal(k, k2) and torch.equal(v, v2)


def test_argument_errors(cuda):
    w = quant.QTensor(torch.zeros(144 * 4, dtype=torch.uint8, device=cuda), "q4_k", (4, 256))
    with pytest.raises(ValueError, match="batch size 9"):
        quant.plain(w, torch.zeros(9, 256, device=cuda, dtype=torch.bfloat16))
    with pytest.raises(ValueError, match="shape mismatch"):
        quant.plain(w, torch.zeros(1, 512, device=cuda, dtype=torch.bfloat16))


@pytest.mark.parametrize("dtype", ["q4_k", "q6_k", "q8_0", "q4_0"])
@pytest.mark.parametrize("rows,K,norm", [(1, 512, True), (3, 2304, True), (4, 4096, False), (8, 2048, True), (2, 14336, False)])
def test_quantised_apart_equals_fused(cuda, dtype, rows, K, norm):
    """mrs_rms_quantize_q8_1 + mrs_mmvq_q8 give the bits of mrs_mmvq_fused (a step of several sequences takes the former)."""
    import ctypes
    from mistralrs_b200 import GGML, lib
    gen = torch.Generator(device=cuda).manual_seed(K + rows)
    x = torch.randn(rows, K, device=cuda, generator=gen).to(torch.bfloat16)
    nw = (1 + 0.1 * torch.randn(K, device=cuda, generator=gen)).to(torch.bfloat16) if norm else None
    w = quant.QTensor(to_dev(make_weight(dtype, 96, K, 3).reshape(-1), cuda), dtype, (96, K))
    want = quant.mmvq_fused(w, x, norm_w=nw)
    q8 = torch.empty(rows * (K // 32) * 36, dtype=torch.uint8, device=cuda)
    got = torch.empty(rows, 96, dtype=torch.bfloat16, device=cuda)
    P, I = (lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else 0)), ctypes.c_int
    st = ctypes.c_void_p(torch.cuda.current_stream(cuda).cuda_stream)
    assert lib().mrs_rms_quantize_q8_1(I(1), P(x), P(nw), ctypes.c_float(1e-5), I(K), I(rows), P(q8), I(0), st) == 0
    null = ctypes.c_void_p(0)
    assert lib().mrs_mmvq_q8(I(GGML[dtype]), I(0), I(1), P(w.data), null, null, P(q8), null, P(got), null, null, I(K), I(96), I(0), I(0), I(rows), I(0),
                             I(0), st) == 0
    assert torch.equal(got, want)


@pytest.mark.parametrize("offset", [0, 1, 8])
def test_one_row_at_any_address(cuda, offset):
    """A row off a 16-byte boundary takes the two launches, one on it the fused launch: the same bits."""
    K = 1024
    w = quant.QTensor(to_dev(make_weight("q4_k", 64, K, 5).reshape(-1), cuda), "q4_k", (64, K))
    gen = torch.Generator(device=cuda).manual_seed(offset)
    buf = torch.randn(K + 16, device=cuda, generator=gen).to(torch.bfloat16)
    x = buf[offset:offset + K]
    aligned = x.clone().reshape(1, K)
    assert torch.equal(quant.plain(w, x).reshape(1, -1), quant.plain(w, aligned))
    assert torch.equal(quant.plain(w, torch.cat([aligned, aligned]))[:1], quant.plain(w, aligned))


@pytest.mark.parametrize("pdl", [0, 1])
@pytest.mark.parametrize("dtype", ["q4_k", "q6_k", "q8_0"])
@pytest.mark.parametrize("rows,K", [(2, 2304), (5, 1024), (8, 2048)])
def test_every_mode_over_rows_quantised_apart(cuda, dtype, rows, K, pdl):
    """QKV, GLU and a residual over rows that a launch before quantised, in the chain of a decode step: one buffer, quantised again behind every
    GEMV that reads it, with and without programmatic launches.  The bits of mrs_mmvq_fused."""
    import ctypes
    from mistralrs_b200 import GGML, lib
    gen = torch.Generator(device=cuda).manual_seed(K + rows)
    rand = lambda *s: torch.randn(*s, device=cuda, generator=gen).to(torch.bfloat16)
    weight = lambda n, seed: quant.QTensor(to_dev(make_weight(dtype, n, K, seed).reshape(-1), cuda), dtype, (n, K))
    x, h, nw = rand(rows, K), rand(rows, K), (1 + 0.1 * rand(K).float()).to(torch.bfloat16)
    wq, wk, wv, gate, up, wo = (weight(n, i) for i, n in enumerate((160, 64, 64, 96, 96, K)))
    res = rand(rows, K)
    want = [*quant.mmvq_fused(wq, x, mode=2, w1=wk, w2=wv, norm_w=nw), quant.mmvq_fused(gate, h, mode=1, w1=up, norm_w=nw),
            quant.mmvq_fused(wo, h, residual=res)]
    got = [torch.empty_like(w) for w in want]
    q8 = torch.empty(rows * (K // 32) * 36, dtype=torch.uint8, device=cuda)
    P, I = (lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else 0)), ctypes.c_int
    st = ctypes.c_void_p(torch.cuda.current_stream(cuda).cuda_stream)

    def apart(mode, inp, norm, ws, residual, outs):
        ws, outs = list(ws) + [None] * (3 - len(ws)), list(outs) + [None] * (3 - len(outs))
        n = [0 if w is None else w.shape[0] for w in ws]
        assert lib().mrs_rms_quantize_q8_1(I(1), P(inp), P(norm), ctypes.c_float(1e-5), I(K), I(rows), P(q8), I(pdl), st) == 0
        assert lib().mrs_mmvq_q8(I(GGML[dtype]), I(mode), I(1), *(P(w.data if w is not None else None) for w in ws), P(q8), P(residual),
                                 *(P(o) for o in outs), I(K), *(I(v) for v in n), I(rows), I(0), I(pdl), st) == 0

    for _ in range(3):
        apart(2, x, nw, (wq, wk, wv), None, got[:3])
        apart(1, h, nw, (gate, up), None, got[3:4])
        apart(0, h, None, (wo,), res, got[4:])
    torch.cuda.synchronize()
    assert all(torch.equal(g, w) for g, w in zip(got, want))


@pytest.mark.parametrize("K,N", [(4096, 64), (5120, 64), (6144, 4096), (8192, 64)])
def test_one_row_captured_and_not(cuda, K, N):
    """In a graph long rows of few results take the two launches, outside one launch: the same bits."""
    ws = [quant.QTensor(to_dev(make_weight("q4_k", N, K, i).reshape(-1), cuda), "q4_k", (N, K)) for i in range(3)]
    x = torch.randn(1, K, device=cuda, generator=torch.Generator(device=cuda).manual_seed(K)).to(torch.bfloat16)
    call = lambda: [quant.plain(ws[0], x), quant.fused_glu(ws[0], ws[1], x, quant.GluActivationType.Silu), *quant.fused_qkv(*ws, x)]
    want = call()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = call()
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("dtype,N,K", [("q4_k", 6501, 2304), ("q4_k", 4100, 2304), ("q5_k", 5297, 2304), ("q6_k", 4450, 2304), ("q8_0", 8193, 1024), ("q4_k", 1100, 14336),
                                       ("q6_k", 1000, 11008), ("q8_0", 34000, 256)])
@pytest.mark.parametrize("rows", [3, 4, 5, 8])
def test_large_matrices_on_tensor_cores(cuda, dtype, rows, N, K):
    """Three (Q8_0: five) to eight rows over at least 5 MB of weights: integer products on the tensor cores against the vector kernel in every mode.  Integer dots
    and their scales are exact in both; f32 sums of at most K / 16 terms in two orders, whose parts stay within 16 of the largest result, differ
    by less than K x 2^-24 of that."""
    import ctypes
    from mistralrs_b200 import lib
    gen = torch.Generator(device=cuda).manual_seed(N)
    weight = lambda n, seed: quant.QTensor(to_dev(make_weight(dtype, n, K, seed).reshape(-1), cuda), dtype, (n, K))
    x = torch.randn(rows, K, device=cuda, generator=gen)
    ws = [weight(N, 1), weight(N, 2), weight(N - 7, 3)]
    call = lambda t: [quant.plain(ws[0], t), *quant.fused_qkv(*ws, t), quant.fused_glu(ws[0], ws[1], t, quant.GluActivationType.Relu)]
    results = []
    try:
        for flags in (16, 0):
            lib().mrs_set_mmvq_flags(ctypes.c_int(flags))
            results.append((call(x), call(x.to(torch.bfloat16))))
    finally:
        lib().mrs_set_mmvq_flags(ctypes.c_int(0))
    (want, want16), (got, got16) = results
    assert all(torch.equal(a, b) for a, b in zip(got, want)) == (dtype == "q8_0" and rows < 5)        # two kernels
    top = [w.abs().max() for w in want]
    for a, b, s in zip(got, want, [*top[:4], 2 * top[1] * top[2]]):
        assert ((a - b).abs() <= K * 2.0 ** -24 * s).all()
    for a, b in zip(got16, want16):           # the same rounding but where a sum lies at its edge
        assert ((a - b).abs() <= 2.0 ** -6 * b.abs().max()).all() and (a != b).float().mean() < 2e-2
    assert lib().mrs_mmq_timeouts() == 0


def test_tensor_core_calls_are_refused_once_a_wait_has_run_out(cuda):
    """The word that a kernel sets when a wait runs out, set here by the host: three to eight rows over 5 MB of weights and prompt attention, whose
    kernels set it too, refuse as the dequantising GEMM does; what runs on kernels without it (a row, small matrices, softcap) goes on."""
    import ctypes
    from mistralrs_b200 import lib, mmq, paged_attn
    weight = lambda n, k: quant.QTensor(to_dev(make_weight("q4_k", n, k, 1).reshape(-1), cuda), "q4_k", (n, k))
    large, small = weight(4608, 2304), weight(64, 256)
    gen = torch.Generator(device=cuda).manual_seed(1)
    x, y = torch.randn(4, 2304, device=cuda, generator=gen), torch.randn(4, 256, device=cuda, generator=gen)
    q = {d: torch.randn(70, 2, d, device=cuda, generator=gen).to(torch.float16) for d in (64, 128)}
    refused = [lambda: quant.plain(large, x), lambda: quant.fused_glu(large, large, x, quant.GluActivationType.Silu),
               lambda: quant.fused_qkv(large, large, large, x)[0], lambda: paged_attn.prefill_attention(q[64], q[64], q[64], 0.125),
               lambda: paged_attn.prefill_attention(q[128], q[128], q[128], 0.1, window_left=20)]
    go_on = [lambda: quant.plain(large, x[:2]), lambda: quant.plain(small, y), lambda: paged_attn.prefill_attention(q[64], q[64], q[64], 0.125, softcap=20.0)]
    want = [[call() for call in calls] for calls in (refused, go_on)]
    assert lib().mrs_mmq_timeouts() == 0
    fn = lib().mrs_mmq_timeout_flag
    fn.restype = ctypes.POINTER(ctypes.c_int32)
    flag = fn()
    try:
        flag[0] = 1
        for call in refused:
            with pytest.raises(RuntimeError, match="702"):
                call()
        assert all(torch.equal(call(), w) for call, w in zip(go_on, want[1]))
        with pytest.raises(RuntimeError, match="ran out"):
            mmq.check_timeouts(cuda)
    finally:
        flag[0] = 0
    assert all(torch.equal(call(), w) for call, w in zip(refused, want[0]))


@pytest.mark.parametrize("dt", ["bf16", "f16", "f32"])
@pytest.mark.parametrize("dtype,N", [(t, 70) for t in ALL_TYPES] + [("q4_k", 4300), ("q5_k", 3500), ("q6_k", 2900), ("q8_0", 2300), ("q3_k", 5400)])
def test_reference_shaped_launchers(cuda, dtype, N, dt):
    """launch_mmvq_gguf_<type>_<dtype>_{plain,fused_glu,fused_qkv} as a caller of the C symbols has them: activation rows padded to 512 columns, results
    with a stride of their own, one to eight rows, below and above 5 MB.  The bits of the Python calls; those against the oracle elsewhere here."""
    import ctypes
    from mistralrs_b200 import lib
    K = 2304
    gen = torch.Generator(device=cuda).manual_seed(N)
    weight = lambda n, seed: quant.QTensor(to_dev(make_weight(dtype, n, K, seed).reshape(-1), cuda), dtype, (n, K))  # noqa: E731
    ws = [weight(N, 1), weight(N, 2), weight(N - 7, 3)]
    P, I = lambda t: ctypes.c_void_p(t.data_ptr()), ctypes.c_int  # noqa: E731
    entry = lambda kind: getattr(lib(), f"launch_mmvq_gguf_{dtype}_{dt}_{kind}")  # noqa: E731
    stream = ctypes.c_void_p(torch.cuda.current_stream(cuda).cuda_stream)
    for rows in range(1, 9):
        x = torch.randn(rows, K, device=cuda, generator=gen).to({"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}[dt])
        y, stride = quant.quantize_q8_1(x), 2560 // 32
        plain, glu = (torch.full((rows, N + 5), -77.0, dtype=x.dtype, device=cuda) for _ in range(2))
        qkv = [torch.empty(rows, w.shape[0], dtype=x.dtype, device=cuda) for w in ws]
        entry("plain")(P(ws[0].data), P(y), P(plain), I(K), I(N), I(stride), I(N + 5), I(rows), stream)
        entry("fused_glu")(P(ws[0].data), P(ws[1].data), P(y), P(glu), I(K), I(N), I(stride), I(N + 5), I(rows), I(0), stream)
        entry("fused_qkv")(*(P(w.data) for w in ws), P(y), *(P(o) for o in qkv), I(K), *(I(w.shape[0]) for w in ws), I(stride), I(rows), stream)
        assert torch.equal(plain[:, :N], quant.plain(ws[0], x)) and bool((plain[:, N:] == -77.0).all()), rows
        assert torch.equal(glu[:, :N], quant.fused_glu(ws[0], ws[1], x, quant.GluActivationType.Silu)) and bool((glu[:, N:] == -77.0).all()), rows
        assert all(torch.equal(a, b) for a, b in zip(qkv, quant.fused_qkv(*ws, x))), rows
    assert lib().mrs_mmq_timeouts() == 0


@pytest.mark.parametrize("dtype,N,K", [("q4_k", 4300, 2304), ("q5_k", 3500, 2304), ("q6_k", 2900, 2304), ("q6_k", 1000, 11008), ("q8_0", 2300, 2304)])
@pytest.mark.parametrize("dt", ["f32", "bf16"])
def test_tensor_core_rows_with_a_residual_against_the_oracle(cuda, dtype, N, K, dt):
    """mmvq_mma_kernel on its own oracle, with the residual of a decode step's projections: the oracle's integer dots to 5e-6 in f32 (as the vector
    kernel); in bf16 the product is rounded, and again after the residual is added."""
    import ctypes
    from mistralrs_b200 import GGML, lib
    wb = make_weight(dtype, N, K, 5)
    w = to_dev(wb.reshape(-1), cuda)
    P, I = lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else 0), ctypes.c_int  # noqa: E731
    stream = ctypes.c_void_p(torch.cuda.current_stream(cuda).cuda_stream)
    code = {"f32": 2, "bf16": 1}[dt]
    for rows in (3, 5, 8):
        y = quant.quantize_q8_1(to_dev(make_acts(rows, K, 6 + rows, dt), cuda, dt), k_padded=K)
        ref = oracle.mmvq_q8_1(dtype, wb, y.cpu().numpy(), K, N, K // 32, rows)      # (over the rows as quantised: 16-bit inputs have ties)
        scale = np.abs(ref).max()
        residual = to_dev((np.random.default_rng(rows).standard_normal((rows, N)) * scale).astype(np.float32), cuda, dt)
        for add in (None, residual):
            out = torch.empty(rows, N, dtype=residual.dtype, device=cuda)
            assert lib().mrs_mmvq_q8(I(GGML[dtype]), I(0), I(code), P(w), P(None), P(None), P(y), P(add), P(out), P(None), P(None), I(K), I(N), I(0), I(0),
                                     I(rows), I(0), I(0), stream) == 0
            want = ref + (0 if add is None else add.double().cpu().numpy())
            err = np.abs(out.double().cpu().numpy() - want)
            step = 0.0 if dt == "f32" else 2.0 ** -8 * (np.abs(want) + (0 if add is None else np.abs(ref)))      # half a place of each rounding, and more
            assert (err <= 5e-6 * scale + 2.0 ** -23 * np.abs(want) + step).all(), (rows, add is None, err.max())
