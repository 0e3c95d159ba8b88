"""Small-batch W4A16 (csrc/w4a16.cu) behind the reference's Marlin symbols: `gptq_marlin_repack` /
`awq_marlin_repack` + `marlin_{gptq,awq}_4bit_{f16,bf16}` driven exactly as `gptq_linear` /
`marlin_matmul` drive them (repack, marlin_permute_scales, forward), against the numpy oracle
(oracle/gptq.py) — and, in test_ref_golden_gpu.py, against the reference's own Marlin kernel."""
import numpy as np
import pytest
import torch

from oracle import gptq as og
from mistralrs_b200 import gptq

pytestmark = pytest.mark.gpu


def _mk(K, N, group, seed):
    rng = np.random.default_rng(seed)
    q = rng.integers(0, 16, size=(K, N))
    g = K if group == -1 else group
    scales = np.exp2(rng.uniform(-8, -6, size=(K // g, N))).astype(np.float16)
    return rng, q, scales, g


def _tol(ref, x, wd, ulp):
    mag = np.abs(x.astype(np.float64)) @ np.abs(wd).astype(np.float64)
    return ulp * np.abs(ref) * 1.01 + 2e-6 * mag + 1e-6


@pytest.mark.parametrize("M", [1, 7, 32, 33, 64, 100, 300])
def test_gptq_marlin_boundary_batches(cuda, M):
    K, N, group = 1024, 576, 128          # 4.5 row tiles (ragged last tile), split-K over a cluster
    rng, q, scales, g = _mk(K, N, group, 1)
    qweight = og.pack_gptq(q)
    x = rng.standard_normal((M, K)).astype(np.float16)
    layer = gptq.GptqMarlinLayer(torch.from_numpy(qweight).to(cuda), torch.from_numpy(scales).to(cuda), group_size=group)
    y = layer.forward_raw(torch.from_numpy(x).to(cuda)).float().cpu().numpy()
    wd = og.dequant_gptq(qweight, scales, None, g)
    ref = og.gemm(x, wd)
    tol = _tol(ref, x, wd, 2.0 ** -11)
    assert (np.abs(y - ref) <= tol).all(), float((np.abs(y - ref) / tol).max())


@pytest.mark.parametrize("K,N,group", [(4096, 4096, 128), (512, 256, 32), (1024, 192, 64), (2048, 128, -1), (14336, 256, 128)])
def test_gptq_marlin_shapes_and_groups(cuda, K, N, group):
    M = 32
    rng, q, scales, g = _mk(K, N, group, 3)
    qweight = og.pack_gptq(q)
    x = (0.5 * rng.standard_normal((M, K))).astype(np.float16)
    layer = gptq.GptqMarlinLayer(torch.from_numpy(qweight).to(cuda), torch.from_numpy(scales).to(cuda), group_size=group)
    y = layer.forward_raw(torch.from_numpy(x).to(cuda)).float().cpu().numpy()
    wd = og.dequant_gptq(qweight, scales, None, g)
    ref = og.gemm(x, wd)
    tol = _tol(ref, x, wd, 2.0 ** -11)
    assert (np.abs(y - ref) <= tol).all(), float((np.abs(y - ref) / tol).max())


def test_gptq_act_order_follows_the_reference_flow(cuda):
    # desc_act checkpoints: the reference sorts the weight rows by group (perm = argsort(g_idx)) at
    # repack time and runs Marlin with contiguous groups on the UNPERMUTED activations
    # (gptq_cuda.rs:573-590, marlin_backend.rs): y = x . W[perm] with scales[k' / group]
    K, N, group, M = 1024, 256, 128, 16
    rng, q, scales, g = _mk(K, N, group, 5)
    g_idx = (rng.permutation(K) // group).astype(np.int32)
    qweight = og.pack_gptq(q)
    x = rng.standard_normal((M, K)).astype(np.float16)
    layer = gptq.GptqMarlinLayer(torch.from_numpy(qweight).to(cuda), torch.from_numpy(scales).to(cuda),
                                 g_idx=torch.from_numpy(g_idx).to(cuda), group_size=group)
    y = layer.forward_raw(torch.from_numpy(x).to(cuda)).float().cpu().numpy()
    perm = np.argsort(g_idx, kind="stable")
    wd = ((q[perm] - 8).astype(np.float32) * scales.astype(np.float32)[np.arange(K) // group]).astype(np.float16).astype(np.float32)
    ref = og.gemm(x, wd)
    tol = _tol(ref, x, wd, 2.0 ** -11)
    assert (np.abs(y - ref) <= tol).all(), float((np.abs(y - ref) / tol).max())


@pytest.mark.parametrize("K,N,group,M", [(512, 384, 128, 40), (448, 160, 64, 9), (1152, 320, 32, 32), (4096, 1024, 128, 32)])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_awq_marlin_boundary(cuda, dt, K, N, group, M):
    """zero points + scale rows staged per iteration: several groups per 128-k iteration (32, 64), a K tail of
    one 64-k chunk (448, 1152 % 128 == 64... 1152 = 9 x 128), ragged last row tile (160, 320; N stays a multiple of the scale permutation width the layer applies), split-K (4096)"""
    rng, q, scales, g = _mk(K, N, group, 2)
    z = rng.integers(0, 16, size=(K // group, N))
    qweight, qzeros = og.pack_awq(q), og.pack_awq(z)
    x = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float32)).to(cuda).to(dt)
    layer = gptq.GptqMarlinLayer(torch.from_numpy(qweight).to(cuda), torch.from_numpy(scales).to(cuda),
                                 qzeros=torch.from_numpy(qzeros).to(cuda), group_size=group, is_awq=True)
    y = layer.forward_raw(x).float().cpu().numpy()
    xs = x.float().cpu().numpy()
    sc = scales if dt == torch.float16 else torch.from_numpy(scales).to(torch.bfloat16).float().numpy()
    gidx = np.arange(K) // group
    wd = (q - z[gidx]).astype(np.float32) * sc.astype(np.float32)[gidx]
    wd = torch.from_numpy(wd).to(dt).float().numpy()           # one rounding of the dequantised weight in dt
    ref = xs.astype(np.float64) @ wd.astype(np.float64)
    ulp = 2.0 ** -11 if dt == torch.float16 else 2.0 ** -8
    tol = _tol(ref, xs, wd, ulp)
    assert (np.abs(y - ref) <= tol).all(), float((np.abs(y - ref) / tol).max())


@pytest.mark.parametrize("M,N,K", [(32, 32000, 4096), (5, 200, 512), (130, 384, 1024)])
def test_dense_linear(cuda, M, N, K):
    rng = np.random.default_rng(7)
    x = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float32)).to(cuda).to(torch.float16)
    w = torch.from_numpy((0.05 * rng.standard_normal((N, K))).astype(np.float32)).to(cuda).to(torch.float16)
    y = gptq.dense_linear(x, w).float()
    ref = x.double() @ w.double().t()
    mag = x.double().abs() @ w.double().abs().t()
    tol = 2.0 ** -11 * ref.abs() * 1.01 + 2e-6 * mag + 1e-6
    assert bool(((y.double() - ref).abs() <= tol).all()), float(((y.double() - ref).abs() / tol).max())


@pytest.mark.parametrize("K,N,group", [(64, 64, 32), (1024, 192, 128), (512, 128, 512), (4096, 1088, 64)])
@pytest.mark.parametrize("awq", [False, True])
def test_scales_in_the_other_format(cuda, awq, K, N, group):
    """f16 scales under bf16 rows and bf16 scales under f16 rows: bit for bit what scales rounded before the call give."""
    gen = torch.Generator(device=cuda).manual_seed(K + N)
    ints = lambda *shape: torch.randint(-2 ** 31, 2 ** 31, shape, dtype=torch.int32, device=cuda, generator=gen)  # noqa: E731
    qweight = ints(K, N // 8) if awq else ints(K // 8, N)
    scales = torch.rand(K // group, N, device=cuda, generator=gen) * 0.02 + 1e-3
    scales[0, :4] = torch.tensor([0.0, 6e-8, -3e-5, 1.5], device=cuda)
    for rows, other in ((torch.bfloat16, torch.float16), (torch.float16, torch.bfloat16)):
        layer = gptq.GptqMarlinLayer(qweight, scales.to(other), ints(K // group, N // 8) if awq else None, group_size=group, is_awq=awq)
        for M in (1, 17, 130):
            x = torch.randn(M, K, device=cuda, generator=gen).to(rows)
            got, kept = layer.forward_raw(x), layer.scales
            layer.scales = kept.to(rows)
            want = layer.forward_raw(x)
            layer.scales = kept
            assert torch.equal(got.view(torch.int16), want.view(torch.int16))


def test_scale_columns_other_than_permuted_are_plain(cuda):
    """mrs_w4a16_gemm and its link of a launch chain: scale_perm 1 and 2 are permutations, every other value has always meant plain columns."""
    import ctypes
    from mistralrs_b200 import lib
    K, N, M = 512, 128, 20
    gen = torch.Generator(device=cuda).manual_seed(1)
    qweight = torch.randint(-2 ** 31, 2 ** 31, (K // 8, N), dtype=torch.int32, device=cuda, generator=gen)
    scales = (torch.rand(K // 128, N, device=cuda, generator=gen) * 0.02 + 1e-3).to(torch.float16)
    layer = gptq.GptqMarlinLayer(qweight, scales, group_size=128)
    x = torch.randn(M, K, device=cuda, generator=gen).to(torch.float16)
    P, I = lambda t: ctypes.c_void_p(t.data_ptr()), ctypes.c_int  # noqa: E731
    stream = ctypes.c_void_p(torch.cuda.current_stream(cuda).cuda_stream)

    def call(perm, link):
        y = torch.empty(M, N, dtype=torch.float16, device=cuda)
        args = (P(x), P(layer.q_weight), P(scales), ctypes.c_void_p(0), P(y), I(M), I(K), I(N), I(128), I(0), I(perm))
        assert (lib().mrs_w4a16_gemm_pdl(*args, I(0), stream) if link else lib().mrs_w4a16_gemm(*args, stream)) == 0
        return y
    want = call(0, False)
    assert all(torch.equal(call(perm, link), want) for perm in (3, 4, 7, 8, -1) for link in (False, True))
    assert not torch.equal(call(1, False), want) and not torch.equal(call(2, True), want)
