"""Prompt attention kernels (csrc/prefill_attn_tc.cu, csrc/prefill_attn.cu) vs a plain fp64 torch reference of the same op:
causal, GQA, ragged lengths, var-len batches, sliding window, soft-cap, both dtypes and head sizes."""
import numpy as np
import pytest
import torch

from mistralrs_b200 import paged_attn

pytestmark = pytest.mark.gpu


def _ref(q, k, v, scale, causal, window=None, softcap=None):
    T, H, D = q.shape
    g = H // k.shape[1]
    qq, kk, vv = q.double(), k.double().repeat_interleave(g, dim=1), v.double().repeat_interleave(g, dim=1)
    s = torch.einsum("thd,jhd->htj", qq, kk) * scale
    if softcap:
        s = softcap * torch.tanh(s / softcap)
    i = torch.arange(T, device=q.device)
    mask = torch.ones(T, T, dtype=torch.bool, device=q.device)
    if causal:
        mask &= i[None, :] <= i[:, None]
    if window is not None:
        mask &= i[None, :] >= i[:, None] - window
    s = s.masked_fill(~mask[None], float("-inf"))
    return torch.einsum("htj,jhd->thd", torch.softmax(s, dim=-1), vv)


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,H,KVH,D", [(37, 4, 2, 128), (128, 8, 2, 64), (333, 8, 8, 128), (1100, 4, 1, 128)])
def test_causal_matches_reference(cuda, dt, T, H, KVH, D):
    gen = torch.Generator(device=cuda).manual_seed(T)
    q = torch.randn(T, H, D, device=cuda, generator=gen).to(dt)
    k = torch.randn(T, KVH, D, device=cuda, generator=gen).to(dt)
    v = torch.randn(T, KVH, D, device=cuda, generator=gen).to(dt)
    scale = 1.0 / np.sqrt(D)
    got = paged_attn.prefill_attention(q, k, v, scale).double()
    want = _ref(q, k, v, scale, True)
    ulp = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11
    # P is rounded to the activation dtype before PV (as flash-attention does) + one output rounding
    assert (got - want).abs().max().item() <= 3 * ulp * want.abs().max().item() + 1e-6


def test_window_softcap_noncausal(cuda):
    T, H, KVH, D = 300, 4, 2, 128
    gen = torch.Generator(device=cuda).manual_seed(1)
    q, k, v = (torch.randn(T, h, D, device=cuda, generator=gen).to(torch.bfloat16) for h in (H, KVH, KVH))
    scale = 1.0 / np.sqrt(D)
    for kw, ref_kw in ((dict(window_left=70), dict(causal=True, window=70)), (dict(softcap=20.0), dict(causal=True, softcap=20.0)),
                       (dict(causal=False), dict(causal=False))):
        got = paged_attn.prefill_attention(q, k, v, scale, **kw).double()
        want = _ref(q, k, v, scale, **ref_kw)
        assert (got - want).abs().max().item() <= 3 * 2.0 ** -8 * want.abs().max().item(), kw


def test_varlen_batch(cuda):
    lens = [5, 130, 64, 257]
    H, KVH, D = 8, 2, 128
    T = sum(lens)
    gen = torch.Generator(device=cuda).manual_seed(2)
    q, k, v = (torch.randn(T, h, D, device=cuda, generator=gen).to(torch.bfloat16) for h in (H, KVH, KVH))
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device=cuda)
    scale = 1.0 / np.sqrt(D)
    got = paged_attn.prefill_attention(q, k, v, scale, cu_seqlens=cu, max_seqlen=max(lens)).double()
    off = 0
    for L in lens:
        want = _ref(q[off:off + L], k[off:off + L], v[off:off + L], scale, True)
        assert (got[off:off + L] - want).abs().max().item() <= 3 * 2.0 ** -8 * want.abs().max().item()
        off += L


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_both_kernels_head_128(cuda, dt):
    """Head sizes 64 and 128 without softcap run on csrc/prefill_attn_tc.cu (tcgen05, S and P in tensor memory);
    mrs_prefill_attn_tc_debug(0, ...) keeps the call on csrc/prefill_attn.cu (mma.sync).  Both against the fp64
    reference, on a ragged multi-tile prompt, causal and not."""
    import ctypes
    from mistralrs_b200 import lib
    T, H, KVH, D = 700, 8, 2, 128
    gen = torch.Generator(device=cuda).manual_seed(9)
    q, k, v = (torch.randn(T, h, D, device=cuda, generator=gen).to(dt) for h in (H, KVH, KVH))
    scale = 1.0 / np.sqrt(D)
    ulp = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11
    try:
        for enable in (0, 1):
            lib().mrs_prefill_attn_tc_debug(ctypes.c_int32(enable), ctypes.c_uint32(0), ctypes.c_uint32(0))
            for causal in (True, False):
                got = paged_attn.prefill_attention(q, k, v, scale, causal=causal).double()
                want = _ref(q, k, v, scale, causal)
                assert torch.isfinite(got).all()
                assert (got - want).abs().max().item() <= 3 * ulp * want.abs().max().item() + 1e-6, (enable, causal)
    finally:
        lib().mrs_prefill_attn_tc_debug(ctypes.c_int32(1), ctypes.c_uint32(0), ctypes.c_uint32(0))


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D,H,KVH", [(64, 14, 2), (128, 6, 2)])
@pytest.mark.parametrize("T", [1, 127, 128, 129, 400])
def test_tensor_memory_kernel_windows_and_head_64(cuda, dt, D, H, KVH, T):
    """Windows and head size 64 on csrc/prefill_attn_tc.cu, at the edges of its tiles of 128 queries and 128 keys, from slices of one packed
    q / k / v buffer, against the fp64 reference: 3 ulp as above (P and the result are each rounded once)."""
    gen = torch.Generator(device=cuda).manual_seed(T + D)
    qkv = torch.randn(T, (H + 2 * KVH) * D, device=cuda, generator=gen).to(dt)
    q, k, v = (t.unflatten(1, (-1, D)) for t in qkv.split([H * D, KVH * D, KVH * D], 1))
    scale = 1.0 / np.sqrt(D)
    ulp = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11
    for causal in (True, False):
        for window in (None, 0, 1, 127, 128, 129, 2 ** 31 - 1):
            got = paged_attn.prefill_attention(q, k, v, scale, causal=causal, window_left=window).double()
            want = _ref(q, k, v, scale, causal, window=window)
            assert (got - want).abs().max().item() <= 3 * ulp * want.abs().max().item() + 1e-6, (causal, window)


@pytest.mark.parametrize("D,window", [(64, None), (64, 50), (128, None), (128, 50)])
def test_sequences_do_not_see_their_neighbours(cuda, D, window):
    """A last tile reaches into the next sequence's rows: what stands there, finite or not, leaves no trace."""
    lens, H, KVH = [70, 128, 0, 200, 5], 4, 2
    gen = torch.Generator(device=cuda).manual_seed(4)
    q, k, v = (torch.randn(sum(lens), h, D, device=cuda, generator=gen).to(torch.bfloat16) for h in (H, KVH, KVH))
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device=cuda)
    run = lambda kk, vv: paged_attn.prefill_attention(q, kk, vv, D ** -0.5, cu_seqlens=cu, max_seqlen=max(lens), window_left=window)  # noqa: E731
    clean = run(k, v)
    for keep in range(len(lens)):
        at = slice(int(cu[keep]), int(cu[keep + 1]))
        kk, vv = torch.full_like(k, float("nan")), torch.full_like(v, float("inf"))
        kk[at], vv[at] = k[at], v[at]
        assert torch.equal(run(kk, vv)[at], clean[at])


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("varlen", [False, True])
def test_values_outside_the_window_of_a_tile_leave_no_trace(cuda, D, varlen):
    """Keys that no row of a tile of 128 queries may see, before its windows or behind its last row, are not multiplied: infinite values there change
    no bit, wherever the windows start."""
    T, H, KVH = 300, 4, 2
    gen = torch.Generator(device=cuda).manual_seed(D)
    q, k, v = (torch.randn(T, h, D, device=cuda, generator=gen).to(torch.bfloat16) for h in (H, KVH, KVH))
    kw = dict(cu_seqlens=torch.tensor([0, T], dtype=torch.int32, device=cuda), max_seqlen=T) if varlen else {}
    for window in (0, 1, 40, 64, 100, 127):
        run = lambda vv: paged_attn.prefill_attention(q, k, vv, D ** -0.5, window_left=window, **kw)  # noqa: E731
        clean, vv = run(v), v.clone()
        vv[:128 - window] = float("inf")      # (of the second tile's rows, 128 .. 255)
        vv[256:] = float("nan")
        assert torch.equal(run(vv)[128:256], clean[128:256]), window


@pytest.fixture(params=[0, 1], ids=["mma.sync", "tcgen05"])
def either_kernel(request):
    """Both prompt kernels for what both take (softcap runs on csrc/prefill_attn.cu whatever is asked for)."""
    import ctypes
    from mistralrs_b200 import lib
    lib().mrs_prefill_attn_tc_debug(ctypes.c_int32(request.param), ctypes.c_uint32(0), ctypes.c_uint32(0))
    yield
    lib().mrs_prefill_attn_tc_debug(ctypes.c_int32(1), ctypes.c_uint32(0), ctypes.c_uint32(0))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_ragged_batches_windows_and_softcap_on_either_kernel(cuda, either_kernel, dt, D):
    """Sequences of several lengths (one of them empty) with every pair of window and softcap, causal and not, on each kernel: 3 ulp as above."""
    lens, H, KVH = [5, 130, 0, 64, 257], 6, 2
    gen = torch.Generator(device=cuda).manual_seed(D)
    q, k, v = (torch.randn(sum(lens), h, D, device=cuda, generator=gen).to(dt) for h in (H, KVH, KVH))
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device=cuda)
    scale, ulp = D ** -0.5, 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11
    for causal in (True, False):
        for window in (None, 0, 63, 70, 128):
            for softcap in (None, 20.0):
                got = paged_attn.prefill_attention(q, k, v, scale, causal=causal, cu_seqlens=cu, max_seqlen=max(lens), window_left=window, softcap=softcap).double()
                for a, b in zip(cu[:-1].tolist(), cu[1:].tolist()):
                    if a < b:
                        want = _ref(q[a:b], k[a:b], v[a:b], scale, causal, window, softcap)
                        assert (got[a:b] - want).abs().max().item() <= 3 * ulp * want.abs().max().item() + 1e-6, (causal, window, softcap, b - a)
