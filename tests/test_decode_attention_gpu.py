"""Decode attention over the HND cache whose products have tokens as rows (up to eight heads a KV head) against attention in 64 bits."""
import numpy as np
import pytest
import torch

from mistralrs_b200 import kv_index, paged_attn

pytestmark = pytest.mark.gpu


def _reference(q, k, v, scale, window, cap):
    """q [H, D], k, v [T, KVH, D]: the query is the last token."""
    H, T = q.shape[0], k.shape[0]
    per = H // k.shape[1]
    out = torch.empty_like(q, dtype=torch.float64)
    j = torch.arange(T, device=q.device)
    for h in range(H):
        s = k[:, h // per].double() @ q[h].double() * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if window is not None:
            s = s.masked_fill(j < T - 1 - window, -torch.inf)
        out[h] = torch.softmax(s, -1) @ v[:, h // per].double()
    return out


@pytest.mark.parametrize("dt,tol", [(torch.bfloat16, 2.0 ** -7), (torch.float16, 2.0 ** -10)])
@pytest.mark.parametrize("group,dim", [(1, 128), (2, 64), (3, 128), (4, 128), (6, 64), (8, 128), (16, 64)])
@pytest.mark.parametrize("page,window,cap", [(16, None, None), (8, None, None), (24, None, 30.0), (48, 70, None), (32, 100, None)])
def test_decode_attention(cuda, dt, tol, group, dim, page, window, cap):
    """Ends of a warp's 16 and a step's 64 tokens, whole pages and parts of them (16 tokens within one or not), windows that begin inside a page, few and
    many tiles (pairs of CTAs and single ones).  Three roundings of 2^-9 (f16 2^-12) a value, probabilities, tiles' results and results: four times that."""
    g = torch.Generator(device="cuda").manual_seed(7 * group + page)
    for lens, split in (([1, 15, 16, 17, 63, 64, 65, 129], 0), ([300, 1, 640, 97], 4), ([1500] * 40 + [33], 8)):
        kv = 2
        pages = [-(-n // page) for n in lens]
        order = (1 + torch.randperm(sum(pages), generator=torch.Generator().manual_seed(3))).tolist()
        tables, at = [], 0
        for n in pages:
            tables.append(order[at:at + n])
            at += n
        tiles = sum(-(-n // split) if split else 1 for n in pages)
        meta = [torch.from_numpy(np.ascontiguousarray(m)).to(cuda) for m in
                (*kv_index.make_paged_kv_tensors(tables, lens, page, sum(pages)), *kv_index.make_paged_kv_decode_tensors(tables, lens, page, split, tiles))]
        k, v = (torch.randn(sum(pages) + 1, kv, page, dim, device=cuda, generator=g).to(dt) for _ in range(2))
        k[0], v[0] = float("nan"), float("nan")                 # no sequence's page
        q = torch.randn(len(lens), kv * group, dim, device=cuda, generator=g).to(dt)
        out = paged_attn.flashinfer_decode(q, k, v, *meta, dim ** -0.5, window_left=window, logits_soft_cap=cap)
        for b in (range(len(lens)) if len(lens) < 10 else (0, 39, 40)):
            rows = [t[torch.tensor(tables[b], device=cuda)].transpose(1, 2).reshape(-1, kv, dim)[:lens[b]] for t in (k, v)]
            want = _reference(q[b], *rows, dim ** -0.5, window, cap)
            assert float((out[b].double() - want).norm() / want.norm()) <= tol, (lens[b], split)


def test_infinite_and_masked_scores(cuda):
    """Keys that give scores of -inf weigh nothing; a NaN in a key stays in its own sequence (whose sums are then not above zero: results of zero, as ever)."""
    page, dim = 16, 128
    tables, lens = [[1, 2], [3, 4]], [30, 30]
    meta = [torch.from_numpy(np.ascontiguousarray(m)).to(cuda) for m in
            (*kv_index.make_paged_kv_tensors(tables, lens, page, 4), *kv_index.make_paged_kv_decode_tensors(tables, lens, page, 0, 2))]
    g = torch.Generator(device="cuda").manual_seed(1)
    k, v = (torch.randn(5, 1, page, dim, device=cuda, generator=g).to(torch.bfloat16) for _ in range(2))
    q = torch.rand(2, 4, dim, device=cuda, generator=g).to(torch.bfloat16) + 0.5
    k[1, 0, 3] = float("-inf")
    k[3, 0, 2] = float("nan")
    out = paged_attn.flashinfer_decode(q, k, v, *meta, dim ** -0.5)
    keep = torch.tensor([i for i in range(30) if i != 3], device=cuda)
    rows = [t[torch.tensor([1, 2], device=cuda)].transpose(1, 2).reshape(-1, 1, dim)[keep] for t in (k, v)]
    want = _reference(q[0], *rows, dim ** -0.5, None, None)
    assert float((out[0].double() - want).norm() / want.norm()) <= 2.0 ** -7
    assert not bool(out[1].any())
