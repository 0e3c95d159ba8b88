"""Several matrices that read the same activations as one launch of the dequantising GEMM (`mmq.forward_many`) against one launch each."""
import ctypes

import pytest
import torch

from mistralrs_b200 import BLOCK_BYTES, BLOCK_ELEMS, GGML, lib, mmq, quant

pytestmark = pytest.mark.gpu

F16_AT = {"q4_k": (0, 2), "q5_k": (0, 2), "q6_k": (208,), "q8_0": (0,), "q4_0": (0,)}


def _matrix(kind, rows, cols, cuda, g):
    raw = torch.randint(0, 256, (rows * cols // BLOCK_ELEMS[kind], BLOCK_BYTES[kind]), dtype=torch.uint8, device=cuda, generator=g)
    for at in F16_AT[kind]:
        d = torch.rand(raw.shape[0], device=cuda, generator=g) * 1e-3
        raw[:, at:at + 2] = d.to(torch.float16).view(torch.uint8).view(-1, 2)
    return quant.QTensor(raw.view(-1), kind, (rows, cols))


def _entry(ws, x):
    """The C entry's answer for these matrices (0: one launch)."""
    ys = [torch.empty(x.shape[0], w.shape[0], dtype=x.dtype, device=x.device) for w in ws]
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    n = [w.shape[0] for w in ws] + [0]
    rc = lib().mrs_mmq_gguf_multi(ctypes.c_int32(GGML[ws[0].dtype]), p(ws[0].data), p(ws[1].data), p(ws[2].data) if len(ws) > 2 else None, p(x), p(ys[0]), p(ys[1]),
                                  p(ys[2]) if len(ws) > 2 else None, *(ctypes.c_int32(v) for v in (x.shape[0], n[0], n[1], n[2], x.shape[1],
                                                                                                1 if x.dtype == torch.bfloat16 else 0)),
                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return rc, ys


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind", ["q4_k", "q5_k", "q6_k", "q8_0"])
@pytest.mark.parametrize("rows,cols", [((1024, 128, 128), 2048), ((1000, 129, 1), 2048), ((2048, 1024), 4096), ((96, 4096, 1300), 2048), ((1536, 1536), 2304)])
def test_many_equal_one_by_one(cuda, kind, dt, rows, cols):
    """Row tiles that end inside a matrix, matrices of one tile, K whole and split over clusters, several token tiles.  Where neither splits K: the same bits.
    Else f32 sums in another order, which turn a rounding of the result here and there: well below 2^-10 of its norm."""
    if kind == "q6_k" and cols % 2048:
        cols = 4096                                  # (rows of a multiple of 16 bytes)
    g = torch.Generator(device=cuda).manual_seed(len(rows) * cols + rows[0])
    ws = [_matrix(kind, r, cols, cuda, g) for r in rows]
    for tokens in (9, 16, 17, 100, 250, 300):
        x = torch.randn(tokens, cols, device=cuda, generator=g).to(dt)
        rc, ys = _entry(ws, x)
        assert rc == 0 or (rc == 801 and tokens > 100)
        for got in ([ys] if rc == 0 else []) + [mmq.forward_many(ws, x)]:
            for y, w in zip(got, ws):
                want = mmq.forward(w, x)
                assert y.shape == want.shape and bool(torch.isfinite(want.float()).all())
                if min(rows) < 1024 and w.shape[0] < 1024:
                    assert torch.equal(y, want), (tokens, w.shape)
                assert float((y.double() - want.double()).norm()) <= 2.0 ** -10 * float(want.double().norm()), (tokens, w.shape)


def test_what_one_launch_declines(cuda):
    """Other block types, results or weights off a 16-byte boundary, rows that are no multiple of 16 bytes, forced weight formats and matrices that fill the GPU
    by themselves are launched one by one; a list of mixed types goes by its neighbours of one type."""
    g = torch.Generator(device=cuda).manual_seed(1)
    x = torch.randn(24, 2048, device=cuda, generator=g).to(torch.bfloat16)
    assert _entry([_matrix("q4_0", 512, 2048, cuda, g) for _ in range(2)], x)[0] == 801
    pair = [_matrix("q8_0", 512, 2048, cuda, g) for _ in range(2)]
    assert _entry(pair, x)[0] == 0
    off = torch.empty(pair[1].data.numel() + 8, dtype=torch.uint8, device=cuda)[8:]
    off.copy_(pair[1].data)
    assert _entry([pair[0], quant.QTensor(off, "q8_0", pair[1].shape)], x)[0] == 801
    six = [_matrix("q6_k", 512, 2304, cuda, g) for _ in range(2)]
    assert _entry(six, torch.randn(24, 2304, device=cuda, generator=g).to(torch.bfloat16))[0] == 801
    mmq.set_weight_format("f16")
    try:
        assert _entry(pair, x)[0] == 801
    finally:
        mmq.set_weight_format("same")
    many = [_matrix("q4_k", 18944, 2048, cuda, g) for _ in range(2)]        # 148 row tiles each
    assert _entry(many, torch.randn(1000, 2048, device=cuda, generator=g).to(torch.bfloat16))[0] == 801
    mixed = [pair[0], pair[1], _matrix("q4_0", 96, 2048, cuda, g), pair[0]]
    for y, w in zip(mmq.forward_many(mixed, x.view(2, 12, 2048)), mixed):
        assert torch.equal(y, mmq.forward(w, x.view(2, 12, 2048))) and y.shape == (2, 12, w.shape[0])
    assert [tuple(y.shape) for y in mmq.forward_many(pair, x[:0])] == [(0, 512), (0, 512)]
    with pytest.raises(ValueError):
        mmq.forward_many([pair[0], six[0]], x)


@pytest.mark.parametrize("kind,tokens,asked", [("q4_0", 24, 0), ("q8_0", 400, 1), ("q4_k", 24, 1)])
def test_what_a_list_costs_the_host(cuda, monkeypatch, kind, tokens, asked):
    """Each matrix is looked at once and each result allocated once, whether the list becomes one launch or is declined; types that never group are not asked for."""
    g = torch.Generator(device=cuda).manual_seed(1)
    ws = [_matrix(kind, 8192, 2048, cuda, g) for _ in range(2)]
    x = torch.randn(tokens, 2048, device=cuda, generator=g).to(torch.bfloat16)
    want = [mmq.forward(w, x) for w in ws]
    seen, check, typed = [], mmq._check, mmq.typed
    monkeypatch.setattr(mmq, "_check", lambda w, xs: seen.append("check") or check(w, xs))
    monkeypatch.setattr(mmq, "typed", lambda name, *a: seen.append(name) or typed(name, *a))
    before = torch.cuda.memory_stats(cuda)["allocation.all.allocated"]
    ys = mmq.forward_many(ws, x)
    assert torch.cuda.memory_stats(cuda)["allocation.all.allocated"] - before == 2
    assert seen.count("check") == 2 and seen.count("mrs_mmq_gguf_multi") == asked
    assert all(float((y.double() - w.double()).norm()) <= 2.0 ** -10 * float(w.double().norm()) for y, w in zip(ys, want))


@pytest.mark.parametrize("kind,rows,cols,tokens,one", [("q5_k", 11008, 4096, 256, False), ("q8_0", 13824, 5120, 256, False), ("q5_k", 11008, 4096, 200, True),
                                                       ("q4_k", 11008, 4096, 256, True), ("q5_k", 16384, 4096, 256, True)])
def test_more_waves_than_alone(cuda, kind, rows, cols, tokens, one):
    """Lists whose one launch has more waves than the matrices have alone are grouped only where that promises much."""
    g = torch.Generator(device=cuda).manual_seed(rows)
    ws = [_matrix(kind, rows, cols, cuda, g) for _ in range(2)]
    x = torch.randn(tokens, cols, device=cuda, generator=g).to(torch.bfloat16)
    rc, _ = _entry(ws, x)
    assert rc == (0 if one else 801)
    for y, w in zip(mmq.forward_many(ws, x), ws):
        want = mmq.forward(w, x)
        assert float((y.double() - want.double()).norm()) <= 2.0 ** -10 * float(want.double().norm())
