"""Prefill (batch > 8) quantized GEMM — mirror of `fast_mmq::plain`
(REF mistralrs-quant/src/gguf/fast_mmq.rs:762-826) on the tcgen05 dequant-GEMM kernel
(`mrs_mmq_gguf`, csrc/mmq_ts.cu).  Unlike the reference there is no activation quantisation
pass: activations stay bf16/f16 and weights are dequantised on the fly into tensor memory."""
import ctypes

import torch

from . import GGML, lib
from .quant import _I, _P, raw_stream, typed

_DT_CODE = {torch.float16: 0, torch.bfloat16: 1}


def _check(w, xs):
    if xs.dtype not in _DT_CODE:
        raise ValueError(f"fast_mmq: input dtype must be BF16 or F16, got {xs.dtype}")
    nrows, ncols = w.shape
    if xs.shape[-1] != ncols:
        raise ValueError(f"fast_mmq: shape mismatch: weight [{nrows}, {ncols}] vs input tail {xs.shape[-1]}")
    if xs.device != w.device:
        raise ValueError("fast_mmq: input and weight are on different devices")
    if ncols % 64:
        raise ValueError("fast_mmq: K must be a multiple of 64")
    return nrows, ncols


def forward(w, xs: torch.Tensor) -> torch.Tensor:
    """w: quant.QTensor [N, K]; xs [..., K] bf16/f16 -> [..., N]."""
    nrows, ncols = _check(w, xs)
    xs = xs.contiguous()
    out = xs.new_empty((*xs.shape[:-1], nrows))
    entry = typed("mrs_mmq_gguf", _I, _P, _P, _P, _I, _I, _I, _I, _P)
    rc = entry(GGML[w.dtype], w.data.data_ptr(), xs.data_ptr(), out.data_ptr(), xs.numel() // ncols, nrows, ncols, _DT_CODE[xs.dtype], raw_stream(xs.device))
    if rc != 0:
        raise RuntimeError(f"mrs_mmq_gguf failed with cudaError {rc}")
    return out


def forward_chained(w, xs: torch.Tensor) -> torch.Tensor:
    """`forward` for weights that nothing in flight writes: begins on them while the launch before it runs."""
    nrows, ncols = _check(w, xs)
    xs = xs.contiguous()
    return _launch("mrs_mmq_gguf_chained", w, xs, xs.numel() // ncols, xs.new_empty((*xs.shape[:-1], nrows)))


def _launch(name, w, xs, M, out):
    nrows, ncols = w.shape
    entry = typed(name, _I, _P, _P, _P, _I, _I, _I, _I, _P)
    rc = entry(GGML[w.dtype], w.data.data_ptr(), xs.data_ptr(), out.data_ptr(), M, nrows, ncols, _DT_CODE[xs.dtype], raw_stream(xs.device))
    if rc != 0:
        raise RuntimeError(f"{name} failed with cudaError {rc}")
    return out


_NOT_SUPPORTED = 801        # cudaErrorNotSupported: nothing was launched, alone is faster or what is possible
_GROUPED = ("q4_k", "q5_k", "q6_k", "q8_0")


def forward_many(ws, xs: torch.Tensor, chained=False):
    """[forward(w, xs) for w in ws], neighbours of one type as one launch (up to three) where that is faster.  chained: as `forward_chained`."""
    if not xs.is_cuda:                     # (refused there)
        return [(forward_chained if chained else forward)(w, xs) for w in ws]
    rows = [_check(w, xs)[0] for w in ws]
    xs = xs.contiguous()
    ncols = xs.shape[-1]
    M = xs.numel() // ncols
    ys = [xs.new_empty((*xs.shape[:-1], n)) for n in rows]
    one, many = ("mrs_mmq_gguf_chained", "mrs_mmq_gguf_multi_chained") if chained else ("mrs_mmq_gguf", "mrs_mmq_gguf_multi")
    i = 0
    while i < len(ws):
        kind, n = ws[i].dtype, 1
        while n < 3 and i + n < len(ws) and ws[i + n].dtype == kind and kind in _GROUPED and M > 0:
            n += 1
        j = i + n
        if n > 1:
            data, to, sizes = [w.data.data_ptr() for w in ws[i:j]], [y.data_ptr() for y in ys[i:j]], rows[i:j]
            if n == 2:
                data.append(None), sizes.append(0), to.append(None)
            entry = typed(many, _I, *[_P] * 7, *[_I] * 6, _P)
            rc = entry(GGML[kind], *data, xs.data_ptr(), *to, M, *sizes, ncols, _DT_CODE[xs.dtype], raw_stream(xs.device))
            if rc == 0:
                i = j
                continue
            if rc != _NOT_SUPPORTED:
                raise RuntimeError(f"{many} failed with cudaError {rc}")
        for k in range(i, j):
            _launch(one, ws[k], xs, M, ys[k])
        i = j
    return ys


def timeout_word(device):
    """The word that a kernel sets when a wait of its runs out on `device`: an int32 in host memory, as a ctypes pointer."""
    with torch.cuda.device(device):
        fn = lib().mrs_mmq_timeout_flag
        fn.restype = ctypes.POINTER(ctypes.c_int32)
        return fn()


def check_timeouts(device):
    """Raises when a wait inside a kernel that shares this word ever ran out on `device`: the dequantising GEMM (ggml and int4 linears), the tensor-core
    GEMV (three to eight rows over large matrices), prompt attention and the resident grid of one-sequence decode steps.  Results since then are
    incomplete.  Reads a word in host memory, so call it once the work in question is done.  Calls that would run on one of these kernels are refused by
    themselves from then on (decode steps of one sequence run as a chain of launches instead); replays of a graph pass no entry point and need this."""
    flag = timeout_word(device)
    if flag and flag[0]:
        raise RuntimeError("a wait inside a linear, prompt attention or a resident decode step ran out: the results of this device are incomplete")


def set_path(path: str):
    """'auto' (default): csrc/mmq_ts.cu when the launch fits it, else csrc/mmq_tc.cu; 'tc': mmq_tc.cu only (A/B, tests)."""
    lib().mrs_mmq_set_path(ctypes.c_int({"auto": 0, "tc": 1}[path]))


def set_weight_format(fmt: str):
    """'same' (default: the activations' 16-bit format), 'f16' or 'bf16' for the dequantised weights."""
    lib().mrs_mmq_set_weight_format(ctypes.c_int({"same": -1, "f16": 0, "bf16": 1}[fmt]))


# ---- the reference's entry points over this kernel (REF mistralrs-quant/src/gguf/fast_mmq.rs:760-826).  In the reference the
# point of the fused forms is ONE activation-quantisation pass shared by the projections; this design never quantises
# activations, so they are the same projections over the same bf16/f16 input — kept under the reference's names so a
# caller written against fast_mmq finds them. ----
def plain(w, xs: torch.Tensor) -> torch.Tensor:
    return forward(w, xs)


def fused_qkv(q_w, k_w, v_w, xs: torch.Tensor):
    return tuple(forward_many([q_w, k_w, v_w], xs))


def fused_glu(gate_w, up_w, xs: torch.Tensor, activation) -> torch.Tensor:
    if tuple(gate_w.shape) != tuple(up_w.shape):
        raise ValueError(f"fast_mmq fused_glu: gate/up shape mismatch {tuple(gate_w.shape)} vs {tuple(up_w.shape)}")
    from . import ops
    return ops.fused_glu(*forward_many([gate_w, up_w], xs), activation)


def fused_ffn(gate_w, up_w, down_w, xs: torch.Tensor, activation) -> torch.Tensor:
    if tuple(gate_w.shape) != tuple(up_w.shape):
        raise ValueError(f"fast_mmq fused_ffn: gate/up shape mismatch {tuple(gate_w.shape)} vs {tuple(up_w.shape)}")
    if not xs.is_cuda:                     # (refused there)
        return forward(down_w, fused_glu(gate_w, up_w, xs, activation))
    # the first launch is a plain one: nothing that was in flight before it runs beside the links
    from . import ops
    return forward_chained(down_w, ops._glu_link(*forward_many([gate_w, up_w], xs), activation))
