"""ctypes front-end of libmrs_b200_seq.so (include/mrs_b200_seq.h): residual streams, gated linear recurrences,
short causal convolutions, windowed attention over a paged cache, expert routing.  PyTorch supplies memory and the
stream; there is no CPU fallback — a missing library is built on first use (nvcc, sm_100a) or the import fails."""
import ctypes
import os
import subprocess

import torch

from . import ExtensionMissing

_HERE = os.path.dirname(os.path.abspath(__file__))
SEQ_LIB_PATH = os.path.join(_HERE, "libmrs_b200_seq.so")
BF16, F32 = 1, 2
ACT_NONE, ACT_SILU, ACT_GELU_TANH, ACT_SIGMOID, ACT_GELU_ERF, ACT_RELU_SQ = 0, 1, 2, 3, 4, 5
GLU_CAPPED = 100
SCORE_SOFTMAX, SCORE_SIGMOID = 0, 1
QK_NORM_NONE, QK_NORM_HEAD, QK_NORM_WHOLE = 0, 1, 2
PAIRS_HALVES, PAIRS_NEIGHBOURS = 0, 1
DTYPE_CODE = {torch.bfloat16: BF16, torch.float32: F32}
_lib = None


def make_target(directory, product):
    """Build `product` with the Makefile in `directory` when it is missing (a fresh checkout)."""
    if os.path.exists(product):
        return
    try:
        subprocess.check_call(["make", "-s", "-j", str(min(8, os.cpu_count() or 1)), "-C", directory], stdout=subprocess.DEVNULL)
    except (OSError, subprocess.CalledProcessError) as e:
        raise ExtensionMissing(f"{product} is missing and `make -C {directory}` failed: {e}") from e
    if not os.path.exists(product):
        raise ExtensionMissing(f"{product} was not produced by `make -C {directory}`")


def ensure_host_lib():
    from . import kv_index
    make_target(os.path.join(_HERE, "host"), kv_index.HOST_LIB_PATH)
    L = kv_index.host_lib()
    if getattr(L, "_seq_types", None) is None:
        L.mrs_state_slots_new.restype = ctypes.c_void_p
        for f in ("capacity", "num_free", "acquire", "slot_of"):
            getattr(L, f"mrs_state_slots_{f}").restype = ctypes.c_int64
        L._seq_types = True
    return L


class ScanArgs(ctypes.Structure):
    _fields_ = [("q", ctypes.c_void_p), ("k", ctypes.c_void_p), ("v", ctypes.c_void_p),
                ("q_ld", ctypes.c_int64), ("k_ld", ctypes.c_int64), ("v_ld", ctypes.c_int64),
                ("dtype", ctypes.c_int), ("act", ctypes.c_int),
                ("heads", ctypes.c_int), ("qk_groups", ctypes.c_int), ("dk", ctypes.c_int), ("dv", ctypes.c_int),
                ("decay_tok", ctypes.c_void_p), ("decay_head", ctypes.c_void_p), ("scale_tok", ctypes.c_void_p),
                ("skip", ctypes.c_void_p), ("state", ctypes.c_void_p),
                ("cu_tok", ctypes.c_void_p), ("past", ctypes.c_void_p), ("slot", ctypes.c_void_p),
                ("n_seq", ctypes.c_int), ("n_tok", ctypes.c_int), ("out", ctypes.c_void_p),
                ("seg_state", ctypes.c_void_p), ("seg_decay", ctypes.c_void_p), ("seg_len", ctypes.c_int), ("n_segs", ctypes.c_int),
                ("decay_vec", ctypes.c_void_p), ("q_scale", ctypes.c_float)]


class GluRule(ctypes.Structure):
    """How a gated feed-forward joins its halves: act(gate) * up, or — act GLU_CAPPED — with g = min(gate, limit) and
    u = clamp(up, -limit, limit): g * sigmoid(slope * g) * (u + shift)."""
    _fields_ = [("act", ctypes.c_int), ("limit", ctypes.c_float), ("slope", ctypes.c_float), ("shift", ctypes.c_float)]

    @classmethod
    def of(cls, act):
        return act if isinstance(act, cls) else cls(int(act), 0.0, 0.0, 0.0)

    @classmethod
    def capped(cls, limit, slope, shift):
        return cls(GLU_CAPPED, float(limit), float(slope), float(shift))


class RmsResidualArgs(ctypes.Structure):
    _fields_ = [("src", ctypes.c_void_p), ("dst", ctypes.c_void_p), ("y", ctypes.c_void_p), ("mult", ctypes.c_float),
                ("hist", ctypes.c_void_p), ("hist_stride", ctypes.c_int64), ("n_hist", ctypes.c_int), ("mix", ctypes.c_void_p),
                ("mixed", ctypes.c_void_p), ("next_w", ctypes.c_void_p), ("eps", ctypes.c_float), ("next_out", ctypes.c_void_p),
                ("dtype", ctypes.c_int), ("n_tok", ctypes.c_int), ("width", ctypes.c_int), ("post_w", ctypes.c_void_p), ("add_vec", ctypes.c_void_p),
                ("next_b", ctypes.c_void_p), ("center", ctypes.c_int), ("rows", ctypes.c_void_p), ("post_center", ctypes.c_int)]


class LatentPrepareArgs(ctypes.Structure):
    _fields_ = [("y", ctypes.c_void_p), ("y_ld", ctypes.c_int64), ("dtype", ctypes.c_int), ("q_col", ctypes.c_int), ("q_rank", ctypes.c_int),
                ("q_norm_w", ctypes.c_void_p), ("q_out", ctypes.c_void_p), ("q_out_ld", ctypes.c_int64),
                ("kv_col", ctypes.c_int), ("kv_rank", ctypes.c_int), ("rot_dim", ctypes.c_int), ("rot_dims", ctypes.c_int),
                ("kv_norm_w", ctypes.c_void_p), ("cos_sin", ctypes.c_void_p), ("eps", ctypes.c_float), ("cache", ctypes.c_void_p),
                ("cache_row", ctypes.c_int64), ("slot_of_tok", ctypes.c_void_p), ("n_tok", ctypes.c_int), ("kv_out", ctypes.c_void_p),
                ("kv_out_ld", ctypes.c_int64), ("pairing", ctypes.c_int), ("rq_heads", ctypes.c_int), ("rq_col", ctypes.c_int),
                ("rq_head", ctypes.c_int64), ("rq_out", ctypes.c_void_p), ("rq_out_ld", ctypes.c_int64), ("rq_out_head", ctypes.c_int64)]


class AttnPrepareArgs(ctypes.Structure):
    _fields_ = [("q", ctypes.c_void_p), ("k", ctypes.c_void_p), ("v", ctypes.c_void_p),
                ("q_ld", ctypes.c_int64), ("k_ld", ctypes.c_int64), ("v_ld", ctypes.c_int64),
                ("dtype", ctypes.c_int), ("norm_mode", ctypes.c_int),
                ("q_norm_w", ctypes.c_void_p), ("k_norm_w", ctypes.c_void_p), ("eps", ctypes.c_float),
                ("heads", ctypes.c_int), ("kv_heads", ctypes.c_int), ("dk", ctypes.c_int), ("dv", ctypes.c_int),
                ("rot_dims", ctypes.c_int), ("cos_sin", ctypes.c_void_p),
                ("k_cache", ctypes.c_void_p), ("v_cache", ctypes.c_void_p), ("slot_of_tok", ctypes.c_void_p), ("n_tok", ctypes.c_int),
                ("pairing", ctypes.c_int), ("norm_last", ctypes.c_int)]


class PagedAttentionArgs(ctypes.Structure):
    _fields_ = [("q", ctypes.c_void_p), ("q_ld", ctypes.c_int64), ("k_cache", ctypes.c_void_p), ("v_cache", ctypes.c_void_p),
                ("dtype", ctypes.c_int), ("heads", ctypes.c_int), ("kv_heads", ctypes.c_int), ("dk", ctypes.c_int), ("dv", ctypes.c_int),
                ("scale", ctypes.c_float), ("window", ctypes.c_int), ("keep_first", ctypes.c_int), ("sink", ctypes.c_void_p),
                ("pages", ctypes.c_void_p), ("pages_ld", ctypes.c_int), ("page_size", ctypes.c_int),
                ("seq_of_tok", ctypes.c_void_p), ("pos_of_tok", ctypes.c_void_p), ("tok_index", ctypes.c_void_p), ("n_tok", ctypes.c_int),
                ("out", ctypes.c_void_p), ("out_ld", ctypes.c_int64), ("out_scale", ctypes.c_float),
                ("k_row", ctypes.c_int64), ("v_row", ctypes.c_int64), ("pool", ctypes.c_int), ("pool_base", ctypes.c_int64),
                ("v_shared", ctypes.c_int), ("out_f32", ctypes.c_int), ("out_head", ctypes.c_int64),
                ("gate", ctypes.c_void_p), ("gate_ld", ctypes.c_int64), ("gate_group", ctypes.c_int), ("gate_act", ctypes.c_int),
                ("chunk", ctypes.c_int)]


class PromptAttentionArgs(ctypes.Structure):
    _fields_ = [("q", ctypes.c_void_p), ("q_ld", ctypes.c_int64), ("k_cache", ctypes.c_void_p), ("v_cache", ctypes.c_void_p),
                ("out", ctypes.c_void_p), ("out_ld", ctypes.c_int64), ("portions", ctypes.c_void_p), ("n_portions", ctypes.c_int),
                ("longest", ctypes.c_int), ("pages", ctypes.c_void_p), ("pages_ld", ctypes.c_int), ("page_size", ctypes.c_int),
                ("heads", ctypes.c_int), ("kv_heads", ctypes.c_int), ("d", ctypes.c_int), ("scale", ctypes.c_float), ("window", ctypes.c_int),
                ("keep_first", ctypes.c_int), ("sink", ctypes.c_void_p), ("pool", ctypes.c_int), ("pool_base", ctypes.c_int64),
                ("every_value_head", ctypes.c_int), ("chunk", ctypes.c_int), ("gate", ctypes.c_void_p), ("gate_ld", ctypes.c_int64),
                ("gate_group", ctypes.c_int), ("gate_act", ctypes.c_int)]


class PromptAttentionTcArgs(ctypes.Structure):
    _fields_ = [("q", ctypes.c_void_p), ("k", ctypes.c_void_p), ("k_shared", ctypes.c_void_p), ("v", ctypes.c_void_p),
                ("q_ld", ctypes.c_int64), ("k_ld", ctypes.c_int64), ("k_shared_ld", ctypes.c_int64), ("v_ld", ctypes.c_int64),
                ("q_rows", ctypes.c_int64), ("k_rows", ctypes.c_int64), ("out", ctypes.c_void_p), ("out_ld", ctypes.c_int64),
                ("segments", ctypes.c_void_p), ("n_segments", ctypes.c_int), ("longest", ctypes.c_int), ("heads", ctypes.c_int),
                ("kv_heads", ctypes.c_int), ("dn", ctypes.c_int), ("dr", ctypes.c_int), ("dv", ctypes.c_int), ("scale", ctypes.c_float),
                ("gate", ctypes.c_void_p), ("gate_ld", ctypes.c_int64), ("gate_group", ctypes.c_int), ("gate_act", ctypes.c_int),
                ("window", ctypes.c_int), ("keep_first", ctypes.c_int), ("held", ctypes.c_void_p), ("sink", ctypes.c_void_p)]


class MoeRouteArgs(ctypes.Structure):
    _fields_ = [("logits", ctypes.c_void_p), ("correction", ctypes.c_void_p), ("n_tok", ctypes.c_int), ("n_experts", ctypes.c_int),
                ("n_groups", ctypes.c_int), ("keep_groups", ctypes.c_int), ("top", ctypes.c_int), ("renorm", ctypes.c_int),
                ("score_fn", ctypes.c_int), ("group_top", ctypes.c_int), ("weight_scale", ctypes.c_float), ("renorm_eps", ctypes.c_float),
                ("experts", ctypes.c_void_p), ("weights", ctypes.c_void_p), ("logits_ld", ctypes.c_int64)]


class MoeSmallArgs(ctypes.Structure):
    _fields_ = [("x", ctypes.c_void_p), ("gate_up", ctypes.c_void_p), ("down", ctypes.c_void_p), ("dtype", ctypes.c_int),
                ("experts", ctypes.c_void_p), ("weights", ctypes.c_void_p), ("n_tok", ctypes.c_int), ("top", ctypes.c_int),
                ("width", ctypes.c_int), ("ff", ctypes.c_int), ("n_ffn", ctypes.c_int), ("rule", GluRule), ("hidden", ctypes.c_void_p),
                ("out", ctypes.c_void_p)]


class MoeGroupedArgs(ctypes.Structure):
    _fields_ = [("x", ctypes.c_void_p), ("up", ctypes.c_void_p), ("down", ctypes.c_void_p), ("dtype", ctypes.c_int), ("counts", ctypes.c_void_p),
                ("order", ctypes.c_void_p), ("n_tok", ctypes.c_int), ("top", ctypes.c_int), ("width", ctypes.c_int), ("ff", ctypes.c_int),
                ("n_ffn", ctypes.c_int), ("gated", ctypes.c_int), ("rule", GluRule), ("hidden", ctypes.c_void_p), ("y", ctypes.c_void_p)]


class MoeBlockArgs(ctypes.Structure):
    _fields_ = ([(n, ctypes.c_void_p) for n in ("x", "router", "logits")] + [("logits_ld", ctypes.c_int64)]
                + [(n, ctypes.c_void_p) for n in ("correction", "up", "down", "scratch")] + [("scratch_bytes", ctypes.c_int64), ("out", ctypes.c_void_p)]
                + [(n, ctypes.c_int) for n in ("dtype", "n_tok", "width", "ff", "n_routes", "n_ffn", "top", "gated", "route", "products", "n_groups",
                                               "keep_groups", "renorm", "group_top")]
                + [("weight_scale", ctypes.c_float), ("renorm_eps", ctypes.c_float), ("rule", GluRule)])


class LatentAttentionArgs(ctypes.Structure):
    _fields_ = [("q", ctypes.c_void_p), ("q_ld", ctypes.c_int64), ("cache", ctypes.c_void_p), ("cache_row", ctypes.c_int64),
                ("out", ctypes.c_void_p), ("out_ld", ctypes.c_int64), ("portions", ctypes.c_void_p), ("cu_tok", ctypes.c_void_p),
                ("past", ctypes.c_void_p), ("n_portions", ctypes.c_int), ("longest", ctypes.c_int), ("pages", ctypes.c_void_p),
                ("pages_ld", ctypes.c_int), ("page_size", ctypes.c_int), ("heads", ctypes.c_int), ("kv_rank", ctypes.c_int),
                ("rot_dim", ctypes.c_int), ("scale", ctypes.c_float), ("window", ctypes.c_int), ("splits", ctypes.c_int),
                ("scratch", ctypes.c_void_p)]


SCAN_SEGMENT = 256                  # tokens per segment when a long portion is scanned as segments side by side
SCAN_SEGMENT_MIN_TOKENS = 1024      # portions shorter than this run in one pass
SCAN_SCRATCH_BYTES = 1 << 30


def lib():
    global _lib
    if _lib is None:
        make_target(os.path.join(_HERE, "csrc", "seq"), SEQ_LIB_PATH)
        _lib = ctypes.CDLL(SEQ_LIB_PATH)
    return _lib


def _p(t, offset=0):
    """Device address of element `offset` of a tensor (None -> NULL)."""
    if t is None:
        return ctypes.c_void_p(0)
    return ctypes.c_void_p(t.data_ptr() + offset * t.element_size())


def _st(t):
    return ctypes.c_int64(torch.cuda.current_stream(t.device).cuda_stream)


def _ok(rc, what):
    if rc != 0:
        raise RuntimeError(f"{what} failed: {'bad argument' if rc < 0 else 'cudaError'} {rc}")


_i, _f, _l = ctypes.c_int, ctypes.c_float, ctypes.c_int64


def embed_streams(table, ids, n_streams):
    T, W = ids.numel(), table.shape[1]
    out = torch.empty(T, n_streams, W, dtype=torch.float32, device=table.device)
    _ok(lib().mrs_seq_embed_streams(_p(table), _i(DTYPE_CODE[table.dtype]), _p(ids), _p(out), _i(T), _i(n_streams), _i(W), _st(table)),
        "embed_streams")
    return out


def streams_read_norm(streams, w_in, norm_w, eps, unit_offset, dtype, rows=None):
    T, S, W = streams.shape
    n = T if rows is None else rows.numel()
    out = torch.empty(n, W, dtype=dtype, device=streams.device)
    _ok(lib().mrs_seq_streams_read_norm(_p(streams), _p(w_in), _p(norm_w), _f(eps), _f(unit_offset), _p(rows), _p(out),
                                        _i(DTYPE_CODE[dtype]), _i(n), _i(S), _i(W), _st(streams)), "streams_read_norm")
    return out


def streams_write(streams, w_mix, w_out, y, next_in=None, next_norm_w=None, eps=0.0, unit_offset=0.0):
    """In place on `streams`; returns the next sublayer's normed input when next_norm_w is given."""
    T, S, W = streams.shape
    nxt = torch.empty(T, W, dtype=y.dtype, device=y.device) if next_norm_w is not None else None
    _ok(lib().mrs_seq_streams_write(_p(streams), _p(w_mix), _p(w_out), _p(y), _i(DTYPE_CODE[y.dtype]), _i(T), _i(S), _i(W),
                                    _p(next_in), _p(next_norm_w), _f(eps), _f(unit_offset), _p(nxt), _st(streams)), "streams_write")
    return nxt


def activate_cols(x, col0, cols, act):
    """x[:, col0:col0 + cols] = act(.) in place."""
    _ok(lib().mrs_seq_activate_cols(_p(x, col0), _l(x.stride(0)), _i(DTYPE_CODE[x.dtype]), _i(x.shape[0]), _i(cols), _i(act), _st(x)),
        "activate_cols")


def glu_split(x, act):
    """act: an activation code (act(gate) * up) or a `GluRule`."""
    T, two = x.shape
    out = torch.empty(T, two // 2, dtype=x.dtype, device=x.device)
    rule = GluRule.of(act)
    _ok(lib().mrs_seq_glu_join(_p(x), _p(out), _i(DTYPE_CODE[x.dtype]), _i(T), _i(two // 2), ctypes.byref(rule), _st(x)), "glu_join")
    return out


def bounded_gate(y, col0, cols, bias, lower):
    """f32 [T, cols]: lower + (1 - lower) * sigmoid(y[:, col0:col0 + cols] + bias)."""
    T = y.shape[0]
    out = torch.empty(T, cols, dtype=torch.float32, device=y.device)
    _ok(lib().mrs_seq_bounded_gate(_p(y, col0), _l(y.stride(0)), _i(DTYPE_CODE[y.dtype]), _p(bias), _p(lower), _i(T), _i(cols), _p(out), _st(y)),
        "bounded_gate")
    return out


def power_gate(y, col0, cols, bias, power):
    """f32 [T, cols]: sigmoid(y[:, col0:col0 + cols] + bias) ** power, formed as exp(power * log_sigmoid(.))."""
    T = y.shape[0]
    out = torch.empty(T, cols, dtype=torch.float32, device=y.device)
    _ok(lib().mrs_seq_power_gate(_p(y, col0), _l(y.stride(0)), _i(DTYPE_CODE[y.dtype]), _p(bias), _f(power), _i(T), _i(cols), _p(out), _st(y)),
        "power_gate")
    return out


def gated_group_norm(x, gate, gate_col, weight, groups, eps, gate_act, gate_first, out, out_col=0, out_scale=1.0):
    """x f32 [T, C]; the gate is columns gate_col.. of `gate`; writes columns out_col.. of `out`."""
    T, C = x.shape
    if gate is None:        # no gate: the plain group norm
        _ok(lib().mrs_seq_gated_group_norm(_p(x), _p(None), _l(0), _p(weight), _p(out, out_col), _l(out.stride(0)), _f(out_scale),
                                           _i(DTYPE_CODE[out.dtype]), _i(T), _i(C), _i(groups), _f(eps), _i(ACT_NONE), _i(0), _st(x)),
            "gated_group_norm")
        return
    _ok(lib().mrs_seq_gated_group_norm(_p(x), _p(gate, gate_col), _l(gate.stride(0)), _p(weight), _p(out, out_col), _l(out.stride(0)),
                                       _f(out_scale), _i(DTYPE_CODE[out.dtype]), _i(T), _i(C), _i(groups), _f(eps), _i(gate_act),
                                       _i(int(gate_first)), _st(x)), "gated_group_norm")


def causal_conv(inp, col0, channels, taps, bias, act, conv_state, batch):
    T = inp.shape[0]
    out = torch.empty(T, channels, dtype=inp.dtype, device=inp.device)
    _ok(lib().mrs_seq_causal_conv(_p(inp), _l(inp.stride(0)), _i(col0), _i(DTYPE_CODE[inp.dtype]), _p(taps), _p(bias), _i(channels),
                                  _i(taps.shape[1]), _i(act), _p(conv_state), _p(batch.cu_tok), _p(batch.past), _p(batch.slot),
                                  _p(batch.seq_of_tok), _i(batch.n_seq), _i(T), _p(out), _st(inp)), "causal_conv")
    return out


def ssm_steps(inp, col0, bias, a_log):
    T, H = inp.shape[0], bias.numel()
    step = torch.empty(T, H, dtype=torch.float32, device=inp.device)
    decay = torch.empty_like(step)
    _ok(lib().mrs_seq_ssm_steps(_p(inp), _l(inp.stride(0)), _i(col0), _i(DTYPE_CODE[inp.dtype]), _p(bias), _p(a_log), _i(H), _i(T),
                                _p(step), _p(decay), _st(inp)), "ssm_steps")
    return step, decay


def linear_scan(q, q_col, k, k_col, v, v_col, heads, qk_groups, dk, dv, state, batch, act=ACT_NONE, decay_tok=None, decay_head=None,
                scale_tok=None, skip=None, decay_vec=None, q_scale=1.0):
    """q / k / v are column ranges (starting at *_col) of 2-D activation tensors; returns o f32 [T, heads * dv].
    decay_vec f32 [T, heads * dk]: every state row has its own decay; with k None the key is the decay's complement.
    q_scale: a constant factor on the queries (applied in f32)."""
    T = q.shape[0]
    out = torch.empty(T, heads * dv, dtype=torch.float32, device=q.device)
    a = ScanArgs()
    a.q, a.v = _p(q, q_col).value, _p(v, v_col).value
    a.q_ld, a.v_ld = q.stride(0), v.stride(0)
    if k is not None:
        a.k, a.k_ld = _p(k, k_col).value, k.stride(0)
    a.decay_vec, a.q_scale = _p(decay_vec).value, float(q_scale)
    a.dtype, a.act = DTYPE_CODE[q.dtype], act
    a.heads, a.qk_groups, a.dk, a.dv = heads, qk_groups, dk, dv
    a.decay_tok, a.decay_head = _p(decay_tok).value, _p(decay_head).value
    a.scale_tok, a.skip = _p(scale_tok).value, _p(skip).value
    a.state = state.data_ptr()
    a.cu_tok, a.past, a.slot = batch.cu_tok.data_ptr(), batch.past.data_ptr(), batch.slot.data_ptr()
    a.n_seq, a.n_tok, a.out = batch.n_seq, T, out.data_ptr()
    longest = getattr(batch, "longest", 0)
    if longest >= SCAN_SEGMENT_MIN_TOKENS:
        seg = SCAN_SEGMENT
        while batch.n_seq * -(-longest // seg) * heads * dk * dv * 4 > SCAN_SCRATCH_BYTES:
            seg *= 2
        n_segs = -(-longest // seg)
        if n_segs > 1:
            seg_state = torch.empty(batch.n_seq * n_segs * heads * dk * dv, dtype=torch.float32, device=q.device)
            seg_decay = torch.empty(batch.n_seq * n_segs * heads * (dk if decay_vec is not None else 1), dtype=torch.float32, device=q.device)
            a.seg_state, a.seg_decay, a.seg_len, a.n_segs = seg_state.data_ptr(), seg_decay.data_ptr(), seg, n_segs
    _ok(lib().mrs_seq_linear_scan(ctypes.byref(a), _st(q)), "linear_scan")
    return out


def qk_norm_store(y, q_col, k_col, v_col, q_norm_w, k_norm_w, eps, heads, kv_heads, dk, dv, k_cache, v_cache, slot_of_tok):
    T, ld = y.shape[0], y.stride(0)
    _ok(lib().mrs_seq_qk_norm_store(_p(y, q_col), _l(ld), _p(y, k_col), _l(ld), _p(y, v_col), _l(ld), _i(DTYPE_CODE[y.dtype]),
                                    _p(q_norm_w), _p(k_norm_w), _f(eps), _i(heads), _i(kv_heads), _i(dk), _i(dv), _p(k_cache),
                                    _p(v_cache), _p(slot_of_tok), _i(T), _st(y)), "qk_norm_store")


def window_attention(y, q_col, k_cache, v_cache, heads, kv_heads, dk, dv, scale, window, batch, page_size, out, out_col=0, out_scale=1.0,
                     tok_index=None):
    """Every token of the step (or those listed in tok_index) against the pages of its sequence."""
    n = y.shape[0] if tok_index is None else tok_index.numel()
    _ok(lib().mrs_seq_window_attention(_p(y, q_col), _l(y.stride(0)), _p(k_cache), _p(v_cache), _i(DTYPE_CODE[y.dtype]), _i(heads),
                                       _i(kv_heads), _i(dk), _i(dv), _f(scale), _i(int(window)), _p(batch.pages), _i(batch.pages.shape[1]),
                                       _i(page_size), _p(batch.seq_of_tok), _p(batch.pos_of_tok), _p(tok_index), _i(n), _p(out, out_col),
                                       _l(out.stride(0)), _f(out_scale), _st(y)), "window_attention")


def scale_rows(x, row0, rows, col0, cols, scale):
    _ok(lib().mrs_seq_scale_rows(_p(x, row0 * x.stride(0) + col0), _l(x.stride(0)), _i(DTYPE_CODE[x.dtype]), _i(rows), _i(cols), _f(scale),
                                 _st(x)), "scale_rows")


def fresh_prompt_attention(y, row0, rows, q_col, k_col, v_col, heads, kv_heads, d, scale, window, out, out_col):
    """Causal (windowed) attention of one sequence's first `rows` tokens over its own fresh q / k / v, through the
    package's prompt-attention kernels (tcgen05 for head sizes 64 and 128, windows too; mma.sync for strides that it declines;
    libmrs_b200.so, built on first use).  q / k / v are column ranges of `y`; writes heads * d columns of `out` from out_col."""
    from . import LIB_PATH, lib as main_lib
    make_target(os.path.join(_HERE, "csrc"), LIB_PATH)
    ld, at = y.stride(0), row0 * y.stride(0)
    rc = main_lib().mrs_prefill_attention(_p(y, at + q_col), _p(y, at + k_col), _p(y, at + v_col), _p(out, row0 * out.stride(0) + out_col),
                                          ctypes.c_void_p(0), _i(0), _i(rows), _i(rows), _i(heads), _i(kv_heads), _i(d), _l(ld), _l(ld),
                                          _l(out.stride(0)), _f(scale), _i(1), _i(window - 1 if window > 0 else -1), _f(0.0),
                                          ctypes.c_uint32(1), ctypes.c_void_p(torch.cuda.current_stream(y.device).cuda_stream))
    _ok(rc, "mrs_prefill_attention")


def moe_route(logits, correction, n_groups, keep_groups, top, renorm=False):
    T, E = logits.shape
    experts = torch.empty(T, top, dtype=torch.int32, device=logits.device)
    weights = torch.empty(T, top, dtype=torch.float32, device=logits.device)
    _ok(lib().mrs_seq_moe_route(_p(logits), _p(correction), _i(T), _i(E), _i(n_groups), _i(keep_groups), _i(top), _i(int(renorm)),
                                _p(experts), _p(weights), _st(logits)), "moe_route")
    return experts, weights


def moe_route_scored(logits, correction, n_groups, keep_groups, top, renorm=False, score_fn=SCORE_SOFTMAX, group_top=1, weight_scale=1.0,
                     renorm_eps=0.0):
    """`moe_route` with its choices open: softmax or sigmoid scores, a group scored by the sum of its group_top largest
    choices, renormalising by (sum + renorm_eps), weights times weight_scale."""
    a, experts, weights = _route_args(logits.device, *logits.shape, correction, n_groups, keep_groups, top, renorm, score_fn, group_top, weight_scale,
                                      renorm_eps)
    a.logits, a.logits_ld = _p(logits).value, logits.stride(0)
    _ok(lib().mrs_seq_moe_route_general(ctypes.byref(a), _st(logits)), "moe_route_scored")
    return experts, weights


def _route_args(device, n_tok, n_experts, correction, n_groups, keep_groups, top, renorm, score_fn, group_top, weight_scale, renorm_eps):
    experts = torch.empty(n_tok, top, dtype=torch.int32, device=device)
    weights = torch.empty(n_tok, top, dtype=torch.float32, device=device)
    a = MoeRouteArgs()
    a.correction, a.n_tok, a.n_experts = _p(correction).value, n_tok, n_experts
    a.n_groups, a.keep_groups, a.top, a.renorm, a.score_fn, a.group_top = n_groups, keep_groups, top, int(renorm), score_fn, group_top
    a.weight_scale, a.renorm_eps, a.experts, a.weights = float(weight_scale), float(renorm_eps), _p(experts).value, _p(weights).value
    return a, experts, weights


def moe_router_fits(width, n_experts, n_tok):
    return bool(lib().mrs_seq_moe_router_fits(_i(width), _i(n_experts), _i(n_tok)))


def moe_router(x, w, correction, n_groups, keep_groups, top, renorm=False, score_fn=SCORE_SOFTMAX, group_top=1, weight_scale=1.0, renorm_eps=0.0):
    """`router_logits` and `moe_route_scored` in one launch (`moe_router_fits`): the same experts and weights."""
    T, W = x.shape
    a, experts, weights = _route_args(x.device, T, w.shape[0], correction, n_groups, keep_groups, top, renorm, score_fn, group_top, weight_scale, renorm_eps)
    _ok(lib().mrs_seq_moe_router(_p(x), _i(DTYPE_CODE[x.dtype]), _p(w), _i(W), ctypes.byref(a), _st(x)), "moe_router")
    return experts, weights


ROUTER_SPREAD = 64      # up to this many tokens `router_logits` forms the product one CTA per (output, token)


def router_logits(x, w, w16=None):
    """f32 [T, routes] = x w^T, w f32 [routes, W].  w16: the same weights in bf16 where that is exact — bf16 rows then take a bf16
    library product with f32 sums and an f32 result, which loses nothing (zero rows may pad w16 at its end; the result is then a
    column range of wider rows); otherwise many rows take a true f32 product."""
    T, W = x.shape
    if T > ROUTER_SPREAD:
        if w16 is not None and x.dtype == torch.bfloat16:
            return torch.mm(x, w16.t(), out_dtype=torch.float32)[:, :w.shape[0]]
        return torch.nn.functional.linear(x.float(), w)
    out = torch.empty(T, w.shape[0], dtype=torch.float32, device=x.device)
    _ok(lib().mrs_seq_router_logits(_p(x), _i(DTYPE_CODE[x.dtype]), _p(w), _i(W), _i(w.shape[0]), _i(T), _p(out), _st(x)), "router_logits")
    return out


# `moe_block` calls the entries of the products below in C.  They stand here for callers with experts and weights of their own choosing, and for the tests, which
# hold the block to them bit for bit: `moe_grouped`, `moe_small`, `moe_small_ungated`, `moe_place`, `moe_gemm`.
def moe_grouped_fits(dtype, width, ff):
    """True when `moe_grouped` takes experts of this size."""
    return bool(lib().mrs_seq_moe_grouped_fits(_i(DTYPE_CODE[dtype]), _i(width), _i(ff)))


def moe_grouped(x, up, down, experts, weights, n_routes, act, gated):
    """Expert feed-forward with every chosen expert's weights read once (a few tokens per expert, no host read): up [E, 2ff, W] (gate |
    up rows) or, not gated, [E, ff, W]; down [E, W, ff].  Expert indices from E on are identities."""
    T, W = x.shape
    top, ff, E = experts.shape[1], down.shape[2], up.shape[0]
    counts, order = moe_sort(experts, n_routes)
    hidden = torch.empty(T * top, ff, dtype=x.dtype, device=x.device)
    y = torch.empty(T * top, W, dtype=x.dtype, device=x.device)
    a = MoeGroupedArgs()
    a.x, a.up, a.down, a.dtype, a.counts, a.order = _p(x).value, _p(up).value, _p(down).value, DTYPE_CODE[x.dtype], _p(counts).value, _p(order).value
    a.n_tok, a.top, a.width, a.ff, a.n_ffn, a.gated, a.rule, a.hidden, a.y = T, top, W, ff, E, int(gated), GluRule.of(act), _p(hidden).value, _p(y).value
    _ok(lib().mrs_seq_moe_grouped(ctypes.byref(a), _st(x)), "moe_grouped")
    some = {"experts": experts, "x": x, "n_ffn": E} if n_routes > E else {}
    return moe_combine(y, None, weights, **some)


def moe_small(x, gate_up, down, experts, weights, act):
    """Expert feed-forward by weight streaming (few tokens): gate_up [E, 2ff, W], down [E, W, ff]; act: a code or a `GluRule`.
    Expert indices from E on are identities: they hand x back."""
    T, W = x.shape
    top, ff = experts.shape[1], down.shape[2]
    hidden = torch.empty(T * top, ff, dtype=x.dtype, device=x.device)
    out = torch.empty(T, W, dtype=x.dtype, device=x.device)
    a = MoeSmallArgs()
    a.x, a.gate_up, a.down, a.dtype = _p(x).value, _p(gate_up).value, _p(down).value, DTYPE_CODE[x.dtype]
    a.experts, a.weights, a.n_tok, a.top, a.width, a.ff, a.n_ffn = _p(experts).value, _p(weights).value, T, top, W, ff, gate_up.shape[0]
    a.rule, a.hidden, a.out = GluRule.of(act), _p(hidden).value, _p(out).value
    _ok(lib().mrs_seq_moe_small(ctypes.byref(a), _st(x)), "moe_small")
    return out


def moe_sort(experts, n_experts):
    n = experts.numel()
    counts = torch.empty(n_experts, dtype=torch.int32, device=experts.device)
    order = torch.empty(n, dtype=torch.int32, device=experts.device)
    _ok(lib().mrs_seq_moe_sort(_p(experts), _i(n), _i(n_experts), _p(counts), _p(order), _st(experts)), "moe_sort")
    return counts, order


def moe_gather(x, order, top, n=None):
    """The first n (None: all) sorted rows."""
    n, W = order.numel() if n is None else int(n), x.shape[1]
    out = torch.empty(n, W, dtype=x.dtype, device=x.device)
    _ok(lib().mrs_seq_moe_gather(_p(x), _i(DTYPE_CODE[x.dtype]), _p(order), _i(n), _i(top), _i(W), _p(out), _st(x)), "moe_gather")
    return out


def moe_place_fits(n_pairs, n_experts):
    return bool(lib().mrs_seq_moe_place_fits(_i(n_pairs), _i(n_experts)))


def moe_place(x, experts, n_experts):
    """`moe_sort` and `moe_gather` in one launch for few pairs (`moe_place_fits`): -> (rows sorted by expert, in each by pair; counts [n_experts]; the
    row of each pair, for `moe_combine`)."""
    n, top, W = experts.numel(), experts.shape[1], x.shape[1]
    ints = torch.empty(n_experts + n, dtype=torch.int32, device=x.device)
    counts, inverse = ints[:n_experts], ints[n_experts:]
    out = torch.empty(n, W, dtype=x.dtype, device=x.device)
    _ok(lib().mrs_seq_moe_place(_p(experts), _i(n), _i(n_experts), _p(x), _i(DTYPE_CODE[x.dtype]), _i(top), _i(W), _p(counts), _p(inverse), _p(out),
                                _st(x)), "moe_place")
    return out, counts, inverse


def moe_gemm_fits(dtype, width, ff, n_experts):
    """True when `moe_gemm` takes both products of experts of this size."""
    return dtype in DTYPE_CODE and all(lib().mrs_seq_moe_gemm_fits(_i(DTYPE_CODE[dtype]), _i(a), _i(b), _i(n_experts)) for a, b in ((ff, width), (width, ff)))


def moe_gemm(rows, weights, counts, act=ACT_NONE, gated=False):
    """One product of all experts on tcgen05: rows [n, K] sorted by expert (`moe_gather`), weights [E, N, K] or, gated, [E, 2N, K] (the
    halves joined by `act`, a code or a `GluRule`); counts from `moe_sort` stay on the device.  -> [n, N]"""
    n, k = rows.shape
    cols = weights.shape[1] // (2 if gated else 1)
    out = torch.empty(n, cols, dtype=rows.dtype, device=rows.device)
    rule = GluRule.of(act)
    _ok(lib().mrs_seq_moe_gemm(_p(rows), _p(weights), _p(counts), _i(n), _i(weights.shape[0]), _i(cols), _i(k), _i(int(gated)), ctypes.byref(rule), _p(out),
                               _st(rows)), "moe_gemm")
    return out


def moe_products(rows, up, down, counts, act, gated):
    """`moe_gemm` of up and, on its result, of down: [n, W].  The second launch begins on its weights while the first one runs."""
    n, W = rows.shape
    ff = down.shape[2]
    hidden, out = (torch.empty(n, c, dtype=rows.dtype, device=rows.device) for c in (ff, W))
    rule = GluRule.of(act)
    _ok(lib().mrs_seq_moe_products(_p(rows), _p(up), _p(down), _p(counts), _i(n), _i(up.shape[0]), _i(W), _i(ff), _i(int(gated)), ctypes.byref(rule),
                                   _p(hidden), _p(out), _st(rows)), "moe_products")
    return out


ROUTE_SOFTMAX, ROUTE_SIGMOID, ROUTE_TOP_SOFTMAX = 0, 1, 2
ONE_LAUNCH, GROUPED, STREAMED = 0, 1, 2


def moe_block(x, router, logits, correction, up, down, top, gated, act, route, products, n_groups=1, keep_groups=1, renorm=False, group_top=1,
              weight_scale=1.0, renorm_eps=0.0):
    """A routed-expert block in one call: router [routes, W] (or logits [T, routes], already formed), the rule, the experts' products by the
    kernels `products` names, the weighted sum: [T, W].  The same results as the calls it stands for."""
    T, W = x.shape
    ff, n_routes, pairs, code = down.shape[2], router.shape[0], T * top, DTYPE_CODE[x.dtype]
    out = torch.empty(T, W, dtype=x.dtype, device=x.device)
    size = pairs * (2 * W + ff) * x.element_size() + 4 * (3 * pairs + n_routes + T * n_routes) + 2048
    scratch = torch.empty(size, dtype=torch.uint8, device=x.device)
    a = MoeBlockArgs(x.data_ptr(), router.data_ptr(), logits.data_ptr() if logits is not None else None, logits.stride(0) if logits is not None else 0,
                     correction.data_ptr() if correction is not None else None, up.data_ptr(), down.data_ptr(), scratch.data_ptr(), size, out.data_ptr(),
                     code, T, W, ff, n_routes, up.shape[0], top, int(gated), route, products, n_groups, keep_groups, int(renorm), group_top, weight_scale,
                     renorm_eps, GluRule.of(act))
    _ok(lib().mrs_seq_moe_block(ctypes.byref(a), _st(x)), "moe_block")
    return out


def moe_gemm_timeouts():
    """Non-zero when a wait inside `moe_gemm`'s kernel ever ran out (synchronises)."""
    return int(lib().mrs_seq_moe_gemm_timeouts())


def moe_combine(sorted_y, order, weights, experts=None, x=None, n_ffn=0, inverse=None):
    """inverse: the row of each pair in sorted_y (`moe_place`); else order, the pair of each row (`moe_sort`); neither: sorted_y is in pair order.  With
    experts and x: the pairs of experts from n_ffn on have no rows in sorted_y, they add their token's row of x."""
    T, top = weights.shape
    W = sorted_y.shape[1]
    out = torch.empty(T, W, dtype=sorted_y.dtype, device=sorted_y.device)
    if inverse is not None:
        _ok(lib().mrs_seq_moe_combine_at(_p(sorted_y), _i(DTYPE_CODE[sorted_y.dtype]), _p(inverse), _p(weights), _p(experts), _p(x), _i(n_ffn), _i(T),
                                         _i(top), _i(W), _p(out), _st(sorted_y)), "moe_combine")
        return out
    inverse = torch.empty(T * top, dtype=torch.int32, device=sorted_y.device) if order is not None else None
    _ok(lib().mrs_seq_moe_combine_some(_p(sorted_y), _i(DTYPE_CODE[sorted_y.dtype]), _p(order), _p(weights), _p(experts), _p(x), _i(n_ffn), _i(T),
                                       _i(top), _i(W), _p(inverse), _p(out), _st(sorted_y)), "moe_combine")
    return out


# ---- single residual with Dynamic Tanh norms ------------------------------------------------------------
def tanh_norm_rows(x, norm, dtype, rows=None):
    """dyt(x[rows]) for the f32 residual x [T, W]; norm = (alpha, weight, bias) f32 on the device."""
    T, W = x.shape
    n = T if rows is None else rows.numel()
    out = torch.empty(n, W, dtype=dtype, device=x.device)
    _ok(lib().mrs_seq_tanh_norm_rows(_p(x), _p(rows), _p(norm[0]), _p(norm[1]), _p(norm[2]), _p(out), _i(DTYPE_CODE[dtype]), _i(n), _i(W),
                                     _st(x)), "tanh_norm_rows")
    return out


def residual_tanh_norm(x, y=None, post=None, extra=None, nxt=None, dtype=None):
    """In place on the f32 residual: x += dyt_post(y); x += extra; returns dyt_next(x) when nxt is given (each part optional)."""
    T, W = x.shape
    dtype = y.dtype if y is not None else dtype
    out = torch.empty(T, W, dtype=dtype, device=x.device) if nxt is not None else None
    post, nxt = post or (None, None, None), nxt or (None, None, None)
    _ok(lib().mrs_seq_residual_tanh_norm(_p(x), _p(y), _i(DTYPE_CODE[dtype]), _p(post[0]), _p(post[1]), _p(post[2]), _p(extra), _p(nxt[0]),
                                         _p(nxt[1]), _p(nxt[2]), _p(out), _i(T), _i(W), _st(x)), "residual_tanh_norm")
    return out


# ---- attention: general preparation, rotation table, sink / kept-first window ---------------------------
def rotation_table(pos_of_tok, freq, mag):
    """f32 [T, half, 2]: mag * (cos, sin)(pos * freq), angles in double.  freq: f64 on the device."""
    T, half = pos_of_tok.numel(), freq.numel()
    out = torch.empty(T, half, 2, dtype=torch.float32, device=freq.device)
    _ok(lib().mrs_seq_rotation_table(_p(pos_of_tok), _p(freq), _i(T), _i(half), _f(mag), _p(out), _st(freq)), "rotation_table")
    return out


def attention_prepare(y, q_col, k_col, v_col, norm_mode, q_norm_w, k_norm_w, eps, heads, kv_heads, dk, dv, k_cache, v_cache, slot_of_tok,
                      cos_sin=None, rot_dims=0, pairing=PAIRS_HALVES, norm_last=False):
    """q | k | v are column ranges of y.  v_col None: the values are the keys as projected.  pairing: which two entries of a
    head turn together.  Norm weights None: ones.  norm_last: the norm is taken of the rotated heads."""
    a = AttnPrepareArgs()
    ld = y.stride(0)
    a.q, a.k, a.q_ld, a.k_ld = _p(y, q_col).value, _p(y, k_col).value, ld, ld
    if v_col is not None:
        a.v, a.v_ld = _p(y, v_col).value, ld
    a.dtype, a.norm_mode = DTYPE_CODE[y.dtype], norm_mode
    a.q_norm_w, a.k_norm_w, a.eps = _p(q_norm_w).value, _p(k_norm_w).value, eps
    a.heads, a.kv_heads, a.dk, a.dv = heads, kv_heads, dk, dv
    a.rot_dims, a.cos_sin, a.pairing, a.norm_last = rot_dims, _p(cos_sin).value, pairing, int(bool(norm_last))
    a.k_cache, a.v_cache, a.slot_of_tok, a.n_tok = k_cache.data_ptr(), v_cache.data_ptr(), slot_of_tok.data_ptr(), y.shape[0]
    _ok(lib().mrs_seq_attention_prepare(ctypes.byref(a), _st(y)), "attention_prepare")


def paged_attention(y, q_col, k_cache, v_cache, heads, kv_heads, dk, dv, scale, window, keep_first, sink, batch, page_size, out, out_col=0,
                    out_scale=1.0, tok_index=None, k_row=0, v_row=0, pool=0, pool_base=0, v_shared=False, v_col=0, out_head=0,
                    chunk=0, gate=None, gate_col=0, gate_group=1, gate_act=ACT_NONE):
    """Every token of the step (or those listed in tok_index) against the pages of its sequence: position i sees j <= i
    with i - j < window (0: all) or j < keep_first; sink [heads] f32 or None.  k_row / v_row: elements between the cache
    rows of neighbouring slots (0: kv_heads * dk / kv_heads * dv).  pool > 0: besides the window, one averaged entry per
    block of `pool` positions wholly before it, read from cache rows pool_base.. (`pool_blocks`).  v_shared: every head
    reads value columns [v_col, v_col + dv) of a row — dv is then several (or all) value heads side by side, and out_head the
    distance between the heads of an output row.  An f32 `out` is written as f32 whatever the activation type.
    chunk > 0: a position sees only its own chunk of `chunk` positions, counted from position 0.  gate: the result is multiplied by
    gate_act of gate's columns from gate_col, one per `gate_group` neighbouring entries (1 or dv)."""
    a = PagedAttentionArgs()
    if gate is not None:
        a.gate, a.gate_ld, a.gate_group, a.gate_act = _p(gate, gate_col).value, gate.stride(0), gate_group, gate_act
    a.k_row, a.v_row = int(k_row), int(v_row)
    a.pool, a.pool_base, a.v_shared = int(pool), int(pool_base), int(bool(v_shared))
    a.out_f32 = int(out.dtype == torch.float32 and y.dtype != torch.float32)
    a.q, a.q_ld, a.k_cache, a.v_cache = _p(y, q_col).value, y.stride(0), k_cache.data_ptr(), _p(v_cache, int(v_col)).value
    a.out_head, a.chunk = int(out_head), int(chunk)
    a.dtype, a.heads, a.kv_heads, a.dk, a.dv = DTYPE_CODE[y.dtype], heads, kv_heads, dk, dv
    a.scale, a.window, a.keep_first, a.sink = scale, int(window), int(keep_first), _p(sink).value
    a.pages, a.pages_ld, a.page_size = batch.pages.data_ptr(), batch.pages.shape[1], page_size
    a.seq_of_tok, a.pos_of_tok, a.tok_index = batch.seq_of_tok.data_ptr(), batch.pos_of_tok.data_ptr(), _p(tok_index).value
    a.n_tok = y.shape[0] if tok_index is None else tok_index.numel()
    a.out, a.out_ld, a.out_scale = _p(out, out_col).value, out.stride(0), out_scale
    _ok(lib().mrs_seq_paged_attention(ctypes.byref(a), _st(y)), "paged_attention")


def tc_attention_fits(dn, dr, dv, *multiples_of_8):
    """True when `tc_attention` takes these head sizes (bf16) and every given stride / first column keeps rows 16-byte aligned."""
    return all(int(v) % 8 == 0 for v in multiples_of_8) and bool(lib().mrs_seq_prompt_attention_tc_fits(_i(dn), _i(dr), _i(dv)))


def tc_attention(q, q_col, k, k_col, v, v_col, segments, n_segments, longest, heads, kv_heads, dn, dr, dv, scale, out, out_col=0, k_shared=None,
                 k_shared_col=0, gate=None, gate_col=0, gate_group=1, gate_act=ACT_NONE, window=0, keep_first=0, held=None, sink=None):
    """Causal attention of segments over DENSE keys and values on tcgen05 (bf16): segments int32 [n, 4] on the device = first query
    row, query rows, first key row, keys before the first query.  q rows: heads * (dn + dr) columns from q_col; k: kv_heads * dn;
    v: kv_heads * dv; k_shared: dr further key columns all heads share.  gate, window, keep_first, sink: as for `paged_attention`;
    held int32 [n, 2]: which positions a segment's dense rows are (`engine.DensePlan.held`; None: every position)."""
    a = PromptAttentionTcArgs()
    a.q, a.k, a.v, a.q_ld, a.k_ld, a.v_ld = _p(q, q_col).value, _p(k, k_col).value, _p(v, v_col).value, q.stride(0), k.stride(0), v.stride(0)
    a.q_rows, a.k_rows = q.shape[0], k.shape[0]
    if dr > 0:
        a.k_shared, a.k_shared_ld = _p(k_shared, k_shared_col).value, k_shared.stride(0)
    a.out, a.out_ld = _p(out, out_col).value, out.stride(0)
    a.segments, a.n_segments, a.longest = segments.data_ptr(), int(n_segments), int(longest)
    a.heads, a.kv_heads, a.dn, a.dr, a.dv, a.scale = heads, kv_heads, dn, dr, dv, float(scale)
    if gate is not None:
        a.gate, a.gate_ld, a.gate_group, a.gate_act = _p(gate, gate_col).value, gate.stride(0), gate_group, gate_act
    a.window, a.keep_first, a.held, a.sink = int(window), int(keep_first), _p(held).value, _p(sink).value
    _ok(lib().mrs_seq_prompt_attention_tc(ctypes.byref(a), _st(q)), "prompt_attention_tc")


def tc_attention_timeouts():
    """Non-zero when a wait inside `tc_attention`'s kernel ever ran out (synchronises)."""
    return int(lib().mrs_seq_prompt_attention_tc_timeouts())


def gather_rows(cache, cols, runs, n_runs, longest, batch, page_size, n_rows):
    """Dense rows [n_rows, cols] of a token-indexed cache [slots, >= cols]: runs int32 [n, 4] on the device = sequence, first
    position, positions, first dense row.  Rows are whole 16-byte groups."""
    out = torch.empty(n_rows, cols, dtype=cache.dtype, device=cache.device)
    size = cache.element_size()
    _ok(lib().mrs_seq_gather_rows(_p(cache), _l(cache.stride(0) * size), _i(cols * size), _p(runs), _i(n_runs), _i(longest), _p(batch.pages),
                                  _i(batch.pages.shape[1]), _i(page_size), _p(out), _l(cols * size), _st(cache)), "gather_rows")
    return out


def pool_rows(n_token_slots, page_size, pool):
    """Cache rows that the averaged blocks of a pool of n_token_slots token rows need (per page: as many as blocks can start in one)."""
    return (n_token_slots // page_size) * (-(-page_size // pool))


def pool_blocks(k_cache, v_cache, k_cols, v_cols, pool, pool_base, batch, page_size):
    """For every token of the step that ends a block of `pool` positions: the block's mean key / value row -> its cache row."""
    _ok(lib().mrs_seq_pool_blocks(_p(k_cache), _p(v_cache), _i(DTYPE_CODE[k_cache.dtype]), _l(k_cols), _l(v_cols), _i(k_cols), _i(v_cols),
                                  _i(pool), _l(pool_base), _p(batch.pages), _i(batch.pages.shape[1]), _i(page_size), _p(batch.seq_of_tok),
                                  _p(batch.pos_of_tok), _i(batch.n_tok), _st(k_cache)), "pool_blocks")


def mix_heads(a, mix, heads, kv_heads, dv, out, gate=None, gate_col=0, gate_act=ACT_NONE):
    """out[t, h] = act(gate[t, h]) * sum_g mix[h, g] * a[t, g, value head of h]; a f32 [T, heads * kv_heads * dv]."""
    _ok(lib().mrs_seq_mix_heads(_p(a), _p(mix), _p(gate, gate_col) if gate is not None else _p(None), _l(gate.stride(0) if gate is not None else 0),
                                _i(gate_act), _p(out), _l(out.stride(0)), _i(DTYPE_CODE[out.dtype]), _i(heads), _i(kv_heads), _i(dv),
                                _i(out.shape[0]), _st(out)), "mix_heads")


def gate_cols(x, gate, gate_col, cols, group, act):
    """x[:, c] *= act(gate[:, gate_col + c // group]) in place for c < cols."""
    _ok(lib().mrs_seq_gate_cols(_p(x), _l(x.stride(0)), _p(gate, gate_col), _l(gate.stride(0)), _i(DTYPE_CODE[x.dtype]), _i(cols), _i(group),
                                _i(act), _i(x.shape[0]), _st(x)), "gate_cols")


def prompt_attention(y, q_col, k_cache, v_cache, batch, page_size, heads, kv_heads, d, scale, window, keep_first, sink, out, out_col=0, pool=0,
                     pool_base=0, every_value_head=False, chunk=0, gate=None, gate_col=0, gate_group=1, gate_act=ACT_NONE):
    """The long portions of the step (batch.long: fresh or continued) on tensor cores: queries from their rows of y, keys
    and values from the pages (bf16, head size 64 or 128).  pool / pool_base: averaged blocks before the window, as for
    `paged_attention`.  every_value_head: `out` is f32 [T, heads * kv_heads * d], every head's weights on every value head.
    chunk > 0: a position sees only its own chunk of `chunk` positions, counted from position 0.  gate: as for `paged_attention`."""
    a = PromptAttentionArgs()
    if gate is not None:
        a.gate, a.gate_ld, a.gate_group, a.gate_act = _p(gate, gate_col).value, gate.stride(0), gate_group, gate_act
    a.q, a.q_ld, a.k_cache, a.v_cache = _p(y, q_col).value, y.stride(0), k_cache.data_ptr(), v_cache.data_ptr()
    a.out, a.out_ld = _p(out, out_col).value, out.stride(0)
    a.portions, a.n_portions, a.longest = batch.long_rows.data_ptr(), len(batch.long), max(n for _, n, _, _ in batch.long)
    a.pages, a.pages_ld, a.page_size = batch.pages.data_ptr(), batch.pages.shape[1], page_size
    a.heads, a.kv_heads, a.d, a.scale = heads, kv_heads, d, float(scale)
    a.window, a.keep_first, a.sink = int(window), int(keep_first), _p(sink).value
    a.pool, a.pool_base, a.every_value_head, a.chunk = int(pool), int(pool_base), int(bool(every_value_head)), int(chunk)
    _ok(lib().mrs_seq_prompt_attention_general(ctypes.byref(a), _st(y)), "prompt_attention")


# ---- stabilised matrix memory ---------------------------------------------------------------------------
def mlstm_gates(raw, heads, cap, m_state, batch):
    """raw f32 [T, 2 * heads] (input gates | forget gates, biases added) -> keep, take, m f32 [T, heads]; advances m_state."""
    T = raw.shape[0]
    keep = torch.empty(T, heads, dtype=torch.float32, device=raw.device)
    take, m_tok = torch.empty_like(keep), torch.empty_like(keep)
    _ok(lib().mrs_seq_mlstm_gates(_p(raw), _p(raw, heads), _l(raw.stride(0)), _f(cap), _i(heads), _p(m_state), _p(batch.cu_tok),
                                  _p(batch.past), _p(batch.slot), _i(batch.n_seq), _i(T), _p(keep), _p(take), _p(m_tok), _st(raw)),
        "mlstm_gates")
    return keep, take, m_tok


def append_ones(y, v_col, heads, dv, dvp):
    out = torch.empty(y.shape[0], heads * dvp, dtype=y.dtype, device=y.device)
    _ok(lib().mrs_seq_append_ones(_p(y, v_col), _l(y.stride(0)), _i(DTYPE_CODE[y.dtype]), _i(heads), _i(dv), _i(dvp), _i(y.shape[0]), _p(out),
                                  _st(y)), "append_ones")
    return out


def mlstm_out_norm(o, dvp, m_tok, q_scale, gate, gate_col, weight, eps, heads, dv, dtype):
    T = o.shape[0]
    out = torch.empty(T, heads * dv, dtype=dtype, device=o.device)
    _ok(lib().mrs_seq_mlstm_out_norm(_p(o), _i(dvp), _p(m_tok), _f(q_scale), _p(gate, gate_col), _l(gate.stride(0)), _p(weight), _f(eps),
                                     _i(heads), _i(dv), _p(out), _l(out.stride(0)), _i(DTYPE_CODE[dtype]), _i(T), _st(o)), "mlstm_out_norm")
    return out


# ---- experts: plain top-k rule, experts without a gate -----------------------------------------------------
def moe_route_top_softmax(logits, top):
    T, E = logits.shape
    experts = torch.empty(T, top, dtype=torch.int32, device=logits.device)
    weights = torch.empty(T, top, dtype=torch.float32, device=logits.device)
    _ok(lib().mrs_seq_moe_route_top_softmax(_p(logits), _i(T), _i(E), _i(top), _p(experts), _p(weights), _st(logits)), "moe_route_top_softmax")
    return experts, weights


def moe_small_ungated(x, up, down, experts, weights, act):
    """Expert feed-forward without a gate by weight streaming (few tokens): up [E, ff, W], down [E, W, ff]."""
    T, W = x.shape
    top, ff = experts.shape[1], down.shape[2]
    code = _i(DTYPE_CODE[x.dtype])
    hidden = torch.empty(T * top, ff, dtype=x.dtype, device=x.device)
    out = torch.empty(T, W, dtype=x.dtype, device=x.device)
    _ok(lib().mrs_seq_moe_up(_p(x), _p(up), code, _p(experts), _i(T), _i(top), _i(W), _i(ff), _i(act), _p(hidden), _st(x)), "moe_up")
    _ok(lib().mrs_seq_moe_down(_p(hidden), _p(down), code, _p(experts), _p(weights), _i(T), _i(top), _i(W), _i(ff), _p(out), _st(x)),
        "moe_down")
    return out


# ---- single residual with RMS norms, a multiplier and a depth-weighted average ---------------------------------
def embed_scaled(table, ids, scale, out):
    """out f32 [T, W] = table[ids] * scale."""
    T, W = ids.numel(), table.shape[1]
    _ok(lib().mrs_seq_embed_scaled(_p(table), _i(DTYPE_CODE[table.dtype]), _p(ids), _f(scale), _p(out), _i(T), _i(W), _st(table)), "embed_scaled")
    return out


def embed_pair(table, pairs, ids, scale, buckets, mul_prev, mul_cur, prev_state, batch, out):
    """out f32 [T, W] = table[ids] * scale + pairs[hash of (previous token, token)]; the table's last row for a sequence's first
    token; prev_state int32 [slots] carries every request's last token from step to step."""
    T, W = ids.numel(), table.shape[1]
    _ok(lib().mrs_seq_embed_pair(_p(table), _p(pairs), _i(DTYPE_CODE[table.dtype]), _p(ids), _f(scale), _l(buckets), _l(mul_prev), _l(mul_cur),
                                 _p(prev_state), _p(batch.cu_tok), _p(batch.past), _p(batch.slot), _p(batch.seq_of_tok), _p(out), _i(T), _i(W),
                                 _st(table)), "embed_pair")
    return out


def rms_residual(src, y=None, mult=1.0, dst=None, hist=None, n_hist=0, mix=None, mixed=None, next_w=None, eps=0.0, dtype=None, post_w=None,
                 add_vec=None, next_b=None, center=False, rows=None, post_center=False, plain_out=None):
    """One pass over an f32 residual [T, W]: v = src + mult * y (y first RMS-normed with post_w when given) + add_vec [W] -> dst;
    v = sum_j mix[j] * hist[j] (hist f32 [>= n_hist, T, W], dst may be one of its entries) -> mixed; returns rms_norm(v) * next_w
    in the activation type when next_w is given — with `center` a layer norm (mean taken off) and with next_b a bias.  rows: the
    norm of these rows of src only (nothing else then happens).  post_center: y's norm is a layer norm.  plain_out [T, W] (without
    next_w): v itself is written there, in its type."""
    T, W = src.shape
    T = T if rows is None else rows.numel()
    dtype = y.dtype if y is not None else dtype
    if plain_out is not None and (next_w is not None or plain_out.dtype != dtype):
        raise ValueError("plain_out takes the residual as it is, in the activation type")
    out = torch.empty(T, W, dtype=dtype, device=src.device) if next_w is not None else plain_out
    a = RmsResidualArgs()
    a.src, a.dst, a.y, a.mult = _p(src).value, _p(dst).value, _p(y).value, float(mult)
    if hist is not None:
        a.hist, a.hist_stride, a.n_hist, a.mix = _p(hist).value, hist.stride(0), int(n_hist), _p(mix).value
    a.mixed, a.next_w, a.eps, a.next_out = _p(mixed).value, _p(next_w).value, float(eps), _p(out).value
    a.dtype, a.n_tok, a.width = DTYPE_CODE[dtype], T, W
    a.post_w, a.add_vec = _p(post_w).value, _p(add_vec).value
    a.next_b, a.center, a.rows, a.post_center = _p(next_b).value, int(bool(center)), _p(rows).value, int(bool(post_center))
    _ok(lib().mrs_seq_rms_residual(ctypes.byref(a), _st(src)), "rms_residual")
    return out


GATED_LOOKUP_SMALL = 8      # up to this many tokens the gate's product is formed inside the lookup kernel


def gated_lookup(x, w_gate, table, col0, ids, act):
    """[T, dim] in the activation type: act(w_gate x) * table[ids, col0:col0 + dim], w_gate [dim, W]."""
    T, W, dim = x.shape[0], x.shape[1], w_gate.shape[0]
    out = torch.empty(T, dim, dtype=x.dtype, device=x.device)
    code, rows, ld = _i(DTYPE_CODE[x.dtype]), _p(table, col0), _l(table.stride(0))
    if T <= GATED_LOOKUP_SMALL and W * 4 <= 48 * 1024:
        _ok(lib().mrs_seq_gated_lookup_small(_p(x), _p(w_gate), rows, ld, _p(ids), code, _i(act), _i(W), _i(dim), _i(T), _p(out), _st(x)),
            "gated_lookup_small")
        return out
    gate = torch.nn.functional.linear(x, w_gate)
    _ok(lib().mrs_seq_gated_lookup(_p(gate), rows, ld, _p(ids), code, _i(act), _i(dim), _i(T), _p(out), _st(x)), "gated_lookup")
    return out


def soft_cap(x, scale, cap):
    """f32 cap * tanh(scale * x / cap) (cap 0: scale * x): logits with a multiplier and a soft cap."""
    out = torch.empty(x.shape, dtype=torch.float32, device=x.device)
    _ok(lib().mrs_seq_soft_cap(_p(x), _i(DTYPE_CODE[x.dtype]), _f(scale), _f(cap), _l(x.numel()), _p(out), _st(x)), "soft_cap")
    return out


# ---- attention through a shared latent -----------------------------------------------------------------------
def latent_prepare(y, q_col, q_rank, q_norm_w, q_out, kv_col, kv_rank, rot_dim, rot_dims, kv_norm_w, cos_sin, eps, cache, slot_of_tok, kv_out=None,
                   pairing=PAIRS_NEIGHBOURS, rotate_q=None):
    """From the columns of y: q_out = rms_norm(query latent) * w; cache[slot] = rms_norm(key/value latent) * w | the shared key
    part turned in pairs (`pairing`).  kv_rank 0: only the query part.  kv_out [T, >= kv_rank]: the normed latent (and, with
    room for it, the shared key part) also as dense rows.  rotate_q = (heads, first column in y, columns between heads, out, first
    column in out, columns between heads in out): the queries' rotated parts [rot_dim] turn in the same pass (out may be y)."""
    a = LatentPrepareArgs()
    a.y, a.y_ld, a.dtype = _p(y).value, y.stride(0), DTYPE_CODE[y.dtype]
    a.q_col, a.q_rank, a.q_norm_w = int(q_col), int(q_rank), _p(q_norm_w).value
    if q_out is not None:
        a.q_out, a.q_out_ld = _p(q_out).value, q_out.stride(0)
    a.kv_col, a.kv_rank, a.rot_dim, a.rot_dims = int(kv_col), int(kv_rank), int(rot_dim), int(rot_dims)
    a.kv_norm_w, a.cos_sin, a.eps = _p(kv_norm_w).value, _p(cos_sin).value, float(eps)
    if kv_rank:
        a.cache, a.cache_row, a.slot_of_tok = _p(cache).value, cache.stride(0), _p(slot_of_tok).value
    a.n_tok, a.pairing = y.shape[0], pairing
    if kv_out is not None:
        a.kv_out, a.kv_out_ld = _p(kv_out).value, kv_out.stride(0)
    if rotate_q is not None:
        heads, col, step, dst, dst_col, dst_step = rotate_q
        a.rq_heads, a.rq_col, a.rq_head = int(heads), int(col), int(step)
        a.rq_out, a.rq_out_ld, a.rq_out_head = _p(dst, dst_col).value, dst.stride(0), int(dst_step)
    _ok(lib().mrs_seq_latent_prepare(ctypes.byref(a), _st(y)), "latent_prepare")


def rotate_pairs(src, src_col, src_head, dst, dst_col, dst_head, heads, dims, rot_dims, cos_sin, pairing=PAIRS_NEIGHBOURS):
    """dst[t, dst_col + h * dst_head + d] = src[t, src_col + h * src_head + d], d < dims, the first rot_dims turned in
    pairs (`pairing`) by cos_sin [T, rot_dims / 2, 2]."""
    _ok(lib().mrs_seq_rotate_heads(_p(src, src_col), _l(src.stride(0)), _l(src_head), _p(dst, dst_col), _l(dst.stride(0)), _l(dst_head),
                                   _i(DTYPE_CODE[src.dtype]), _i(heads), _i(dims), _i(rot_dims), _i(pairing), _p(cos_sin), _i(src.shape[0]),
                                   _st(src)),
        "rotate_pairs")


def latent_attention_fits(kv_rank, rot_dim):
    """True when the tensor-core latent kernel takes these sizes (bf16 only)."""
    return bool(lib().mrs_seq_latent_attention_fits(_i(kv_rank), _i(rot_dim)))


def latent_prompt_attention(qa, latent, heads, kv_rank, rot_dim, scale, window, batch, page_size, out, portions=None, n_portions=0, longest=0):
    """Absorbed latent attention on tensor cores of every sequence of the step — prompt portions of any length and single
    decoded tokens alike (a token's heads are rows of one tile; the window's latents are fetched once for all of them) — or of
    the given portions int32 [n, 4] on the device (first row of qa / out, rows, positions cached before, sequence).  Steps too
    small to fill the GPU share a row tile's keys among several CTAs."""
    a = LatentAttentionArgs()
    a.q, a.q_ld, a.cache, a.cache_row, a.out, a.out_ld = _p(qa).value, qa.stride(0), _p(latent).value, latent.stride(0), _p(out).value, out.stride(0)
    if portions is None:
        a.cu_tok, a.past, a.n_portions, a.longest = batch.cu_tok.data_ptr(), batch.past.data_ptr(), batch.n_seq, batch.longest
    else:
        a.portions, a.n_portions, a.longest = portions.data_ptr(), int(n_portions), int(longest)
    a.pages, a.pages_ld, a.page_size = batch.pages.data_ptr(), batch.pages.shape[1], page_size
    a.heads, a.kv_rank, a.rot_dim, a.scale, a.window = heads, kv_rank, rot_dim, float(scale), int(window)
    reach = batch.pages.shape[1] * page_size                     # the same for every replay of a captured step
    floats = ctypes.c_int64(0)
    a.splits = lib().mrs_seq_latent_attention_plan(_i(a.n_portions), _i(a.longest), _i(heads), _i(kv_rank),
                                                   _i(min(reach, window) if window > 0 else reach), ctypes.byref(floats))
    if a.splits > 1:
        scratch = torch.empty(floats.value, dtype=torch.float32, device=qa.device)
        a.scratch = scratch.data_ptr()
    _ok(lib().mrs_seq_latent_attention_general(ctypes.byref(a), _st(qa)), "latent_attention")


def latent_attention(qa, latent, heads, kv_rank, rot_dim, scale, window, batch, page_size, out, tok_index=None):
    """Absorbed latent attention of every token of the step: qa [T, heads * (kv_rank + rot_dim)] against the cached latent
    rows [slots, >= kv_rank + rot_dim] as one key/value head (values = the rows' first kv_rank columns); out [T, heads * kv_rank]."""
    paged_attention(qa, 0, latent, latent, heads, 1, kv_rank + rot_dim, kv_rank, scale, window, 0, None, batch, page_size, out,
                    tok_index=tok_index, k_row=latent.stride(0), v_row=latent.stride(0))
