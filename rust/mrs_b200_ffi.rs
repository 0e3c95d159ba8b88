//! B200-native entry points of libmrs_b200 (GENERATED by scripts/gen_rust_ffi.py from include/*.h — do not edit).
//! Link with `cargo:rustc-link-lib=dylib=mrs_b200` (and `dylib=mrs_b200_seq` for the mrs_seq_* entry points of mrs_b200_seq.h); the reference-named symbols are declared by the
//! reference's own ffi.rs files and resolve against the same library.
#![allow(dead_code)]
use std::ffi::c_void;

extern "C" {
    // ---- mrs_b200_model.h
    pub fn mrs_tp_allreduce_residual(ctx: *const c_void, slot: i32, residual: *const c_void, out: *mut c_void, count: i32, dtype: i32, pdl: i32, stream: *mut c_void) -> i32;
    pub fn mrs_llama_resident_bytes(n_heads: i32, head_dim: i32, padded_tiles: i32) -> i64;
    pub fn mrs_llama_decode_step(s: *const c_void, stream: *mut c_void) -> i32;
    pub fn mrs_decode_advance(block_tables: *const i32, max_blocks_per_seq: i32, context_lens: *mut i32, batch: i32, block_size: i32, split_pages: i32, padded_tiles: i32, positions: *mut i32, slot_mapping: *mut i64, kv_indptr: *mut i32, kv_indices: *mut i32, kv_last_page_len: *mut i32, request_indices: *mut i32, kv_tile_indices: *mut i32, o_indptr: *mut i32, kv_chunk_size: *mut i32, block_valid_mask: *mut u8, max_pos: i32, error_flag: *mut i32, stream: *mut c_void) -> i32;
    pub fn mrs_embedding_gather(ggml_type: i32, table: *const c_void, cols: i32, ids: *const i32, n: i32, out: *mut c_void, act_dtype: i32, stream: *mut c_void) -> i32;
    pub fn mrs_argmax(logits: *const c_void, rows: i32, cols: i32, act_dtype: i32, out: *mut i32, scratch: *mut c_void, pdl: i32, stream: *mut c_void) -> i32;
    pub fn mrs_gptq_decode_step(s: *const c_void, stream: *mut c_void) -> i32;
    pub fn mrs_w4a16_gemm_pdl(x: *const c_void, w_tiles: *const c_void, scales: *const c_void, qzeros: *const i32, y: *mut c_void, M: i32, K: i32, N: i32, group: i32, dtype: i32, scale_perm: i32, pdl: i32, stream: *mut c_void) -> i32;
    pub fn mrs_dense_linear_pdl(x: *const c_void, w: *const c_void, y: *mut c_void, M: i32, K: i32, N: i32, dtype: i32, pdl: i32, stream: *mut c_void) -> i32;
    pub fn mrs_add_rms_norm_pdl(x: *const c_void, residual: *const c_void, weight: *const c_void, residual_dst: *mut c_void, norm_dst: *mut c_void, nrows: i32, ncols: i32, eps: f32, dtype: i32, pdl: i32, stream: *mut c_void);
    pub fn mrs_split_glu_pdl(input: *const c_void, output: *mut c_void, rows: u32, split_size: u32, activation: i32, dtype: i32, pdl: i32, stream: *mut c_void);
    // ---- mrs_b200_ops.h
    pub fn mrs_rms_norm_f16(x: *const c_void, weight: *const c_void, dst: *mut c_void, nrows: i32, ncols: i32, eps: f32, stream: i64);
    pub fn mrs_rms_norm_bf16(x: *const c_void, weight: *const c_void, dst: *mut c_void, nrows: i32, ncols: i32, eps: f32, stream: i64);
    pub fn mrs_rms_norm_f32(x: *const c_void, weight: *const c_void, dst: *mut c_void, nrows: i32, ncols: i32, eps: f32, stream: i64);
    // ---- mrs_b200_paged_attn.h
    pub fn mrs_swap_blocks(src: *const c_void, dst: *mut c_void, block_bytes: i64, pairs: *const i64, n_pairs: i64, stream: *mut c_void) -> i32;
    pub fn mrs_paged_decode_fused(q: *mut c_void, k_new: *mut c_void, v_new: *mut c_void, key_cache: *mut c_void, value_cache: *mut c_void, rope_cos: *const c_void, rope_sin: *const c_void, positions: *const i32, slot_mapping: *const i64, kv_indptr: *const i32, kv_indices: *const i32, kv_last_page_len: *const i32, request_indices: *const i32, kv_tile_indices: *const i32, o_indptr: *const i32, kv_chunk_size_ptr: *const i32, block_valid_mask: *const u8, o: *mut c_void, tmp_v: *mut c_void, tmp_s: *mut f32, counters: *mut i32, batch_size: i32, padded_batch_size: i32, num_qo_heads: i32, num_kv_heads: i32, head_size: i32, page_size: i32, sm_scale: f32, dtype: u32, pdl: i32, stream: *mut c_void) -> i32;
    pub fn mrs_paged_decode_fused_strided(q: *mut c_void, k_new: *mut c_void, v_new: *mut c_void, key_cache: *mut c_void, value_cache: *mut c_void, rope_cos: *const c_void, rope_sin: *const c_void, positions: *const i32, slot_mapping: *const i64, kv_indptr: *const i32, kv_indices: *const i32, kv_last_page_len: *const i32, request_indices: *const i32, kv_tile_indices: *const i32, o_indptr: *const i32, kv_chunk_size_ptr: *const i32, block_valid_mask: *const u8, o: *mut c_void, tmp_v: *mut c_void, tmp_s: *mut f32, counters: *mut i32, batch_size: i32, padded_batch_size: i32, num_qo_heads: i32, num_kv_heads: i32, head_size: i32, page_size: i32, sm_scale: f32, dtype: u32, pdl: i32, q_stride_n: i64, kv_new_stride: i64, stream: *mut c_void) -> i32;
    pub fn mrs_prefill_attention(q: *const c_void, k: *const c_void, v: *const c_void, out: *mut c_void, cu_seqlens: *const i32, batch: i32, total_tokens: i32, max_seqlen: i32, num_heads: i32, num_kv_heads: i32, head_dim: i32, q_stride: i64, kv_stride: i64, o_stride: i64, softmax_scale: f32, causal: i32, window_left: i32, softcap: f32, dtype: u32, stream: *mut c_void) -> i32;
    pub fn mrs_prefill_attention_tc(q: *const c_void, k: *const c_void, v: *const c_void, out: *mut c_void, cu_seqlens: *const i32, batch: i32, total_tokens: i32, max_seqlen: i32, num_heads: i32, num_kv_heads: i32, head_dim: i32, q_stride: i64, kv_stride: i64, o_stride: i64, softmax_scale: f32, causal: i32, window_left: i32, softcap: f32, dtype: u32, stream: *mut c_void) -> i32;
    pub fn mrs_prefill_attn_tc_debug(enable: i32, lbo: u32, sbo: u32);
    pub fn mrs_set_attn_flags(flags: i32);
    // ---- mrs_b200_quant.h
    pub fn mrs_set_pdl(enabled: i32);
    pub fn mrs_set_mmvq_flags(flags: i32);
    pub fn mrs_set_mmvq_ctas_per_sm(n: i32);
    pub fn mrs_mmvq_has_wide() -> i32;
    pub fn mrs_mmvq_fused(ggml_type: i32, mode: i32, dt: i32, w0: *const c_void, w1: *const c_void, w2: *const c_void, x: *const c_void, norm_w: *const c_void, eps: f32, residual: *const c_void, dst0: *mut c_void, dst1: *mut c_void, dst2: *mut c_void, K: i32, n0: i32, n1: i32, n2: i32, b_size: i32, activation: i32, pdl: i32, stream: *mut c_void) -> i32;
    pub fn mrs_rms_quantize_q8_1(dt: i32, x: *const c_void, norm_w: *const c_void, eps: f32, K: i32, b_size: i32, q8: *mut c_void, pdl: i32, stream: *mut c_void) -> i32;
    pub fn mrs_mmvq_q8(ggml_type: i32, mode: i32, dt: i32, w0: *const c_void, w1: *const c_void, w2: *const c_void, q8: *const c_void, residual: *const c_void, dst0: *mut c_void, dst1: *mut c_void, dst2: *mut c_void, K: i32, n0: i32, n1: i32, n2: i32, b_size: i32, activation: i32, pdl: i32, stream: *mut c_void) -> i32;
    pub fn mrs_mmvq_rows(ggml_type: i32, mode: i32, dt: i32, w0: *const c_void, w1: *const c_void, w2: *const c_void, x: *const c_void, q8: *mut c_void, dst0: *mut c_void, dst1: *mut c_void, dst2: *mut c_void, K: i32, n0: i32, n1: i32, n2: i32, b_size: i32, activation: i32, stream: *mut c_void) -> i32;
    pub fn mrs_mmvq_fused_qkv_mixed(type_qk: i32, type_v: i32, dt: i32, wq: *const c_void, wk: *const c_void, wv: *const c_void, x: *const c_void, norm_w: *const c_void, eps: f32, q: *mut c_void, k: *mut c_void, v: *mut c_void, K: i32, nq: i32, nk: i32, nv: i32, b_size: i32, pdl: i32, stream: *mut c_void) -> i32;
    pub fn mrs_mmq_gguf(ggml_type: i32, w: *const c_void, x: *const c_void, y: *mut c_void, M: i32, N: i32, K: i32, dtype: i32, stream: *mut c_void) -> i32;
    pub fn mrs_mmq_set_weight_format(fmt: i32);
    pub fn mrs_mmq_set_path(path: i32);
    pub fn mrs_mmq_gguf_ts(ggml_type: i32, w: *const c_void, x: *const c_void, y: *mut c_void, M: i32, N: i32, K: i32, dtype: i32, stream: *mut c_void) -> i32;
    pub fn mrs_mmq_gguf_multi(ggml_type: i32, w0: *const c_void, w1: *const c_void, w2: *const c_void, x: *const c_void, y0: *mut c_void, y1: *mut c_void, y2: *mut c_void, M: i32, n0: i32, n1: i32, n2: i32, K: i32, dtype: i32, stream: *mut c_void) -> i32;
    pub fn mrs_mmq_timeouts() -> i32;
    pub fn mrs_mmq_timeout_flag() -> *mut i32;
    pub fn mrs_gptq_gemm(x: *const c_void, qweight: *const i32, scales: *const c_void, qzeros: *const i32, g_idx: *const i32, y: *mut c_void, M: i32, K: i32, N: i32, group_size: i32, is_awq: i32, stream: *mut c_void) -> i32;
    pub fn mrs_marlin_4bit(inputs: *const c_void, weight: *const i32, scales: *const c_void, zeros: *const c_void, out: *mut c_void, m: i32, k: i32, n: i32, groupsize: i32, dtype: i32, scale_dtype: i32, is_awq: i32, stream: i64) -> i32;
    pub fn mrs_w4a16_gemm(x: *const c_void, w_tiles: *const c_void, scales: *const c_void, qzeros: *const i32, y: *mut c_void, M: i32, K: i32, N: i32, group: i32, dtype: i32, scale_perm: i32, stream: *mut c_void) -> i32;
    pub fn mrs_dense_linear(x: *const c_void, w: *const c_void, y: *mut c_void, M: i32, K: i32, N: i32, dtype: i32, stream: *mut c_void) -> i32;
    pub fn mrs_gguf_affine_repack_f16(format: i32, source: *const c_void, payload: *mut c_void, scales: *mut c_void, offsets: *mut c_void, k: i32, n: i32, padded_n: i32, stream: usize) -> i32;
    pub fn mrs_gguf_affine_repack_bf16(format: i32, source: *const c_void, payload: *mut c_void, scales: *mut c_void, offsets: *mut c_void, k: i32, n: i32, padded_n: i32, stream: usize) -> i32;
    // ---- mrs_b200_seq.h
    pub fn mrs_seq_embed_streams(table: *const c_void, dtype: i32, ids: *const i32, streams: *mut f32, n_tok: i32, n_streams: i32, width: i32, stream: i64) -> i32;
    pub fn mrs_seq_streams_read_norm(streams: *const f32, w_in: *const f32, norm_w: *const f32, eps: f32, unit_offset: f32, rows: *const i32, out: *mut c_void, dtype: i32, n_rows: i32, n_streams: i32, width: i32, stream: i64) -> i32;
    pub fn mrs_seq_streams_write(streams: *mut f32, w_mix: *const f32, w_out: *const f32, y: *const c_void, dtype: i32, n_tok: i32, n_streams: i32, width: i32, next_in: *const f32, next_norm_w: *const f32, eps: f32, unit_offset: f32, next_out: *mut c_void, stream: i64) -> i32;
    pub fn mrs_seq_tanh_norm_rows(x: *const f32, rows: *const i32, alpha: *const f32, weight: *const f32, bias: *const f32, out: *mut c_void, dtype: i32, n_rows: i32, width: i32, stream: i64) -> i32;
    pub fn mrs_seq_residual_tanh_norm(x: *mut f32, y: *const c_void, dtype: i32, post_alpha: *const f32, post_weight: *const f32, post_bias: *const f32, extra: *const f32, next_alpha: *const f32, next_weight: *const f32, next_bias: *const f32, next_out: *mut c_void, n_tok: i32, width: i32, stream: i64) -> i32;
    pub fn mrs_seq_embed_scaled(table: *const c_void, dtype: i32, ids: *const i32, scale: f32, out: *mut f32, n_tok: i32, width: i32, stream: i64) -> i32;
    pub fn mrs_seq_embed_pair(table: *const c_void, pairs: *const c_void, dtype: i32, ids: *const i32, scale: f32, buckets: i64, mul_prev: i64, mul_cur: i64, prev_state: *mut i32, cu_tok: *const i32, past: *const i32, slot: *const i32, seq_of_tok: *const i32, out: *mut f32, n_tok: i32, width: i32, stream: i64) -> i32;
    pub fn mrs_seq_rms_residual(args: *const c_void, stream: i64) -> i32;
    pub fn mrs_seq_gated_lookup(gate: *const c_void, table: *const c_void, table_ld: i64, ids: *const i32, dtype: i32, act: i32, dim: i32, n_tok: i32, out: *mut c_void, stream: i64) -> i32;
    pub fn mrs_seq_gated_lookup_small(x: *const c_void, w: *const c_void, table: *const c_void, table_ld: i64, ids: *const i32, dtype: i32, act: i32, width: i32, dim: i32, n_tok: i32, out: *mut c_void, stream: i64) -> i32;
    pub fn mrs_seq_activate_cols(x: *mut c_void, ld: i64, dtype: i32, n_tok: i32, cols: i32, act: i32, stream: i64) -> i32;
    pub fn mrs_seq_glu_split(x: *const c_void, out: *mut c_void, dtype: i32, n_tok: i32, half: i32, act: i32, stream: i64) -> i32;
    pub fn mrs_seq_glu_join(x: *const c_void, out: *mut c_void, dtype: i32, n_tok: i32, half: i32, rule: *const c_void, stream: i64) -> i32;
    pub fn mrs_seq_bounded_gate(raw: *const c_void, raw_ld: i64, dtype: i32, bias: *const f32, lower: *const f32, n_tok: i32, cols: i32, gate: *mut f32, stream: i64) -> i32;
    pub fn mrs_seq_power_gate(raw: *const c_void, raw_ld: i64, dtype: i32, bias: *const f32, power: f32, n_tok: i32, cols: i32, gate: *mut f32, stream: i64) -> i32;
    pub fn mrs_seq_soft_cap(x: *const c_void, dtype: i32, scale: f32, cap: f32, n: i64, out: *mut f32, stream: i64) -> i32;
    pub fn mrs_seq_gated_group_norm(x: *const f32, gate: *const c_void, gate_ld: i64, weight: *const f32, out: *mut c_void, out_ld: i64, out_scale: f32, dtype: i32, n_tok: i32, cols: i32, groups: i32, eps: f32, gate_act: i32, gate_first: i32, stream: i64) -> i32;
    pub fn mrs_seq_causal_conv(in: *const c_void, in_ld: i64, col0: i32, dtype: i32, taps: *const f32, bias: *const f32, channels: i32, n_taps: i32, act: i32, conv_state: *mut f32, cu_tok: *const i32, past: *const i32, slot: *const i32, seq_of_tok: *const i32, n_seq: i32, n_tok: i32, out: *mut c_void, stream: i64) -> i32;
    pub fn mrs_seq_ssm_steps(in: *const c_void, in_ld: i64, col0: i32, dtype: i32, bias: *const f32, a_log: *const f32, heads: i32, n_tok: i32, step: *mut f32, decay: *mut f32, stream: i64) -> i32;
    pub fn mrs_seq_linear_scan(args: *const c_void, stream: i64) -> i32;
    pub fn mrs_seq_mlstm_gates(raw_in: *const f32, raw_forget: *const f32, raw_ld: i64, cap: f32, heads: i32, m_state: *mut f32, cu_tok: *const i32, past: *const i32, slot: *const i32, n_seq: i32, n_tok: i32, keep: *mut f32, take: *mut f32, m_tok: *mut f32, stream: i64) -> i32;
    pub fn mrs_seq_append_ones(v: *const c_void, v_ld: i64, dtype: i32, heads: i32, dv: i32, dvp: i32, n_tok: i32, vaug: *mut c_void, stream: i64) -> i32;
    pub fn mrs_seq_mlstm_out_norm(o: *const f32, dvp: i32, m_tok: *const f32, q_scale: f32, gate: *const c_void, gate_ld: i64, weight: *const f32, eps: f32, heads: i32, dv: i32, out: *mut c_void, out_ld: i64, dtype: i32, n_tok: i32, stream: i64) -> i32;
    pub fn mrs_seq_qk_norm_store(q: *mut c_void, q_ld: i64, k: *mut c_void, k_ld: i64, v: *const c_void, v_ld: i64, dtype: i32, q_norm_w: *const f32, k_norm_w: *const f32, eps: f32, heads: i32, kv_heads: i32, dk: i32, dv: i32, k_cache: *mut c_void, v_cache: *mut c_void, slot_of_tok: *const i64, n_tok: i32, stream: i64) -> i32;
    pub fn mrs_seq_window_attention(q: *const c_void, q_ld: i64, k_cache: *const c_void, v_cache: *const c_void, dtype: i32, heads: i32, kv_heads: i32, dk: i32, dv: i32, scale: f32, window: i32, pages: *const i32, pages_ld: i32, page_size: i32, seq_of_tok: *const i32, pos_of_tok: *const i32, tok_index: *const i32, n_tok: i32, out: *mut c_void, out_ld: i64, out_scale: f32, stream: i64) -> i32;
    pub fn mrs_seq_attention_prepare(args: *const c_void, stream: i64) -> i32;
    pub fn mrs_seq_rotation_table(pos_of_tok: *const i32, freq: *const f64, n_tok: i32, half: i32, mag: f32, cos_sin: *mut f32, stream: i64) -> i32;
    pub fn mrs_seq_paged_attention(args: *const c_void, stream: i64) -> i32;
    pub fn mrs_seq_pool_blocks(k_cache: *mut c_void, v_cache: *mut c_void, dtype: i32, k_row: i64, v_row: i64, k_cols: i32, v_cols: i32, pool: i32, pool_base: i64, pages: *const i32, pages_ld: i32, page_size: i32, seq_of_tok: *const i32, pos_of_tok: *const i32, n_tok: i32, stream: i64) -> i32;
    pub fn mrs_seq_mix_heads(a: *const f32, mix: *const f32, gate: *const c_void, gate_ld: i64, gate_act: i32, out: *mut c_void, out_ld: i64, dtype: i32, heads: i32, kv_heads: i32, dv: i32, n_tok: i32, stream: i64) -> i32;
    pub fn mrs_seq_gate_cols(x: *mut c_void, x_ld: i64, gate: *const c_void, gate_ld: i64, dtype: i32, cols: i32, group: i32, act: i32, n_tok: i32, stream: i64) -> i32;
    pub fn mrs_seq_prompt_attention(q: *const c_void, q_ld: i64, k_cache: *const c_void, v_cache: *const c_void, out: *mut c_void, out_ld: i64, portions: *const i32, n_portions: i32, longest: i32, pages: *const i32, pages_ld: i32, page_size: i32, heads: i32, kv_heads: i32, d: i32, scale: f32, window: i32, keep_first: i32, sink: *const f32, stream: i64) -> i32;
    pub fn mrs_seq_prompt_attention_pooled(q: *const c_void, q_ld: i64, k_cache: *const c_void, v_cache: *const c_void, out: *mut c_void, out_ld: i64, portions: *const i32, n_portions: i32, longest: i32, pages: *const i32, pages_ld: i32, page_size: i32, heads: i32, kv_heads: i32, d: i32, scale: f32, window: i32, keep_first: i32, sink: *const f32, pool: i32, pool_base: i64, every_value_head: i32, stream: i64) -> i32;
    pub fn mrs_seq_prompt_attention_general(args: *const c_void, stream: i64) -> i32;
    pub fn mrs_seq_prompt_attention_tc(args: *const c_void, stream: i64) -> i32;
    pub fn mrs_seq_prompt_attention_tc_fits(dn: i32, dr: i32, dv: i32) -> i32;
    pub fn mrs_seq_prompt_attention_tc_timeouts() -> i32;
    pub fn mrs_seq_gather_rows(cache: *const c_void, cache_row_bytes: i64, row_bytes: i32, runs: *const i32, n_runs: i32, longest: i32, pages: *const i32, pages_ld: i32, page_size: i32, out: *mut c_void, out_row_bytes: i64, stream: i64) -> i32;
    pub fn mrs_seq_latent_prepare(args: *const c_void, stream: i64) -> i32;
    pub fn mrs_seq_rotate_pairs(in: *const c_void, in_ld: i64, in_head: i64, out: *mut c_void, out_ld: i64, out_head: i64, dtype: i32, heads: i32, dims: i32, rot_dims: i32, cos_sin: *const f32, n_tok: i32, stream: i64) -> i32;
    pub fn mrs_seq_rotate_heads(in: *const c_void, in_ld: i64, in_head: i64, out: *mut c_void, out_ld: i64, out_head: i64, dtype: i32, heads: i32, dims: i32, rot_dims: i32, pairing: i32, cos_sin: *const f32, n_tok: i32, stream: i64) -> i32;
    pub fn mrs_seq_latent_attention_fits(kv_rank: i32, rot_dim: i32) -> i32;
    pub fn mrs_seq_latent_attention(q: *const c_void, q_ld: i64, cache: *const c_void, cache_row: i64, out: *mut c_void, out_ld: i64, portions: *const i32, cu_tok: *const i32, past: *const i32, n_portions: i32, longest: i32, pages: *const i32, pages_ld: i32, page_size: i32, heads: i32, kv_rank: i32, rot_dim: i32, scale: f32, window: i32, stream: i64) -> i32;
    pub fn mrs_seq_latent_attention_general(args: *const c_void, stream: i64) -> i32;
    pub fn mrs_seq_latent_attention_plan(n_portions: i32, longest: i32, heads: i32, kv_rank: i32, max_keys: i32, scratch_floats: *mut i64) -> i32;
    pub fn mrs_seq_scale_rows(x: *mut c_void, ld: i64, dtype: i32, rows: i32, cols: i32, scale: f32, stream: i64) -> i32;
    pub fn mrs_seq_moe_route(logits: *const f32, correction: *const f32, n_tok: i32, n_experts: i32, n_groups: i32, keep_groups: i32, top: i32, renorm: i32, experts: *mut i32, weights: *mut f32, stream: i64) -> i32;
    pub fn mrs_seq_moe_route_scored(logits: *const f32, correction: *const f32, n_tok: i32, n_experts: i32, n_groups: i32, keep_groups: i32, top: i32, renorm: i32, score_fn: i32, group_top: i32, weight_scale: f32, experts: *mut i32, weights: *mut f32, stream: i64) -> i32;
    pub fn mrs_seq_moe_route_general(args: *const c_void, stream: i64) -> i32;
    pub fn mrs_seq_moe_router(x: *const c_void, dtype: i32, w: *const f32, width: i32, args: *const c_void, stream: i64) -> i32;
    pub fn mrs_seq_moe_router_fits(width: i32, n_experts: i32, n_tok: i32) -> i32;
    pub fn mrs_seq_router_logits(x: *const c_void, dtype: i32, w: *const f32, width: i32, n_experts: i32, n_tok: i32, logits: *mut f32, stream: i64) -> i32;
    pub fn mrs_seq_moe_gate_up(x: *const c_void, gate_up: *const c_void, dtype: i32, experts: *const i32, n_tok: i32, top: i32, width: i32, ff: i32, act: i32, hidden: *mut c_void, stream: i64) -> i32;
    pub fn mrs_seq_moe_down(hidden: *const c_void, down: *const c_void, dtype: i32, experts: *const i32, weights: *const f32, n_tok: i32, top: i32, width: i32, ff: i32, out: *mut c_void, stream: i64) -> i32;
    pub fn mrs_seq_moe_gate_up_rule(x: *const c_void, gate_up: *const c_void, dtype: i32, experts: *const i32, n_tok: i32, top: i32, width: i32, ff: i32, rule: *const c_void, hidden: *mut c_void, stream: i64) -> i32;
    pub fn mrs_seq_moe_small(args: *const c_void, stream: i64) -> i32;
    pub fn mrs_seq_moe_grouped(args: *const c_void, stream: i64) -> i32;
    pub fn mrs_seq_moe_grouped_fits(dtype: i32, width: i32, ff: i32) -> i32;
    pub fn mrs_seq_moe_route_top_softmax(logits: *const f32, n_tok: i32, n_experts: i32, top: i32, experts: *mut i32, weights: *mut f32, stream: i64) -> i32;
    pub fn mrs_seq_moe_up(x: *const c_void, up: *const c_void, dtype: i32, experts: *const i32, n_tok: i32, top: i32, width: i32, ff: i32, act: i32, hidden: *mut c_void, stream: i64) -> i32;
    pub fn mrs_seq_moe_sort(experts: *const i32, n_pairs: i32, n_experts: i32, counts: *mut i32, order: *mut i32, stream: i64) -> i32;
    pub fn mrs_seq_moe_gather(x: *const c_void, dtype: i32, order: *const i32, n_pairs: i32, top: i32, width: i32, sorted: *mut c_void, stream: i64) -> i32;
    pub fn mrs_seq_moe_gemm(sorted: *const c_void, weights: *const c_void, counts: *const i32, n_rows: i32, n_ffn: i32, n: i32, k: i32, gated: i32, rule: *const c_void, out: *mut c_void, stream: i64) -> i32;
    pub fn mrs_seq_moe_gemm_fits(dtype: i32, n: i32, k: i32, n_ffn: i32) -> i32;
    pub fn mrs_seq_moe_products(sorted: *const c_void, up: *const c_void, down: *const c_void, counts: *const i32, n_rows: i32, n_ffn: i32, width: i32, ff: i32, gated: i32, rule: *const c_void, hidden: *mut c_void, out: *mut c_void, stream: i64) -> i32;
    pub fn mrs_seq_moe_gemm_timeouts() -> i32;
    pub fn mrs_seq_moe_combine(sorted_y: *const c_void, dtype: i32, order: *const i32, weights: *const f32, n_tok: i32, top: i32, width: i32, scratch_inverse: *mut i32, out: *mut c_void, stream: i64) -> i32;
    pub fn mrs_seq_moe_combine_some(sorted_y: *const c_void, dtype: i32, order: *const i32, weights: *const f32, experts: *const i32, x: *const c_void, n_ffn: i32, n_tok: i32, top: i32, width: i32, scratch_inverse: *mut i32, out: *mut c_void, stream: i64) -> i32;
    pub fn mrs_seq_moe_place_fits(n_pairs: i32, n_experts: i32) -> i32;
    pub fn mrs_seq_moe_place(experts: *const i32, n_pairs: i32, n_experts: i32, x: *const c_void, dtype: i32, top: i32, width: i32, counts: *mut i32, inverse: *mut i32, sorted: *mut c_void, stream: i64) -> i32;
    pub fn mrs_seq_moe_combine_at(sorted_y: *const c_void, dtype: i32, inverse: *const i32, weights: *const f32, experts: *const i32, x: *const c_void, n_ffn: i32, n_tok: i32, top: i32, width: i32, out: *mut c_void, stream: i64) -> i32;
    pub fn mrs_seq_moe_block(args: *const c_void, stream: i64) -> i32;
}
