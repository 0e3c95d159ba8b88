/*
 * mrs_oracle.h — CPU ORACLE (TEST INFRASTRUCTURE, NOT PRODUCT).
 *
 * A plain-C restatement of the arithmetic of mistral.rs's quantized-linear + paged-KV-attention
 * hot path.  Only tests/, __graft_entry__.smoke() and bench.py's cpu_baseline / --impl reference
 * legs may load this library, and only as the checker / the CPU timing baseline.  The product
 * (mistral.rs_b200/) never links, imports or calls anything in oracle/.
 *
 * Pinning status: the block decoders are pinned against gguf-py 0.19.0 `gguf.quants.dequantize`
 * (tests/golden/gguf_dequant_*.npz, generated by tests/golden/make_gguf_golden.py) and the
 * Q8_1 arithmetic, cache scatter, RoPE, GLU and RMSNorm functions are pinned against the
 * reference's own CUDA kernels (oracle/_ref, built from its tree by oracle/build_ref.sh) through
 * the committed fixture tests/golden/ref_golden.npz produced by tests/golden/make_ref_golden.py.
 * The candle CPU path (Q8_K activations) is NOT in the reference's tree (git dependency
 * huggingface/candle@35d7ae7c, v0.11.0): mrs_qmatmul_cpu restates the published
 * llama.cpp/candle k-quants algorithm and is "parity unpinned" against candle itself.
 */
#ifndef MRS_ORACLE_H
#define MRS_ORACLE_H
#include <stddef.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

/* ggml dtype codes (the reference's GgmlDType numbering, candle quantized/mod.rs) */
enum {
  MRS_Q4_0 = 2, MRS_Q4_1 = 3, MRS_Q5_0 = 6, MRS_Q5_1 = 7, MRS_Q8_0 = 8, MRS_Q8_1 = 9,
  MRS_Q2_K = 10, MRS_Q3_K = 11, MRS_Q4_K = 12, MRS_Q5_K = 13, MRS_Q6_K = 14, MRS_Q8_K = 15
};
/* activation dtype codes used across the reference's C ABI: 0=f16 1=bf16 2=f32 */
enum { MRS_F16 = 0, MRS_BF16 = 1, MRS_F32 = 2 };

int    mrs_block_elems(int ggml_type);   /* 32 or 256, 0 if unsupported */
int    mrs_block_bytes(int ggml_type);   /* bytes per block */

/* scalar conversions (round-to-nearest-even) */
float    mrs_f16_to_f32(uint16_t h);
uint16_t mrs_f32_to_f16(float f);
float    mrs_bf16_to_f32(uint16_t h);
uint16_t mrs_f32_to_bf16(float f);
/* round f32 through dtype (0 f16 / 1 bf16 / 2 f32) */
float    mrs_round_dtype(float f, int dtype);

/* Exact block decoders: out[n] = deq(blocks), n multiple of the block size.
 * Layouts: mistralrs-quant/kernels/mmvq_gguf/mmvq_gguf.cu:134-225. */
int mrs_dequantize(int ggml_type, const void *blocks, float *out, int64_t n);

/* Q8_1 activation quantiser — mmvq_gguf.cu:1220-1251 (warp amax / butterfly sum,
 * d = amax/127, q = roundf(x/d), ds = half2(d, sum)); rows padded with zeros to kx_padded.
 * y: block_q8_1[rows * kx_padded/32], 36 bytes each. */
void mrs_quantize_q8_1(const float *x, void *y, int kx, int kx_padded, int rows);

/* GEMV in the reference GPU decode numerics (Q8_1 activations, integer block dots,
 * scale products evaluated exactly in double): out[b*nrows + r].
 * vec_dot formulas: mmvq_gguf.cu:244-450, indexing :458-684. */
int mrs_mmvq_q8_1(int ggml_type, const void *w, const void *y_q8_1, double *out,
                  int ncols, int nrows, int stride_col_y_blocks, int batch);

/* EXACT: out = sum_k deq(w[r,k]) * x[b,k] in double */
int mrs_matmul_exact(int ggml_type, const void *w, const float *x, double *out,
                     int ncols, int nrows, int batch);

/* The reference's CPU path restated (candle QMatMul::forward: activations -> Q8_K for
 * k-quants / Q8_0 for 32-wide types, integer block dots, f32 accumulate), rows split over
 * `threads` pthreads.  Returns 0 on success. */
int mrs_qmatmul_cpu(int ggml_type, const void *w, const float *x, float *out,
                    int ncols, int nrows, int batch, int threads);

/* GLU activation (mmvq_gguf.cu:52-88 / ops.cu:806-847), act in GluActivationType 0..4 */
float mrs_glu_act(float x, int act);
/* fused_glu: out = dtype(act(a)) * b, product rounded in dtype (ops.cu:848-969) */
void mrs_fused_glu(const float *a, const float *b, float *out, int64_t n, int act, int dtype);

/* RMSNorm: out = dtype(x * rsqrt(mean(x^2)+eps) * w) (core layers.rs:403-413 -> candle rms_norm);
 * add variant: sum = dtype(x+res); normed from the rounded sum (core/src/cuda/sort.cu:403-428) */
void mrs_rms_norm(const float *x, const float *w, float *out, int rows, int cols, float eps, int dtype);
void mrs_add_rms_norm(const float *x, const float *res, const float *w, float *sum_out,
                      float *norm_out, int rows, int cols, float eps, int dtype);

/* RoPE in place, per-op rounding in dtype (quant/kernels/rotary/rotary.cu:10-100).
 * q: [tokens, q_stride], k: [tokens, k_stride]; cos/sin: [max_pos, rot_half]; positions may be
 * NULL (then row t of cos/sin is used). rot_half is the reference's `rot_dim` argument. */
void mrs_rotary(float *q, float *k, const float *cos, const float *sin, const uint32_t *positions,
                int is_neox, int head_size, int64_t tokens, int rot_half, int num_heads,
                int num_kv_heads, int64_t q_stride, int64_t k_stride, int dtype);

/* Llama-3 rope tables (core/src/layers.rs:1071-1160): cos/sin [max_pos, head_dim/2] f32 */
void mrs_llama3_rope_table(float *cos, float *sin, int max_pos, int head_dim, float theta,
                           int use_scaling, float factor, float low_freq_factor,
                           float high_freq_factor, int original_max_pos);

/* KV cache scatter. layout 0 = vLLM ([NB,KVH,D/x,BS,x] keys, [NB,KVH,D,BS] values;
 * reshape_and_cache_kernel.cu:32-87), layout 1 = FlashInfer HND ([NB,KVH,BS,D];
 * flashinfer_decode.cu:20-54).  Element type is 16-bit (raw copy). slot -1 = skip. */
void mrs_reshape_and_cache(const uint16_t *key, const uint16_t *value, uint16_t *key_cache,
                           uint16_t *value_cache, const int64_t *slot_mapping, int num_tokens,
                           int num_heads, int head_size, int block_size, int x, int key_stride,
                           int value_stride, int layout);

/* Decode attention over a paged cache, f32 maths, double accumulation.
 * (pagedattention.cuh:110-485 / flashinfer decode.cuh).  q: [S, q_stride] f32 (already
 * widened), caches 16-bit of `dtype`; block_tables [S, max_blocks]; out [S,H,D] f32. */
void mrs_paged_attention(const float *q, const uint16_t *key_cache, const uint16_t *value_cache,
                         const int32_t *block_tables, const int32_t *context_lens, float *out,
                         int num_seqs, int num_heads, int num_kv_heads, int head_size,
                         int block_size, int max_blocks, int q_stride, float scale,
                         float softcap, int layout, int x, int dtype);

#ifdef __cplusplus
}
#endif
#endif
