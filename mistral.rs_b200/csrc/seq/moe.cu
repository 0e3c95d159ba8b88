// moe.cu — mixture of experts: the routing rule (softmax or sigmoid scores, a choice bias that does not enter the weights,
// selection limited to the best groups of neighbouring experts, a group scored by its largest choice or by the sum of its
// few largest), the expert feed-forward for small batches as two weight-streaming kernels, and the sort / gather / combine
// steps around per-expert matrix products for large ones.  Experts from index n_ffn on are identities: they have no weights
// and hand their input back.
#include <limits.h>

#include "seq_common.cuh"

namespace seq {

constexpr int ROUTE_MAX_EXPERTS = 1024;

// The routing rule for one token by one warp: z are its logits; score and choice [n_experts] and gscore [n_groups] are shared memory
// of the warp; experts and weights are the token's `top` results.
__device__ __forceinline__ void route_token(const float *z, const mrs_seq_moe_route_args &a, float *score, float *choice, float *gscore, int lane,
                                            int32_t *experts, float *weights) {
  const int n_experts = a.n_experts, n_groups = a.n_groups, keep_groups = a.keep_groups, top = a.top, renorm = a.renorm, score_fn = a.score_fn;
  const int group_top = a.group_top;
  const float weight_scale = a.weight_scale, renorm_eps = a.renorm_eps, *correction = a.correction;
  float inv = 1.0f;
  if (score_fn == MRS_SEQ_SCORE_SIGMOID) {
    for (int e = lane; e < n_experts; e += 32) score[e] = sigmoid_f(z[e]);
  } else {
    float mx = -INFINITY;
    for (int e = lane; e < n_experts; e += 32) mx = fmaxf(mx, z[e]);
    mx = warp_max(mx);
    float sum = 0.0f;
    for (int e = lane; e < n_experts; e += 32) {
      const float p = expf(z[e] - mx);
      score[e] = p;
      sum += p;
    }
    sum = warp_sum(sum);
    inv = 1.0f / sum;
  }
  for (int e = lane; e < n_experts; e += 32) {
    const float s = score[e] * inv;
    score[e] = s;
    choice[e] = s + (correction ? correction[e] : 0.0f);
  }
  __syncwarp();
  const int per = n_experts / n_groups;
  if (keep_groups < n_groups) {
    for (int gi = lane; gi < n_groups; gi += 32) {
      float best = -INFINITY;
      if (group_top <= 1) {
        for (int e = gi * per; e < (gi + 1) * per; e++) best = fmaxf(best, choice[e]);
      } else {      // the sum of the group's group_top largest choices: take them one by one, below the last one taken
        float total = 0.0f, last = INFINITY;
        int last_e = -1;
        for (int r = 0; r < group_top && r < per; r++) {
          float bv = -INFINITY;
          int be = -1;
          for (int e = gi * per; e < (gi + 1) * per; e++) {
            const float v = choice[e];
            if ((v < last || (v == last && e > last_e)) && (be < 0 || v > bv)) { bv = v; be = e; }
          }
          if (be < 0) break;
          total += bv;
          last = bv;
          last_e = be;
        }
        best = total;
      }
      gscore[gi] = best;
    }
    __syncwarp();
    // take the keep_groups best groups one by one (ties: the lower index); a taken group is marked with +inf
    for (int r = 0; r < keep_groups; r++) {
      float bv = -INFINITY;
      int bi = 0x7fffffff;
      for (int gi = lane; gi < n_groups; gi += 32) {
        const float v = gscore[gi];
        if (v != INFINITY && (v > bv || (v == bv && gi < bi))) { bv = v; bi = gi; }
      }
      for (int m = 16; m > 0; m >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, m);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, m);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
      }
      if (lane == 0 && bi < n_groups) gscore[bi] = INFINITY;
      __syncwarp();
    }
    for (int e = lane; e < n_experts; e += 32)
      if (gscore[e / per] != INFINITY) choice[e] = -INFINITY;
    __syncwarp();
  }
  // (choice r waits in lane r: weights that went to memory and came back for the division made half of the kernel's time)
  float wsum = 0.0f, my_w = 0.0f;
  int my_e = 0;
  const bool held = top <= 32;
  for (int r = 0; r < top; r++) {
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    for (int e = lane; e < n_experts; e += 32) {
      const float v = choice[e];
      if (!(v != v) && (v > bv || (v == bv && e < bi)) && v != -INFINITY) { bv = v; bi = e; }
    }
    for (int m = 16; m > 0; m >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, m);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, m);
      if (oi != 0x7fffffff && (bi == 0x7fffffff || ov > bv || (ov == bv && oi < bi))) { bv = ov; bi = oi; }
    }
    if (bi == 0x7fffffff) bi = 0;   // fewer eligible experts than `top`: weight 0
    const float wv = bv == -INFINITY ? 0.0f : score[bi];
    if (lane == r) { my_e = bi; my_w = wv; }
    if (lane == 0) {
      if (!held) { experts[r] = bi; weights[r] = wv; }
      if (bv != -INFINITY) choice[bi] = -INFINITY;
    }
    wsum += wv;
    __syncwarp();
  }
  if (held) {
    if (lane < top) {
      if (renorm && wsum + renorm_eps > 0.0f) my_w /= wsum + renorm_eps;
      if (weight_scale != 1.0f) my_w *= weight_scale;
      experts[lane] = my_e;
      weights[lane] = my_w;
    }
    return;
  }
  if (renorm && lane == 0 && wsum + renorm_eps > 0.0f)
    for (int r = 0; r < top; r++) weights[r] /= wsum + renorm_eps;
  if (weight_scale != 1.0f && lane == 0)
    for (int r = 0; r < top; r++) weights[r] *= weight_scale;
}

// one warp per token; scores and choices of all experts in shared memory
__global__ void moe_route_kernel(const mrs_seq_moe_route_args a) {
  extern __shared__ float sm[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int t = blockIdx.x * nw + wib;
  wait_for_previous();
  let_next_start();
  if (t >= a.n_tok) return;
  float *score = sm + (size_t)wib * (2 * a.n_experts + a.n_groups), *choice = score + a.n_experts, *gscore = choice + a.n_experts;
  route_token(a.logits + (int64_t)t * (a.logits_ld > 0 ? a.logits_ld : a.n_experts), a, score, choice, gscore, lane, a.experts + (int64_t)t * a.top, a.weights + (int64_t)t * a.top);
}

// The router's product for few tokens, in f32: one CTA per (output, token), so that a decode step's router rows come through many SMs
template <typename T, int VEC>
__global__ void __launch_bounds__(128) router_logits_kernel(const T *__restrict__ x, const float *__restrict__ w, int width, int n_experts, float *__restrict__ logits) {
  __shared__ float red[33];
  let_next_start();
  const float *wr = w + (int64_t)blockIdx.x * width;
  const T *xr = x + (int64_t)blockIdx.y * width;
  float s = 0.0f;
#pragma unroll 4
  for (int c = threadIdx.x * VEC; c < width; c += 128 * VEC) {
    if (VEC == 4) {
      const float4 a = *(const float4 *)(wr + c), b = load4<T>(xr + c);
      s = fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, s))));
    } else {
      s = fmaf(wr[c], to_f32<T>(xr[c]), s);
    }
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) logits[(int64_t)blockIdx.y * n_experts + blockIdx.x] = s;
}

// The two steps above in one launch for few tokens and few experts: one CTA per token, 128 threads per product, each product summed in
// the order of router_logits_kernel (the same bits), then the routing rule by the first warp.  Bound by latency: the router's rows come
// to every CTA from L2 at one SM's rate, and a group of 128 threads takes its products one after the other, so their size and number draw
// the line.  us of two launches / one, 1, 8 and 32 tokens: 8 experts of 1024 columns 5.5 / 4.4, 5.8 / 4.5, 5.9 / 4.5; 16 of 2048 5.6 / 5.2, 5.8 /
// 5.4, 6.1 / 5.5; beyond it 16 of 4096 5.8 / 6.2, 6.2 / 6.3, 6.6 / 6.5, 32 of 1024 5.3 / 6.3, 5.7 / 6.4, 6.1 / 6.6.
constexpr int ROUTE_FUSED_GROUPS = 8, ROUTE_FUSED_EXPERTS = 16, ROUTE_FUSED_TOKENS = 64, ROUTE_FUSED_WEIGHTS = 32768;
template <typename T, int VEC>
__global__ void __launch_bounds__(128 * ROUTE_FUSED_GROUPS) router_route_kernel(const T *__restrict__ x, const float *__restrict__ w, int width,
                                                                                const mrs_seq_moe_route_args a) {
  constexpr int E = ROUTE_FUSED_EXPERTS;
  __shared__ float part[E][4], z[E], score[E], choice[E], gscore[E];
  const int t = blockIdx.x, group = threadIdx.x >> 7, i = threadIdx.x & 127, lane = threadIdx.x & 31, warp = i >> 5;
  const T *xr = x + (int64_t)t * width;
  wait_for_previous();
  let_next_start();
  for (int e = group; e < a.n_experts; e += ROUTE_FUSED_GROUPS) {
    const float *wr = w + (int64_t)e * width;
    float s = 0.0f;
#pragma unroll 4
    for (int c = i * VEC; c < width; c += 128 * VEC) {
      if (VEC == 4) {
        const float4 p = *(const float4 *)(wr + c), q = load4<T>(xr + c);
        s = fmaf(p.x, q.x, fmaf(p.y, q.y, fmaf(p.z, q.z, fmaf(p.w, q.w, s))));
      } else {
        s = fmaf(wr[c], to_f32<T>(xr[c]), s);
      }
    }
    s = warp_sum(s);
    if (lane == 0) part[e][warp] = s;
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  for (int e = lane; e < a.n_experts; e += 32) z[e] = (part[e][0] + part[e][2]) + (part[e][1] + part[e][3]);
  __syncwarp();
  route_token(z, a, score, choice, gscore, lane, a.experts + (int64_t)t * a.top, a.weights + (int64_t)t * a.top);
}

// hidden[t][k][r] = act(gate_up[e][r] . x_t) * (gate_up[e][ff + r] . x_t): one warp per output element;
// blockIdx.y is the (token, k) pair, pairs laid out [token][k]
template <typename T>
__global__ void __launch_bounds__(256) moe_gate_up_kernel(const T *__restrict__ x, const T *__restrict__ gate_up,
                                                          const int32_t *__restrict__ experts, int top, int width, int ff,
                                                          const mrs_seq_glu_rule rule, int n_ffn, T *__restrict__ hidden) {
  extern __shared__ __align__(16) float xs[];   // [width]
  const int pair = blockIdx.y, tok = pair / top;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int e = experts[pair];
  if (e >= n_ffn) return;
  for (int c = threadIdx.x; c < width; c += blockDim.x) xs[c] = to_f32<T>(x[(int64_t)tok * width + c]);
  __syncthreads();
  const T *w = gate_up + (int64_t)e * 2 * ff * width;
  const bool vec = width % Vec16<T>::N == 0 && ((uintptr_t)gate_up % 16) == 0;
  for (int r = blockIdx.x * nw + wib; r < ff; r += gridDim.x * nw) {
    const float ag = warp_row_dot<T>(w + (int64_t)r * width, xs, width, lane, vec);
    const float au = warp_row_dot<T>(w + (int64_t)(ff + r) * width, xs, width, lane, vec);
    if (lane == 0) {
      // the products leave the "matrix product" in the activation type, as the large-batch path's do
      const float gt = to_f32<T>(from_f32<T>(ag)), up = to_f32<T>(from_f32<T>(au));
      hidden[(int64_t)pair * ff + r] = from_f32<T>(glu_join(gt, up, rule));
    }
  }
}

// the plain rule, one warp per token: the `top` largest logits (ties: the lower index), softmax over those alone
__global__ void moe_route_top_softmax_kernel(const float *__restrict__ logits, int n_tok, int n_experts, int top,
                                             int32_t *__restrict__ experts, float *__restrict__ weights) {
  extern __shared__ float sm[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int t = blockIdx.x * nw + wib;
  wait_for_previous();
  let_next_start();
  if (t >= n_tok) return;
  float *z = sm + (size_t)wib * n_experts;
  for (int e = lane; e < n_experts; e += 32) z[e] = logits[(int64_t)t * n_experts + e];
  __syncwarp();
  float first = 0.0f, sum = 0.0f;
  for (int r = 0; r < top; r++) {
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    for (int e = lane; e < n_experts; e += 32) {
      const float v = z[e];
      if (v == v && (bi == 0x7fffffff ? v >= bv : v > bv)) { bv = v; bi = e; }   // NaN never wins; a taken expert holds NaN
    }
    for (int m = 16; m > 0; m >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, m);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, m);
      if (oi != 0x7fffffff && (bi == 0x7fffffff || ov > bv || (ov == bv && oi < bi))) { bv = ov; bi = oi; }
    }
    if (bi == 0x7fffffff) { bi = 0; bv = -INFINITY; }
    if (r == 0) first = bv;                       // the largest logit: the softmax's reference point
    const float p = expf(bv - first);
    sum += p;
    if (lane == 0) {
      experts[(int64_t)t * top + r] = bi;
      weights[(int64_t)t * top + r] = p;
      z[bi] = __int_as_float(0x7fc00000);
    }
    __syncwarp();
  }
  if (lane == 0)
    for (int r = 0; r < top; r++) weights[(int64_t)t * top + r] /= sum;
}

// hidden[t][k][r] = act(up[e][r] . x_t): experts without a gate; the layout of moe_gate_up_kernel
template <typename T>
__global__ void __launch_bounds__(256) moe_up_kernel(const T *__restrict__ x, const T *__restrict__ up, const int32_t *__restrict__ experts,
                                                     int top, int width, int ff, int act, T *__restrict__ hidden) {
  extern __shared__ __align__(16) float xs[];   // [width]
  const int pair = blockIdx.y, tok = pair / top;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int e = experts[pair];
  for (int c = threadIdx.x; c < width; c += blockDim.x) xs[c] = to_f32<T>(x[(int64_t)tok * width + c]);
  __syncthreads();
  const T *w = up + (int64_t)e * ff * width;
  const bool vec = width % Vec16<T>::N == 0 && ((uintptr_t)up % 16) == 0;
  for (int r = blockIdx.x * nw + wib; r < ff; r += gridDim.x * nw) {
    const float a = warp_row_dot<T>(w + (int64_t)r * width, xs, width, lane, vec);
    if (lane == 0) hidden[(int64_t)pair * ff + r] = from_f32<T>(apply_act(to_f32<T>(from_f32<T>(a)), act));
  }
}

// out[t][r] = sum_k weights[t][k] * (down[e_k][r] . hidden[t][k]), an identity expert's part being x[t][r]
template <typename T>
__global__ void __launch_bounds__(256) moe_down_kernel(const T *__restrict__ hidden, const T *__restrict__ down,
                                                       const int32_t *__restrict__ experts, const float *__restrict__ weights, int top,
                                                       int width, int ff, const T *__restrict__ x, int n_ffn, T *__restrict__ out) {
  extern __shared__ __align__(16) float hs[];   // [top][ff]
  const int t = blockIdx.y, lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int k = 0; k < top; k++) {
    if (experts[(int64_t)t * top + k] >= n_ffn) continue;
    for (int c = threadIdx.x; c < ff; c += blockDim.x) hs[k * ff + c] = to_f32<T>(hidden[((int64_t)t * top + k) * ff + c]);
  }
  __syncthreads();
  const bool vec = ff % Vec16<T>::N == 0 && ((uintptr_t)down % 16) == 0;
  for (int r = blockIdx.x * nw + wib; r < width; r += gridDim.x * nw) {
    float acc = 0.0f;
    for (int k = 0; k < top; k++) {
      const int e = experts[(int64_t)t * top + k];
      float a;
      if (e >= n_ffn) a = to_f32<T>(x[(int64_t)t * width + r]);
      else a = to_f32<T>(from_f32<T>(warp_row_dot<T>(down + ((int64_t)e * width + r) * ff, hs + k * ff, ff, lane, vec)));
      acc = fmaf(weights[(int64_t)t * top + k], a, acc);
    }
    if (lane == 0) out[(int64_t)t * width + r] = from_f32<T>(acc);
  }
}

// ---- few tokens per expert: every weight read once per step ---------------------------------------------------------
// N neighbouring elements of a 16-byte group as f32
template <typename T> __device__ __forceinline__ void unpack16(const uint4 raw, float *v);
template <> __device__ __forceinline__ void unpack16<float>(const uint4 raw, float *v) {
  v[0] = __uint_as_float(raw.x); v[1] = __uint_as_float(raw.y); v[2] = __uint_as_float(raw.z); v[3] = __uint_as_float(raw.w);
}
template <> __device__ __forceinline__ void unpack16<__nv_bfloat16>(const uint4 raw, float *v) {
  const uint32_t u[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    v[2 * i] = __uint_as_float(u[i] << 16);
    v[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
  }
}

// dots of four weight rows with P rows held in shared memory (row stride n elements of T); n a multiple of the 16-byte group
template <typename T, int P>
__device__ __forceinline__ void four_row_dots(const T *const *w, const T *xs, int n, int lane, float (*acc)[P]) {
  constexpr int N = Vec16<T>::N;
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int p = 0; p < P; p++) acc[r][p] = 0.0f;
#pragma unroll 2
  for (int c = lane * N; c < n; c += 32 * N) {
    uint4 raw[4];
#pragma unroll
    for (int r = 0; r < 4; r++) raw[r] = __ldcs((const uint4 *)(w[r] + c));
    float wv[4][N];
#pragma unroll
    for (int r = 0; r < 4; r++) unpack16<T>(raw[r], wv[r]);
#pragma unroll
    for (int p = 0; p < P; p++) {
      float xv[N];
      unpack16<T>(*(const uint4 *)(xs + (size_t)p * n + c), xv);
#pragma unroll
      for (int i = 0; i < N; i++)
#pragma unroll
        for (int r = 0; r < 4; r++) acc[r][p] = fmaf(wv[r][i], xv[i], acc[r][p]);
    }
  }
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int p = 0; p < P; p++) acc[r][p] = warp_sum(acc[r][p]);
}

struct GroupedParams {
  const void *in, *weights;          // rows [.][n] per token (UP) or per pair; weights [n_ffn][rows][n]
  const int32_t *counts, *order;     // per expert; pairs sorted by expert
  int top, n, rows, ff;              // n: length of a dot; rows: weight rows of an expert; ff: hidden size
  mrs_seq_glu_rule rule;
  void *out;                         // [pairs][ff] (UP) or [pairs][rows]
};

// One CTA = a block of an expert's output rows, for all its pairs (P at a time).  UP: out[pair] = join / act of the first product,
// GATED with rows r and ff + r side by side; else the plain product.  Four weight rows per warp and step.
template <typename T, bool UP, bool GATED, int P>
__device__ __forceinline__ void grouped_chunk(const GroupedParams &a, const T *w, const int32_t *pairs, int n_pairs, T *xs, int out_rows) {
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int groups = a.n / Vec16<T>::N;
  __syncthreads();                   // the rows of the previous chunk are no longer read
  for (int i = threadIdx.x; i < P * groups; i += blockDim.x) {
    const int p = i / groups, c = i % groups;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (p < n_pairs) v = ((const uint4 *)((const T *)a.in + (int64_t)(UP ? pairs[p] / a.top : pairs[p]) * a.n))[c];
    ((uint4 *)xs)[i] = v;
  }
  __syncthreads();
  constexpr int STEP = GATED ? 2 : 4;                     // output rows per warp and step
  for (int r0 = (blockIdx.x * nw + wib) * STEP; r0 < out_rows; r0 += gridDim.x * nw * STEP) {
    const T *row[4];
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const int o = min(r0 + (GATED ? r >> 1 : r), out_rows - 1);
      row[r] = w + (int64_t)(GATED && (r & 1) ? a.ff + o : o) * a.n;
    }
    float acc[4][P];
    four_row_dots<T, P>(row, xs, a.n, lane, acc);
    if (lane == 0) {
#pragma unroll
      for (int o = 0; o < STEP; o++) {
        if (r0 + o >= out_rows) break;
#pragma unroll
        for (int p = 0; p < P; p++) {
          if (p >= n_pairs) break;
          // the products leave the "matrix product" in the activation type, as the large-batch path's do
          const float v0 = to_f32<T>(from_f32<T>(acc[GATED ? 2 * o : o][p]));
          float v = v0;
          if (UP) v = GATED ? glu_join(v0, to_f32<T>(from_f32<T>(acc[(2 * o + 1) & 3][p])), a.rule) : apply_act(v0, a.rule.act);
          ((T *)a.out)[(int64_t)pairs[p] * out_rows + r0 + o] = from_f32<T>(v);
        }
      }
    }
  }
}

template <typename T, bool UP, bool GATED>
__global__ void __launch_bounds__(256) moe_grouped_kernel(const GroupedParams a, int per_chunk) {
  extern __shared__ __align__(16) uint8_t raw_sm[];
  const int e = blockIdx.y, n = a.counts[e];
  if (n == 0) return;
  __shared__ int first;
  if (threadIdx.x < 32) {                                  // where the expert's pairs start in the sorted list
    int s = 0;
    for (int i = threadIdx.x; i < e; i += 32) s += a.counts[i];
    for (int m = 16; m > 0; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    if (threadIdx.x == 0) first = s;
  }
  __syncthreads();
  const T *w = (const T *)a.weights + (int64_t)e * a.rows * a.n;
  const int out_rows = UP ? a.ff : a.rows;
  for (int p0 = 0; p0 < n; p0 += per_chunk) {
    const int left = min(per_chunk, n - p0);
    const int32_t *pairs = a.order + first + p0;
    if (left <= 2) grouped_chunk<T, UP, GATED, 2>(a, w, pairs, left, (T *)raw_sm, out_rows);
    else if (left <= 4) grouped_chunk<T, UP, GATED, 4>(a, w, pairs, left, (T *)raw_sm, out_rows);
    else grouped_chunk<T, UP, GATED, 8>(a, w, pairs, left, (T *)raw_sm, out_rows);
  }
}

// ---- sorted path --------------------------------------------------------------------------------------------------
// single CTA: counts per expert, then every (token, k) pair takes the next free row of its expert's range
__global__ void moe_sort_kernel(const int32_t *__restrict__ experts, int n_pairs, int n_experts, int32_t *__restrict__ counts,
                                int32_t *__restrict__ order) {
  extern __shared__ int32_t cnt[];   // [n_experts] counts, then [n_experts] running offsets
  int32_t *off = cnt + n_experts;
  for (int e = threadIdx.x; e < n_experts; e += blockDim.x) cnt[e] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < n_pairs; i += blockDim.x) atomicAdd(&cnt[experts[i]], 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    int run = 0;
    for (int e = 0; e < n_experts; e++) {
      off[e] = run;
      run += cnt[e];
      counts[e] = cnt[e];
    }
  }
  __syncthreads();
  // rows of one expert may land in any order: each row's product does not depend on its place
  for (int i = threadIdx.x; i < n_pairs; i += blockDim.x) order[atomicAdd(&off[experts[i]], 1)] = i;
}

// U: the unit of the copies, T itself or uint4 (rows in whole 16-byte groups; width then counts those)
template <typename U>
__global__ void moe_gather_kernel(const U *__restrict__ x, const int32_t *__restrict__ order, int top, int width, U *__restrict__ sorted) {
  const int i = blockIdx.x, t = order[i] / top;
  for (int c = threadIdx.x; c < width; c += blockDim.x) sorted[(int64_t)i * width + c] = x[(int64_t)t * width + c];
}

__global__ void moe_inverse_kernel(const int32_t *__restrict__ order, int n_pairs, int32_t *__restrict__ inverse) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_pairs) inverse[order[i]] = i;
}

// The three above for few pairs, in one launch: CTA i finds pair i's row (pairs of lower experts, and earlier ones of its own) by looking at
// all pairs, copies its token there, and counts the pairs of expert i.  Bound by the launch: 128 pairs of 2048 columns took 6.5 us in three
// launches (sort 1.9, gather 2.3, inverse 2.3) and as many calls from the host
// (32 tokens to 4 of 16 experts, the whole layer: 107.3 us so, 100.5 with the one).  Each CTA reads all pairs: MOE_PLACE_PAIRS is the line.
constexpr int MOE_PLACE_PAIRS = 2048;
template <typename U>
__global__ void __launch_bounds__(128) moe_place_kernel(const int32_t *__restrict__ experts, int n_pairs, int n_experts, const U *__restrict__ x, int top,
                                                        int width, int32_t *__restrict__ counts, int32_t *__restrict__ inverse, U *__restrict__ sorted) {
  __shared__ int32_t red[2][4];
  wait_for_previous();
  let_next_start();
  const int i = blockIdx.x, own = i < n_pairs ? experts[i] : 0;
  int before = 0, mine = 0;
  for (int j = threadIdx.x; j < n_pairs; j += 128) {
    const int e = experts[j];
    before += e < own || (e == own && j < i);
    mine += e == i;
  }
  before = __reduce_add_sync(0xffffffffu, before);
  mine = __reduce_add_sync(0xffffffffu, mine);
  if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = before; red[1][threadIdx.x >> 5] = mine; }
  __syncthreads();
  const int at = red[0][0] + red[0][1] + red[0][2] + red[0][3];
  if (threadIdx.x == 0) {
    if (i < n_experts) counts[i] = red[1][0] + red[1][1] + red[1][2] + red[1][3];
    if (i < n_pairs) inverse[i] = at;
  }
  if (i >= n_pairs) return;
  const U *from = x + (int64_t)(i / top) * width;
  for (int c = threadIdx.x; c < width; c += 128) sorted[(int64_t)at * width + c] = from[c];
}

// inverse NULL: rows of sorted_y are in the order of the pairs.  experts NULL: every pair has a row in sorted_y; else pairs of experts from n_ffn on take their token's row of x
template <typename T, int VEC>
__global__ void moe_combine_kernel(const T *__restrict__ sorted_y, const int32_t *__restrict__ inverse, const float *__restrict__ weights,
                                   const int32_t *__restrict__ experts, const T *__restrict__ x, int n_ffn, int top, int width,
                                   T *__restrict__ out) {
  wait_for_previous();
  const int t = blockIdx.x;
  for (int c = threadIdx.x * VEC; c < width; c += blockDim.x * VEC) {
    float acc[VEC];
#pragma unroll
    for (int e = 0; e < VEC; e++) acc[e] = 0.0f;
    for (int k = 0; k < top; k++) {
      const int64_t pair = (int64_t)t * top + k;
      const T *row = experts && experts[pair] >= n_ffn ? x + (int64_t)t * width : sorted_y + (inverse ? (int64_t)inverse[pair] : pair) * width;
      const float w = weights[pair];
      if (VEC == 4) {
        const float4 v = load4<T>(row + c);
        acc[0] = fmaf(w, v.x, acc[0]);
        acc[1 % VEC] = fmaf(w, v.y, acc[1 % VEC]);
        acc[2 % VEC] = fmaf(w, v.z, acc[2 % VEC]);
        acc[3 % VEC] = fmaf(w, v.w, acc[3 % VEC]);
      } else {
        acc[0] = fmaf(w, to_f32<T>(row[c]), acc[0]);
      }
    }
    if (VEC == 4) store4<T>(out + (int64_t)t * width + c, make_float4(acc[0], acc[1 % VEC], acc[2 % VEC], acc[3 % VEC]));
    else out[(int64_t)t * width + c] = from_f32<T>(acc[0]);
  }
}

}  // namespace seq

using namespace seq;

extern "C" int mrs_seq_moe_route(const float *logits, const float *correction, int n_tok, int n_experts, int n_groups, int keep_groups,
                                 int top, int renorm, int32_t *experts, float *weights, int64_t stream) {
  return mrs_seq_moe_route_scored(logits, correction, n_tok, n_experts, n_groups, keep_groups, top, renorm, MRS_SEQ_SCORE_SOFTMAX, 1, 1.0f,
                                  experts, weights, stream);
}

extern "C" int mrs_seq_moe_route_scored(const float *logits, const float *correction, int n_tok, int n_experts, int n_groups, int keep_groups,
                                        int top, int renorm, int score_fn, int group_top, float weight_scale, int32_t *experts,
                                        float *weights, int64_t stream) {
  const mrs_seq_moe_route_args a = {logits, correction, n_tok, n_experts, n_groups, keep_groups, top, renorm, score_fn, group_top, weight_scale, 0.0f,
                                    experts, weights, 0};
  return mrs_seq_moe_route_general(&a, stream);
}

static bool route_args_ok(const mrs_seq_moe_route_args &a) {
  return a.n_experts >= 1 && a.n_experts <= ROUTE_MAX_EXPERTS && a.n_groups >= 1 && a.n_experts % a.n_groups == 0 && a.keep_groups >= 1 &&
         a.keep_groups <= a.n_groups && a.top >= 1 && a.top <= a.n_experts && a.group_top >= 1 && a.renorm_eps >= 0.0f &&
         (a.score_fn == MRS_SEQ_SCORE_SOFTMAX || a.score_fn == MRS_SEQ_SCORE_SIGMOID);
}

extern "C" int mrs_seq_router_logits(const void *x, int dtype, const float *w, int width, int n_experts, int n_tok, float *logits, int64_t stream) {
  if (n_tok <= 0) return 0;
  if (!x || !w || !logits || width <= 0 || n_experts <= 0 || n_tok > 65535) return -2;
  const bool vec = width % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0;
  const dim3 grid(n_experts, n_tok);
  cudaStream_t st = (cudaStream_t)stream;
  SEQ_DISPATCH_DTYPE(dtype, {
    if (vec) router_logits_kernel<T, 4><<<grid, 128, 0, st>>>((const T *)x, w, width, n_experts, logits);
    else router_logits_kernel<T, 1><<<grid, 128, 0, st>>>((const T *)x, w, width, n_experts, logits);
  });
  return launch_status();
}

extern "C" int mrs_seq_moe_route_general(const mrs_seq_moe_route_args *args, int64_t stream) {
  const mrs_seq_moe_route_args &a = *args;
  const int n_tok = a.n_tok, n_experts = a.n_experts, n_groups = a.n_groups;
  if (n_tok <= 0) return 0;
  if (!route_args_ok(a)) return -2;
  const int warps = 4;
  const size_t bytes = (size_t)warps * (2 * n_experts + n_groups) * sizeof(float);
  return launch_after(moe_route_kernel, (n_tok + warps - 1) / warps, warps * 32, bytes, (cudaStream_t)stream, a);
}

extern "C" int mrs_seq_moe_router_fits(int width, int n_experts, int n_tok) {
  return width > 0 && n_experts >= 1 && n_experts <= ROUTE_FUSED_EXPERTS && n_tok >= 0 && n_tok <= ROUTE_FUSED_TOKENS &&
         (int64_t)width * n_experts <= ROUTE_FUSED_WEIGHTS;
}

extern "C" int mrs_seq_moe_router(const void *x, int dtype, const float *w, int width, const mrs_seq_moe_route_args *args, int64_t stream) {
  const mrs_seq_moe_route_args &a = *args;
  if (a.n_tok <= 0) return 0;
  if (!x || !w || !a.experts || !a.weights || !route_args_ok(a) || !mrs_seq_moe_router_fits(width, a.n_experts, a.n_tok)) return -2;
  const bool vec = width % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0;
  constexpr int threads = 128 * ROUTE_FUSED_GROUPS;
  SEQ_DISPATCH_DTYPE(dtype, {
    return vec ? launch_after(router_route_kernel<T, 4>, a.n_tok, threads, 0, (cudaStream_t)stream, (const T *)x, w, width, a)
               : launch_after(router_route_kernel<T, 1>, a.n_tok, threads, 0, (cudaStream_t)stream, (const T *)x, w, width, a);
  });
  return launch_status();
}

extern "C" int mrs_seq_moe_route_top_softmax(const float *logits, int n_tok, int n_experts, int top, int32_t *experts, float *weights,
                                             int64_t stream) {
  if (n_tok <= 0) return 0;
  if (n_experts < 1 || n_experts > ROUTE_MAX_EXPERTS || top < 1 || top > n_experts) return -2;
  const int warps = 4;
  return launch_after(moe_route_top_softmax_kernel, (n_tok + warps - 1) / warps, warps * 32, (size_t)warps * n_experts * sizeof(float),
                      (cudaStream_t)stream, logits, n_tok, n_experts, top, experts, weights);
}

extern "C" int mrs_seq_moe_up(const void *x, const void *up, int dtype, const int32_t *experts, int n_tok, int top, int width, int ff,
                              int act, void *hidden, int64_t stream) {
  if (n_tok <= 0) return 0;
  if ((size_t)width * sizeof(float) > 160 * 1024) return -2;
  const int warps = 8, bx = (ff + warps - 1) / warps;
  const size_t bytes = (size_t)width * sizeof(float);
  SEQ_DISPATCH_DTYPE(dtype, {
    auto kern = moe_up_kernel<T>;
    static size_t allowed = 48 * 1024;
    if (bytes > allowed) {
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
      allowed = bytes;
    }
    kern<<<dim3(bx < 256 ? bx : 256, n_tok * top), warps * 32, bytes, (cudaStream_t)stream>>>((const T *)x, (const T *)up, experts, top, width,
                                                                                             ff, act, (T *)hidden);
  });
  return launch_status();
}

extern "C" int mrs_seq_moe_gate_up(const void *x, const void *gate_up, int dtype, const int32_t *experts, int n_tok, int top, int width,
                                   int ff, int act, void *hidden, int64_t stream) {
  const mrs_seq_glu_rule rule = {act, 0.0f, 0.0f, 0.0f};
  return mrs_seq_moe_gate_up_rule(x, gate_up, dtype, experts, n_tok, top, width, ff, &rule, hidden, stream);
}

static int gate_up_some(const void *x, const void *gate_up, int dtype, const int32_t *experts, int n_tok, int top, int width, int ff,
                        const mrs_seq_glu_rule *rule, int n_ffn, void *hidden, int64_t stream) {
  if (n_tok <= 0) return 0;
  if (!rule) return -2;
  if ((size_t)width * sizeof(float) > 160 * 1024) return -2;
  const int warps = 8, bx = (ff + warps - 1) / warps;
  const size_t bytes = (size_t)width * sizeof(float);
  SEQ_DISPATCH_DTYPE(dtype, {
    auto kern = moe_gate_up_kernel<T>;
    static size_t allowed = 48 * 1024;
    if (bytes > allowed) {
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
      allowed = bytes;
    }
    kern<<<dim3(bx < 256 ? bx : 256, n_tok * top), warps * 32, bytes, (cudaStream_t)stream>>>(
        (const T *)x, (const T *)gate_up, experts, top, width, ff, *rule, n_ffn, (T *)hidden);
  });
  return launch_status();
}

extern "C" int mrs_seq_moe_gate_up_rule(const void *x, const void *gate_up, int dtype, const int32_t *experts, int n_tok, int top, int width,
                                        int ff, const mrs_seq_glu_rule *rule, void *hidden, int64_t stream) {
  return gate_up_some(x, gate_up, dtype, experts, n_tok, top, width, ff, rule, INT_MAX, hidden, stream);
}

static int down_some(const void *hidden, const void *down, int dtype, const int32_t *experts, const float *weights, int n_tok, int top, int width,
                     int ff, const void *x, int n_ffn, void *out, int64_t stream) {
  if (n_tok <= 0) return 0;
  const size_t bytes = (size_t)top * ff * sizeof(float);
  if (bytes > 160 * 1024) return -2;
  const int warps = 8, bx = (width + warps - 1) / warps;
  SEQ_DISPATCH_DTYPE(dtype, {
    auto kern = moe_down_kernel<T>;
    static size_t allowed = 48 * 1024;
    if (bytes > allowed) {
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
      allowed = bytes;
    }
    kern<<<dim3(bx < 256 ? bx : 256, n_tok), warps * 32, bytes, (cudaStream_t)stream>>>(
        (const T *)hidden, (const T *)down, experts, weights, top, width, ff, (const T *)x, n_ffn, (T *)out);
  });
  return launch_status();
}

extern "C" int mrs_seq_moe_down(const void *hidden, const void *down, int dtype, const int32_t *experts, const float *weights, int n_tok,
                                int top, int width, int ff, void *out, int64_t stream) {
  return down_some(hidden, down, dtype, experts, weights, n_tok, top, width, ff, nullptr, INT_MAX, out, stream);
}

extern "C" int mrs_seq_moe_small(const mrs_seq_moe_small_args *args, int64_t stream) {
  const mrs_seq_moe_small_args &a = *args;
  if (!a.x || a.n_ffn < 0) return -2;
  const int rc = gate_up_some(a.x, a.gate_up, a.dtype, a.experts, a.n_tok, a.top, a.width, a.ff, &a.rule, a.n_ffn, a.hidden, stream);
  if (rc != 0) return rc;
  return down_some(a.hidden, a.down, a.dtype, a.experts, a.weights, a.n_tok, a.top, a.width, a.ff, a.x, a.n_ffn, a.out, stream);
}

extern "C" int mrs_seq_moe_sort(const int32_t *experts, int n_pairs, int n_experts, int32_t *counts, int32_t *order, int64_t stream) {
  if (n_pairs <= 0) return 0;
  moe_sort_kernel<<<1, 1024, 2 * n_experts * sizeof(int32_t), (cudaStream_t)stream>>>(experts, n_pairs, n_experts, counts, order);
  return launch_status();
}

extern "C" int mrs_seq_moe_place_fits(int n_pairs, int n_experts) { return n_pairs > 0 && n_pairs <= MOE_PLACE_PAIRS && n_experts <= MOE_PLACE_PAIRS; }
extern "C" int mrs_seq_moe_place(const int32_t *experts, int n_pairs, int n_experts, const void *x, int dtype, int top, int width, int32_t *counts,
                                 int32_t *inverse, void *sorted, int64_t stream) {
  if (!mrs_seq_moe_place_fits(n_pairs, n_experts)) return -2;
  const int grid = n_pairs > n_experts ? n_pairs : n_experts;
  const int64_t row_bytes = (int64_t)width * (dtype == MRS_SEQ_BF16 ? 2 : 4);
  if (row_bytes % 16 == 0 && (((uintptr_t)x | (uintptr_t)sorted) & 15) == 0) {
    return launch_after(moe_place_kernel<uint4>, grid, 128, 0, (cudaStream_t)stream, experts, n_pairs, n_experts, (const uint4 *)x, top,
                             (int)(row_bytes / 16), counts, inverse, (uint4 *)sorted);
  }
  SEQ_DISPATCH_DTYPE(dtype, {
    return launch_after(moe_place_kernel<T>, grid, 128, 0, (cudaStream_t)stream, experts, n_pairs, n_experts, (const T *)x, top, width, counts,
                             inverse, (T *)sorted);
  });
  return launch_status();
}

extern "C" int mrs_seq_moe_gather(const void *x, int dtype, const int32_t *order, int n_pairs, int top, int width, void *sorted,
                                  int64_t stream) {
  if (n_pairs <= 0) return 0;
  const int64_t row_bytes = (int64_t)width * (dtype == MRS_SEQ_BF16 ? 2 : 4);
  if (row_bytes % 16 == 0 && (((uintptr_t)x | (uintptr_t)sorted) & 15) == 0) {
    moe_gather_kernel<uint4><<<n_pairs, 128, 0, (cudaStream_t)stream>>>((const uint4 *)x, order, top, (int)(row_bytes / 16), (uint4 *)sorted);
    return launch_status();
  }
  SEQ_DISPATCH_DTYPE(dtype, (moe_gather_kernel<T><<<n_pairs, 128, 0, (cudaStream_t)stream>>>((const T *)x, order, top, width, (T *)sorted)));
  return launch_status();
}

// shared memory of a grouped launch: as many rows per chunk (8, 4 or 2) as fit; 0: none do
static int grouped_rows(int n, int dtype) {
  const size_t row = (size_t)n * (dtype == MRS_SEQ_BF16 ? 2 : 4);
  for (int p = 8; p >= 2; p /= 2)
    if (p * row <= 200 * 1024) return p;
  return 0;
}

extern "C" int mrs_seq_moe_grouped_fits(int dtype, int width, int ff) {
  const int group = dtype == MRS_SEQ_BF16 ? 8 : 4;
  return width > 0 && ff > 0 && width % group == 0 && ff % group == 0 && grouped_rows(width, dtype) >= 4 && grouped_rows(ff, dtype) >= 4 ? 1 : 0;
}

extern "C" int mrs_seq_moe_grouped(const mrs_seq_moe_grouped_args *args, int64_t stream) {
  const mrs_seq_moe_grouped_args &a = *args;
  if (a.n_tok <= 0 || a.n_ffn <= 0) return 0;
  if (!a.x || !a.up || !a.down || !a.counts || !a.order || !a.hidden || !a.y || a.n_ffn > 65535 || !mrs_seq_moe_grouped_fits(a.dtype, a.width, a.ff)) return -2;
  if (((uintptr_t)a.x | (uintptr_t)a.up | (uintptr_t)a.down | (uintptr_t)a.hidden) & 15) return -3;
  const int warps = 8;
  const size_t elem = a.dtype == MRS_SEQ_BF16 ? 2 : 4;
#define SEQ_GROUPED(UP, GATED, P, ROWS)                                                                                       \
  {                                                                                                                           \
    auto kern = moe_grouped_kernel<T, UP, GATED>;                                                                             \
    const int per = grouped_rows(P.n, a.dtype), step = (GATED ? 2 : 4) * warps;                                               \
    const size_t bytes = (size_t)per * P.n * elem;                                                                            \
    static size_t allowed = 48 * 1024;                                                                                        \
    if (bytes > allowed) {                                                                                                    \
      const cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);            \
      if (err != cudaSuccess) return (int)err;                                                                                \
      allowed = bytes;                                                                                                        \
    }                                                                                                                         \
    const int blocks = (ROWS + step - 1) / step, most = (148 * 8 + a.n_ffn - 1) / a.n_ffn;                                    \
    kern<<<dim3(blocks < most ? blocks : most, a.n_ffn), warps * 32, bytes, (cudaStream_t)stream>>>(P, per);                  \
  }
  GroupedParams up = {a.x, a.up, a.counts, a.order, a.top, a.width, a.gated ? 2 * a.ff : a.ff, a.ff, a.rule, a.hidden};
  GroupedParams down = {a.hidden, a.down, a.counts, a.order, a.top, a.ff, a.width, a.ff, a.rule, a.y};
  SEQ_DISPATCH_DTYPE(a.dtype, {
    if (a.gated) SEQ_GROUPED(true, true, up, a.ff)
    else SEQ_GROUPED(true, false, up, a.ff)
    SEQ_GROUPED(false, false, down, a.width)
  });
#undef SEQ_GROUPED
  return launch_status();
}

// inverse: the row of each pair in sorted_y, or null: the order of the pairs
extern "C" int mrs_seq_moe_combine_at(const void *sorted_y, int dtype, const int32_t *inverse, const float *weights, const int32_t *experts, const void *x,
                                      int n_ffn, int n_tok, int top, int width, void *out, int64_t stream) {
  if (n_tok <= 0) return 0;
  if (experts && !x) return -2;
  const bool vec = width % 4 == 0 && (((uintptr_t)sorted_y | (uintptr_t)x | (uintptr_t)out) & 15) == 0;
  const int th = width >= 1024 ? 256 : 128;
#define SEQ_COMBINE(V)                                                                                                        \
  return launch_after(moe_combine_kernel<T, V>, n_tok, th, 0, (cudaStream_t)stream, (const T *)sorted_y, inverse,        \
                           weights, experts, (const T *)x, n_ffn, top, width, (T *)out)
  SEQ_DISPATCH_DTYPE(dtype, {
    if (vec) SEQ_COMBINE(4);
    else SEQ_COMBINE(1);
  });
#undef SEQ_COMBINE
  return launch_status();
}
extern "C" int mrs_seq_moe_combine_some(const void *sorted_y, int dtype, const int32_t *order, const float *weights, const int32_t *experts,
                                        const void *x, int n_ffn, int n_tok, int top, int width, int32_t *scratch_inverse, void *out,
                                        int64_t stream) {
  if (n_tok <= 0) return 0;
  if (experts && !x) return -2;
  const int n_pairs = n_tok * top;
  if (order) moe_inverse_kernel<<<(n_pairs + 255) / 256, 256, 0, (cudaStream_t)stream>>>(order, n_pairs, scratch_inverse);
  return mrs_seq_moe_combine_at(sorted_y, dtype, order ? scratch_inverse : nullptr, weights, experts, x, n_ffn, n_tok, top, width, out, stream);
}

extern "C" int mrs_seq_moe_combine(const void *sorted_y, int dtype, const int32_t *order, const float *weights, int n_tok, int top,
                                   int width, int32_t *scratch_inverse, void *out, int64_t stream) {
  return mrs_seq_moe_combine_some(sorted_y, dtype, order, weights, nullptr, nullptr, 0, n_tok, top, width, scratch_inverse, out, stream);
}

// The whole block behind one call: the steps are the entries above, their buffers one piece of scratch.  For calls from the host, whose
// six calls of a front end with a tensor each took longer than the kernels of small experts (32 experts of 5 MB, 8 tokens: 79 us of which
// the kernels make 43).
extern "C" int mrs_seq_moe_block(const mrs_seq_moe_block_args *args, int64_t stream) {
  const mrs_seq_moe_block_args &a = *args;
  if (a.n_tok <= 0) return 0;
  if (!a.x || !a.up || !a.down || !a.out || !a.scratch || (!a.router && !a.logits) || a.width <= 0 || a.ff <= 0 || a.top < 1 || a.n_ffn < 1 ||
      a.n_routes < a.n_ffn || (a.dtype != MRS_SEQ_BF16 && a.dtype != MRS_SEQ_F32))
    return -2;
  const int64_t pairs = (int64_t)a.n_tok * a.top, elem = a.dtype == MRS_SEQ_BF16 ? 2 : 4;
  if (pairs > INT_MAX) return -2;
  int64_t used = 0;
  auto piece = [&](int64_t bytes) {
    void *at = (uint8_t *)a.scratch + used;
    used += (bytes + 255) / 256 * 256;
    return at;
  };
  const bool fused = !a.logits && a.route != MRS_SEQ_ROUTE_TOP_SOFTMAX && mrs_seq_moe_router_fits(a.width, a.n_routes, a.n_tok);
  float *logits = a.logits || fused ? nullptr : (float *)piece((int64_t)a.n_tok * a.n_routes * 4);
  int32_t *experts = (int32_t *)piece(pairs * 4);
  float *weights = (float *)piece(pairs * 4);
  const bool streams = a.products == MRS_SEQ_PRODUCTS_STREAMED;
  int32_t *counts = streams ? nullptr : (int32_t *)piece((int64_t)a.n_routes * 4), *at = streams ? nullptr : (int32_t *)piece(pairs * 4);
  void *hidden = piece(pairs * a.ff * elem), *y = streams ? nullptr : piece(pairs * a.width * elem);
  void *rows = a.products == MRS_SEQ_PRODUCTS_ONE_LAUNCH ? piece(pairs * a.width * elem) : nullptr;
  if (used > a.scratch_bytes || ((uintptr_t)a.scratch & 15)) return -3;

  int rc = 0;
  const mrs_seq_moe_route_args r = {a.logits ? a.logits : logits, a.correction, a.n_tok, a.n_routes, a.n_groups, a.keep_groups, a.top, a.renorm,
                                    a.route == MRS_SEQ_ROUTE_SIGMOID ? MRS_SEQ_SCORE_SIGMOID : MRS_SEQ_SCORE_SOFTMAX, a.group_top, a.weight_scale,
                                    a.renorm_eps, experts, weights, a.logits ? a.logits_ld : 0};
  if (logits) rc = mrs_seq_router_logits(a.x, a.dtype, a.router, a.width, a.n_routes, a.n_tok, logits, stream);
  if (rc != 0) return rc;
  if (fused) rc = mrs_seq_moe_router(a.x, a.dtype, a.router, a.width, &r, stream);
  else if (a.route != MRS_SEQ_ROUTE_TOP_SOFTMAX) rc = mrs_seq_moe_route_general(&r, stream);
  else if (a.logits && a.logits_ld != a.n_routes) return -2;
  else rc = mrs_seq_moe_route_top_softmax(r.logits, a.n_tok, a.n_routes, a.top, experts, weights, stream);
  if (rc != 0) return rc;

  const bool identities = a.n_routes > a.n_ffn;
  if (streams) {
    if (a.gated) {
      const mrs_seq_moe_small_args s = {a.x, a.up, a.down, a.dtype, experts, weights, a.n_tok, a.top, a.width, a.ff, a.n_ffn, a.rule, hidden, a.out};
      return mrs_seq_moe_small(&s, stream);
    }
    if (identities) return -2;
    rc = mrs_seq_moe_up(a.x, a.up, a.dtype, experts, a.n_tok, a.top, a.width, a.ff, a.rule.act, hidden, stream);
    return rc != 0 ? rc : mrs_seq_moe_down(hidden, a.down, a.dtype, experts, weights, a.n_tok, a.top, a.width, a.ff, a.out, stream);
  }
  const int32_t *inverse = nullptr;
  if (a.products == MRS_SEQ_PRODUCTS_GROUPED) {
    rc = mrs_seq_moe_sort(experts, (int)pairs, a.n_routes, counts, at, stream);
    if (rc != 0) return rc;
    const mrs_seq_moe_grouped_args g = {a.x, a.up, a.down, a.dtype, counts, at, a.n_tok, a.top, a.width, a.ff, a.n_ffn, a.gated, a.rule, hidden, y};
    rc = mrs_seq_moe_grouped(&g, stream);
  } else {
    if (a.dtype != MRS_SEQ_BF16) return -2;
    rc = mrs_seq_moe_place(experts, (int)pairs, a.n_routes, a.x, a.dtype, a.top, a.width, counts, at, rows, stream);
    if (rc != 0) return rc;
    inverse = at;
    rc = mrs_seq_moe_products(rows, a.up, a.down, counts, (int)pairs, a.n_ffn, a.width, a.ff, a.gated, &a.rule, hidden, y, stream);
  }
  return rc != 0 ? rc
                 : mrs_seq_moe_combine_at(y, a.dtype, inverse, weights, identities ? experts : nullptr, identities ? a.x : nullptr, identities ? a.n_ffn : 0,
                                          a.n_tok, a.top, a.width, a.out, stream);
}
