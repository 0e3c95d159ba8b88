// moe_gemm.cu — the matrix products of routed experts on the 5th-gen tensor cores (tcgen05 + TMEM), all experts in ONE launch: rows
// sorted by expert, row counts read on the device, so a step needs no host read and can be captured.  The first product's two
// halves meet in the epilogue (gate and up rows of an expert fill the two halves of one weight tile), so only the joined hidden
// rows are written.
//
// Persistent CTAs (one per SM) walk the tiles of 128 rows x 256 weight rows; 320 threads:
//   warp 0      TMA: row tiles and weight tiles of 64 columns through a 4-stage ring (SWIZZLE_128B boxes of 128 rows);
//   warp 1      MMA issuer: 128 x 256 accumulators in tensor memory, two of them, so the epilogue of a tile runs beside the
//               products of the next;
//   warps 2..9  epilogue, thread = row = TMEM lane, two warps share a row's columns: activation or join in f32 (the sigmoids with
//               the fast exponential and division: the result is rounded to bf16), rows written 16 bytes at a time.
// Tiles are ordered expert by expert, weight tile by weight tile, row tiles innermost: the CTAs that run at one time share
// weight tiles.  Rows past an expert's last belong to its neighbour (or are zeros): each accumulator row depends on its own
// input row alone and is stored only where it belongs.
//
// In a step of few rows the weights' bytes are the bound, and the launches around the two products are half as long as one of them
// (16 experts of 25 MB, 32 tokens to 4 of them, in a graph: 81 us of 94).  So every launch of the chain may begin while the one before
// it runs, and the second product fetches the first weights of its tiles before it waits for the hidden rows: 86 us.
//
// Every wait has a limit; a wait that runs out sets a device flag (mrs_seq_moe_gemm_timeouts) and ends the CTA.
#include "seq_common.cuh"
#include "seq_tc.cuh"

namespace seqg {
using namespace seqtc;

constexpr int BM = 128, BN = 256, BK = 64, STAGES = 4, EPI_WARPS = 8, THREADS = 64 + 32 * EPI_WARPS, MAX_EXPERTS = 1024;
constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int SMEM = STAGES * STAGE_BYTES + 256;
constexpr uint32_t TCOLS = 512;
constexpr int N_BARS = 2 * STAGES + 5;      // full, empty per stage; accumulator full, empty per buffer; drain

struct Params {
  const int32_t *counts;       // rows per expert
  int n_ffn, n, k;             // experts; output columns per expert (GATED: 2 n weight rows, gate rows then up rows); length of a dot
  mrs_seq_glu_rule rule;
  __nv_bfloat16 *out;          // [sorted rows][n]
  bool early;                  // the launch before this one is not the writer of counts and weights: they are read while it still runs
};

__device__ int g_timeouts = 0;

__device__ __forceinline__ bool wait(uint64_t *bar, uint32_t parity) { return wait_bounded(bar, parity, &g_timeouts); }

__device__ __forceinline__ float fast_sigmoid(float z) { return __fdividef(1.0f, 1.0f + __expf(-z)); }

// 32 columns of a row: v = join(v, u) (GATED) or act(v)
template <bool GATED> __device__ __forceinline__ void finish(uint32_t *v, const uint32_t *u, const mrs_seq_glu_rule &rule) {
  auto f = [](uint32_t x) { return __uint_as_float(x); };
  if (GATED && rule.act == MRS_SEQ_GLU_CAPPED) {
#pragma unroll
    for (int i = 0; i < 32; i++) {
      const float g = fminf(f(v[i]), rule.limit), w = fminf(fmaxf(f(u[i]), -rule.limit), rule.limit);
      v[i] = __float_as_uint(g * fast_sigmoid(rule.slope * g) * (w + rule.shift));
    }
  } else if (GATED && rule.act == MRS_SEQ_ACT_SILU) {
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __float_as_uint(f(v[i]) * fast_sigmoid(f(v[i])) * f(u[i]));
  } else if (!GATED && rule.act == MRS_SEQ_ACT_RELU_SQ) {
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __float_as_uint(seq::relu_sq_f(f(v[i])));
  } else if (GATED || rule.act != MRS_SEQ_ACT_NONE) {
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __float_as_uint(GATED ? seq::glu_join(f(v[i]), f(u[i]), rule) : seq::apply_act(f(v[i]), rule.act));
  }
}

struct Tile {
  int a_row, rows, b_row0, b_row1, col;      // first input row, rows of it that are the expert's, weight rows of the two halves, first output column
};

template <bool GATED>
__global__ void __launch_bounds__(THREADS, 1) moe_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const Params p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ int tiles_before[MAX_EXPERTS + 1], rows_before[MAX_EXPERTS + 1];
  uint64_t *bars = (uint64_t *)(smem + STAGES * STAGE_BYTES);
  uint64_t *full = bars, *empty = bars + STAGES, *acc_full = bars + 2 * STAGES, *acc_empty = acc_full + 2, *drain = acc_empty + 2;
  uint32_t *tmem_slot = (uint32_t *)(bars + N_BARS);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int cols = GATED ? BN / 2 : BN;                // output columns of a tile
  const int n_tiles = (p.n + cols - 1) / cols;

  if (!p.early) seq::wait_for_previous();
  if (smem_u32(smem) & 1023) {               // the swizzled boxes need it; never seen
    seq::wait_for_previous();
    if (threadIdx.x == 0) atomicExch(&g_timeouts, 2);
    return;
  }
  if (warp == 0) {                           // running sums of row tiles and rows over the experts
    int tiles = 0, rows = 0;
    for (int e0 = 0; e0 < p.n_ffn; e0 += 32) {
      const int c = e0 + lane < p.n_ffn ? p.counts[e0 + lane] : 0;
      int a = (c + BM - 1) / BM, b = c;
      for (int d = 1; d < 32; d <<= 1) {
        const int ua = __shfl_up_sync(0xffffffffu, a, d), ub = __shfl_up_sync(0xffffffffu, b, d);
        if (lane >= d) { a += ua; b += ub; }
      }
      if (e0 + lane < p.n_ffn) { tiles_before[e0 + lane + 1] = tiles + a; rows_before[e0 + lane + 1] = rows + b; }
      tiles += __shfl_sync(0xffffffffu, a, 31);
      rows += __shfl_sync(0xffffffffu, b, 31);
    }
    if (lane == 0) tiles_before[0] = rows_before[0] = 0;
  }
  if (warp == 1) {
    if (lane < N_BARS) {
      mbar_init(&bars[lane], lane == 2 * STAGES + 2 || lane == 2 * STAGES + 3 ? (uint32_t)EPI_WARPS : 1u);      // acc_empty: the epilogue warps
      fence_mbar_init();
    }
    __syncwarp();
    tmem_alloc(tmem_slot, TCOLS);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __reduce_max_sync(0xffffffffu, *tmem_slot);
  const int total = tiles_before[p.n_ffn] * n_tiles, k_steps = (p.k + BK - 1) / BK;

  auto tile_of = [&](int t) {
    int lo = 0, hi = p.n_ffn;                // the expert with tiles_before[e] * n_tiles <= t < tiles_before[e + 1] * n_tiles
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (tiles_before[mid] * n_tiles <= t) lo = mid;
      else hi = mid;
    }
    const int m_tiles = tiles_before[lo + 1] - tiles_before[lo], r = t - tiles_before[lo] * n_tiles;
    const int nt = r / m_tiles, mt = r % m_tiles;
    Tile x;
    x.a_row = rows_before[lo] + mt * BM;
    x.rows = min(BM, rows_before[lo + 1] - x.a_row);
    x.col = nt * cols;
    x.b_row0 = (GATED ? 2 * lo : lo) * p.n + x.col;
    x.b_row1 = GATED ? x.b_row0 + p.n : x.b_row0 + BN / 2;
    return x;
  };

  if (warp == 0) {
    // ===================== TMA producer =====================
    auto load_weights = [&](const Tile &x, int ks, int s) {
      uint8_t *b_s = smem + s * STAGE_BYTES + A_BYTES;
      mbar_arrive_expect_tx_warp(full + s, STAGE_BYTES);
      tma_load_2d_warp(b_s, &tmap_b, ks * BK, x.b_row0, full + s);
      tma_load_2d_warp(b_s + B_BYTES / 2, &tmap_b, ks * BK, x.b_row1, full + s);
    };
    int it = 0, ahead = 0;                   // ahead: stages whose weights are on their way
    if (p.early && (int)blockIdx.x < total) {
      const Tile x = tile_of(blockIdx.x);
      for (; ahead < min(STAGES, k_steps); ahead++) load_weights(x, ahead, ahead);
    }
    seq::wait_for_previous();
    seq::let_next_start();
    bool ok = true;
    for (int t = blockIdx.x; ok && t < total; t += gridDim.x) {
      const Tile x = tile_of(t);
      for (int ks = 0; ks < k_steps; ks++, it++) {
        const int s = it % STAGES;
        if (it >= ahead) {
          ok = wait(empty + s, ((it / STAGES) & 1) ^ 1);
          if (!ok) break;
          load_weights(x, ks, s);
        }
        tma_load_2d_warp(smem + s * STAGE_BYTES, &tmap_a, ks * BK, x.a_row, full + s);
      }
    }
    // copies in flight land before the CTA may end
    for (int i = max(0, it - STAGES); i < it; i++) wait(full + i % STAGES, (i / STAGES) & 1);
  } else if (warp == 1) {
    // ===================== MMA issuer =====================
    // c = f32 (bit 4), a / b = bf16 (bits 7, 10), N >> 3 at bit 17, M >> 4 at bit 24
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
    int it = 0, j = 0;
    bool ok = true;
    seq::wait_for_previous();
    for (int t = blockIdx.x; ok && t < total; t += gridDim.x, j++) {
      const uint32_t t_acc = tmem_base + (uint32_t)((j & 1) * BN);
      ok = wait(acc_empty + (j & 1), ((j >> 1) & 1) ^ 1);
      if (!ok) break;
      tc_fence_after();
      for (int ks = 0; ks < k_steps; ks++, it++) {
        const int s = it % STAGES;
        ok = wait(full + s, (it / STAGES) & 1);
        if (!ok) break;
        tc_fence_after();
        const uint64_t ad = umma_desc_sw128(smem + s * STAGE_BYTES), bd = umma_desc_sw128(smem + s * STAGE_BYTES + A_BYTES);
#pragma unroll
        for (int c = 0; c < BK / 16; c++) umma_ss_warp(t_acc, ad + (uint64_t)(2 * c), bd + (uint64_t)(2 * c), idesc, (ks | c) ? 1u : 0u);
        umma_commit_warp(empty + s);
      }
      if (ok) umma_commit_warp(acc_full + (j & 1));
    }
    if (it > 0) {                            // no product is in flight when tensor memory is freed
      umma_commit_warp(drain);
      wait(drain, 0);
    }
  } else {
    // ===================== epilogue: thread = row of the tile =====================
    const int q4 = warp & 3, r = q4 * 32 + lane, part = (warp - 2) >> 2;      // a warp reads its own quarter of the TMEM lanes
    const uint32_t lane_off = (uint32_t)(q4 * 32) << 16;
    int j = 0;
    seq::wait_for_previous();
    for (int t = blockIdx.x; t < total; t += gridDim.x, j++) {
      const Tile x = tile_of(t);
      const bool ok = __all_sync(0xffffffffu, wait(acc_full + (j & 1), (j >> 1) & 1));
      if (!ok) break;
      tc_fence_after();
      const uint32_t t_acc = tmem_base + (uint32_t)((j & 1) * BN) + lane_off;
      const bool stores = r < x.rows;
      __nv_bfloat16 *orow = p.out + (int64_t)(x.a_row + r) * p.n + x.col;
#pragma unroll 1
      for (int c0 = part * (cols / 2); c0 < (part + 1) * (cols / 2); c0 += 32) {
        if (x.col + c0 >= p.n) break;
        uint32_t v[32], u[32];
        tmem_ld_32x32(t_acc + (uint32_t)c0, v);
        if (GATED) tmem_ld_32x32(t_acc + (uint32_t)(BN / 2 + c0), u);
        if (!stores) continue;
        finish<GATED>(v, u, p.rule);
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          if (x.col + c0 + i >= p.n) break;
          uint4 pk;
          uint32_t *w = (uint32_t *)&pk;
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const __nv_bfloat162 hh = __floats2bfloat162_rn(__uint_as_float(v[i + 2 * e]), __uint_as_float(v[i + 2 * e + 1]));
            w[e] = *(const uint32_t *)&hh;
          }
          *(uint4 *)(orow + c0 + i) = pk;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty + (j & 1));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TCOLS);
}

}  // namespace seqg

extern "C" int mrs_seq_moe_gemm_fits(int dtype, int n, int k, int n_ffn) {
  return dtype == MRS_SEQ_BF16 && n >= 8 && n % 8 == 0 && k >= 8 && k % 8 == 0 && n_ffn >= 1 && n_ffn <= seqg::MAX_EXPERTS ? 1 : 0;
}

extern "C" int mrs_seq_moe_gemm_timeouts(void) {
  int v = 0;
  const cudaError_t e = cudaMemcpyFromSymbol(&v, seqg::g_timeouts, sizeof(int));
  return e == cudaSuccess ? v : -(int)e;
}

namespace seqg {
static int launch(const void *sorted, const void *weights, const int32_t *counts, int n_rows, int n_ffn, int n, int k, int gated, const mrs_seq_glu_rule *rule,
                  void *out, bool early, int64_t stream) {
  if (!sorted || !weights || !counts || !out || !rule || !mrs_seq_moe_gemm_fits(MRS_SEQ_BF16, n, k, n_ffn)) return -2;
  if (((uintptr_t)sorted | (uintptr_t)weights | (uintptr_t)out) & 15) return -3;
  CUtensorMap ta, tb;
  // weights: the next 64 columns of a row are wanted next, and one 256-byte fetch brings both.  16 experts of 25 MB, 32 tokens to 4 of
  // them: 88.1 us with fetches of 128 bytes, 86.0 so (16 sorted rows at a time instead of 128 made no difference at all)
  if (!tc_make_map_2d(&ta, sorted, (uint64_t)n_rows, (uint64_t)k, BK, BM, 1) ||
      !tc_make_map_2d(&tb, weights, (uint64_t)n_ffn * n * (gated ? 2 : 1), (uint64_t)k, BK, BN / 2, 1, CU_TENSOR_MAP_L2_PROMOTION_L2_256B))
    return -4;
  static bool raised = false;
  if (!raised) {
    cudaError_t e = cudaFuncSetAttribute(moe_gemm_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(moe_gemm_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    raised = true;
  }
  Params p = {};
  p.counts = counts; p.n_ffn = n_ffn; p.n = n; p.k = k; p.rule = *rule; p.out = (__nv_bfloat16 *)out; p.early = early;
  const int cols = gated ? BN / 2 : BN;
  const int64_t most = ((int64_t)(n_rows + BM - 1) / BM + (n_ffn < n_rows ? n_ffn : n_rows)) * ((n + cols - 1) / cols);      // tiles at any split of the rows
  const int grid = (int)(most < 148 ? most : 148);
  return seq::launch_after(gated ? moe_gemm_kernel<true> : moe_gemm_kernel<false>, grid, THREADS, SMEM, (cudaStream_t)stream, ta, tb, p);
}
}  // namespace seqg

extern "C" int mrs_seq_moe_gemm(const void *sorted, const void *weights, const int32_t *counts, int n_rows, int n_ffn, int n, int k, int gated,
                                const mrs_seq_glu_rule *rule, void *out, int64_t stream) {
  return n_rows <= 0 ? 0 : seqg::launch(sorted, weights, counts, n_rows, n_ffn, n, k, gated, rule, out, false, stream);
}

// The second launch may read counts and its weights early: the first one began after all that came before it had ended.
extern "C" int mrs_seq_moe_products(const void *sorted, const void *up, const void *down, const int32_t *counts, int n_rows, int n_ffn, int width, int ff,
                                    int gated, const mrs_seq_glu_rule *rule, void *hidden, void *out, int64_t stream) {
  if (n_rows <= 0) return 0;
  if (!down || !out || (((uintptr_t)down | (uintptr_t)out) & 15) || !mrs_seq_moe_gemm_fits(MRS_SEQ_BF16, width, ff, n_ffn)) return -2;
  const mrs_seq_glu_rule none = {};
  const int rc = seqg::launch(sorted, up, counts, n_rows, n_ffn, ff, width, gated, rule, hidden, false, stream);
  return rc != 0 ? rc : seqg::launch(hidden, down, counts, n_rows, n_ffn, width, ff, 0, &none, out, true, stream);
}
