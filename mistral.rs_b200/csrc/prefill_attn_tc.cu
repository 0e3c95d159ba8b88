// prefill_attn_tc.cu — causal (var-len) prompt attention on the 5th-gen tensor cores (tcgen05 + TMEM), head sizes 64 and 128.
//
// Same contract and arithmetic class as prefill_attn.cu (REF mistralrs-core/src/paged_attention/layers/
// paged_attention.rs:1413-1475 -> flash_attn_varlen): S = QK^T and O = PV on 16-bit MMAs with
// f32 accumulation, online softmax in f32 (base-2 exponent, scale folded), P rounded to the activation dtype before
// the second GEMM.  mrs_prefill_attention routes here without softcap; prefill_attn.cu (mma.sync) keeps every other case.
//
// One CTA = 128 query rows of one (sequence, head), 128-token K/V tiles, 192 threads:
//   warp 0      TMA: Q once (SWIZZLE_128B boxes of 64 d), then a K and a V tile at a time;
//   warp 1      MMA issuer (one elected lane, warp-convergent):
//                 S_j  = Q K_j^T      SS form, both operands K-major in shared memory, M128 N128 K16 x D / 16
//                 O   += P_j V_j      TS form: P (16-bit pairs) is the A operand in TENSOR MEMORY, V is the B operand
//                                     straight from its row-major [token][d] tile = MN-major SWIZZLE_128B
//                                     (no transpose pass): M128 N = D K16 x 8
//   warps 2..5  softmax + correction + epilogue, thread = query row = TMEM lane: tcgen05.ld the S row (two passes:
//               max, then exp2 / sum / pack), tcgen05.st P IN PLACE over the first 64 columns of S (a row is private
//               to its thread, and chunk c of P lands on columns the thread has already read), rescale O in TMEM only
//               when some row's maximum moved (warp vote), finally O / l -> global.
// The per-tile chain S -> softmax -> PV is latency-bound, so the kernel is laid out for TWO CTAs per SM instead of a deeper pipeline inside
// one: single K / V stages (96 KB of shared memory), 256 TMEM columns — S / P [0,128), O from 128 on — and the other CTA's MMAs fill this
// one's softmax.  (Two chains of one CTA over the same K / V tiles, with S and P side by side in tensor memory, tiles of 80 keys and an issuer
// each, took 1720 clocks for 128 keys of 128 rows against 2300, but their exponentials ran in step, and clocks fell to 1.6 GHz: 89 us where this
// takes 75, and slower up to 1000 tokens.)
// What bounds it: exponentials (16 a clock and SM), products (1024 clocks a tile) and the latencies between them, then the power limit.
// One B200, us in a captured graph before / after waits in one piece, products issued four at a time, heavy query tiles of all heads first
// and loads that start before the rest of the CTA is set up; 32 heads on 8 of size 128, bf16: 300 tokens 9.2 / 8.8, 1000 20.6 / 18.6, 2900
// 100 / 76, 2900 + 1921 + 2631 212 / 191.  Against prefill_attn.cu, which had them before: head size 64, 14 heads on 2, 3000 tokens 248 / 46;
// size 128 with a window of 1023, 3000 tokens 395 / 73; 17 tokens of either 6.2 / 5.4 and 7.4 / 7.0.
#include "tc_common.cuh"

#include <math.h>
#include <stdio.h>
#include <type_traits>

namespace mrs {

constexpr int FT_BM = 128, FT_BN = 128;
constexpr int FT_THREADS = 32 * 6;
constexpr uint32_t FT_TCOLS = 256;
constexpr uint32_t FT_WAIT_LIMIT = 1u << 22;
template <int D> constexpr int ft_tile_bytes() { return FT_BN * D * 2; }         // D / 64 boxes [128 rows][64 d]
template <int D> constexpr int ft_smem() { return 1024 + 3 * ft_tile_bytes<D>() + 256; }   // Q + K + V + barriers

struct FtParams {
  void *o;
  const int32_t *cu_seqlens;   // [B + 1] or nullptr (single sequence of length T)
  int *timeouts;               // set when a wait runs out
  int T, H, KVH;
  int64_t o_stride;            // elements between consecutive tokens of the output
  float scale_log2;            // softmax_scale * log2(e)
  float slack;                 // how far a row's maximum may outgrow the exponent's reference point (base 2)
  int causal, window_left;     // (window_left: WINDOW)
  uint32_t v_lbo, v_sbo;       // MN-major descriptor strides of the V operand, bytes
};

// Products of a tile by the whole warp, one elected lane issuing (operands in uniform registers; descriptor fields as in umma_desc_sw128).
// S = Q K^T over 64 d: both operands 32 bytes on inside the SWIZZLE_128B atom each time.
__device__ __forceinline__ void ft_mma_s4(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred e, p, q;\n\t.reg .b32 l, m;\n\t.reg .b64 x, y;\n\t"
      "elect.sync _|e, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.eq.b32 q, %3, %3;\n\t"
      "shr.u32 l, %1, 4;\n\tor.b32 l, l, 0x10000;\n\tshr.u32 m, %2, 4;\n\tor.b32 m, m, 0x10000;\n\t"
      "mov.b64 x, {l, %5};\n\tmov.b64 y, {m, %5};\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %3, p;\n\t"
      "add.u32 l, l, 2;\n\tadd.u32 m, m, 2;\n\tmov.b64 x, {l, %5};\n\tmov.b64 y, {m, %5};\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %3, q;\n\t"
      "add.u32 l, l, 2;\n\tadd.u32 m, m, 2;\n\tmov.b64 x, {l, %5};\n\tmov.b64 y, {m, %5};\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %3, q;\n\t"
      "add.u32 l, l, 2;\n\tadd.u32 m, m, 2;\n\tmov.b64 x, {l, %5};\n\tmov.b64 y, {m, %5};\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %3, q;\n\t"
      "}" ::"r"(d), "r"(a), "r"(b), "r"(idesc), "r"(accumulate), "n"((1024 >> 4) | (1 << 14) | (2 << 29))
      : "memory");
}
// O += P V over 16 tokens (lo, hi: the words of V's descriptor)
__device__ __forceinline__ void ft_mma_o(uint32_t d, uint32_t a, uint32_t lo, uint32_t hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred e, p;\n\t.reg .b64 x;\n\telect.sync _|e, 0xffffffff;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 x, {%2, %3};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], x, %4, p;\n\t}" ::"r"(d), "r"(a), "r"(lo), "r"(hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void tmem_ld_32x32_nowait(uint32_t taddr, uint32_t *r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st_x16(uint32_t taddr, const uint32_t *r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::
          "r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// By the whole warp.  False when the phase did not complete within the limit: the caller then ends its part of the CTA.  (A tile passes six waits in
// turn; a loop that left PTX to vote in each round took 81 us for 2900 tokens, 32 heads on 8, this one 75.)
__device__ __forceinline__ bool ft_wait(uint64_t *bar, uint32_t parity, int *timeouts) {
  if (mbar_wait_warp(bar, parity, FT_WAIT_LIMIT)) return true;
  *(volatile int *)timeouts = 1;
  return false;
}

template <int D, bool BF, bool WINDOW>
__global__ void __launch_bounds__(FT_THREADS, 2)
prefill_attn_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                       const __grid_constant__ CUtensorMap tmap_v, const FtParams p) {
  constexpr int TILE = ft_tile_bytes<D>(), BOX = FT_BN * 128, BOXES = D / 64;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t *q_s = smem, *k_s = smem + TILE, *v_s = smem + 2 * TILE;
  uint64_t *bars = (uint64_t *)(smem + 3 * TILE);
  uint64_t *q_full = bars, *k_full = bars + 1, *k_empty = bars + 2, *v_full = bars + 3, *v_empty = bars + 4, *s_full = bars + 5,
           *p_full = bars + 6, *pv_done = bars + 7, *v_clean = bars + 8;
  uint32_t *tmem_slot = (uint32_t *)(bars + 9);
  int *const late = p.timeouts;

  // (the warp index from lane 0: the compiler then knows that a warp's branches are uniform and keeps the issuer's operands in uniform registers)
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int h = blockIdx.x, b = blockIdx.y;
  const int kvh = h / (p.H / p.KVH);
  int seq0 = 0, len = p.T;
  if (p.cu_seqlens != nullptr) { seq0 = p.cu_seqlens[b]; len = p.cu_seqlens[b + 1] - seq0; }
  const int ntile_q = (len + FT_BM - 1) / FT_BM;
  const int qt = (int)gridDim.z - 1 - (int)blockIdx.z;      // heavy (late) query tiles of all heads and sequences first
  if (qt >= ntile_q) return;
  const int q0 = qt * FT_BM;
  const int q_hi = min(len, q0 + FT_BM) - 1;
  const int kv_end = p.causal ? (q_hi + 1) : len;
  // Tiles start at the first key that a row of the tile may see, wherever that lies (a tile's row needs no alignment): nothing before it is read.
  const int first = WINDOW ? max(0, q0 - p.window_left) : 0;
  const int nt = (kv_end - first + FT_BN - 1) / FT_BN;
  // Past the last key that a row may see the last tile holds later tokens' rows or the next sequence's: masked scores in S, but a value times a
  // probability of zero, which is not zero where that value is no finite number.  The producer clears them.
  const bool ragged = (WINDOW || p.cu_seqlens != nullptr) && first + nt * FT_BN > kv_end;

  // The producer initialises the barriers and goes on to its first loads; the CTA barrier, which it does not wait for, orders that before the
  // others' first wait.
  uint32_t tmem_base = 0u;
  if (warp == 0) {
    if (lane < 9) mbar_init(&bars[lane], lane == 6 ? 4u : 1u);      // p_full: the four softmax warps
    fence_mbar_init();
    __syncwarp();
    asm volatile("bar.arrive 1, %0;" ::"n"(FT_THREADS) : "memory");
  } else {
    if (warp == 1) tmem_alloc(tmem_slot, FT_TCOLS);
    tc_fence_before();
    asm volatile("bar.sync 1, %0;" ::"n"(FT_THREADS) : "memory");
    tc_fence_after();
    tmem_base = __reduce_max_sync(0xffffffffu, *tmem_slot);
  }
  const uint32_t t_s = tmem_base, t_p = tmem_base, t_o = tmem_base + 128u;   // P overwrites the head of S

  if (warp == 0) {
    // ===================== TMA producer =====================
    auto load = [&](uint8_t *dst, const CUtensorMap *map, int x, int row, uint64_t *bar) {
      mbar_arrive_expect_tx_warp(bar, TILE);
#pragma unroll
      for (int i = 0; i < BOXES; i++) tma_load_2d_warp(dst + i * BOX, map, x + 64 * i, row, bar);
    };
    bool ok = true;
    int nk = 0, nv = 0;
    load(q_s, &tmap_q, h * D, seq0 + q0, q_full);
    for (int j = 0; j < nt; j++) {
      const int ph = j & 1, row = seq0 + first + j * FT_BN;
      ok = ft_wait(k_empty, ph ^ 1, late);
      if (!ok) break;
      load(k_s, &tmap_k, kvh * D, row, k_full);
      nk++;
      ok = ft_wait(v_empty, ph ^ 1, late);
      if (!ok) break;
      load(v_s, &tmap_v, kvh * D, row, v_full);
      nv++;
    }
    // copies in flight land before the CTA may end
    ft_wait(q_full, 0, late);
    if (nk > 0) ft_wait(k_full, (nk - 1) & 1, late);
    if (nv > 0) ft_wait(v_full, (nv - 1) & 1, late);
    if (ok && ragged) {
      const int r0 = kv_end - first - (nt - 1) * FT_BN;                            // rows r0 .. 127 of the last tile
      for (int i = lane; i < (FT_BN - r0) * 8 * BOXES; i += 32) {            // (a row of a box is 128 bytes wherever the swizzle puts its parts)
        const int x = i / ((FT_BN - r0) * 8), y = i - x * (FT_BN - r0) * 8;
        sts128(smem_u32(v_s) + (uint32_t)(x * BOX + r0 * 128 + y * 16), make_uint4(0u, 0u, 0u, 0u));
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(v_clean);
    }
  } else if (warp == 1) {
    // ===================== MMA issuer =====================
    constexpr uint32_t fmt = BF ? 1u : 0u;
    // c = f32 (bit 4), a / b format (bits 7, 10), b_major = MN (bit 16) for the PV product, N >> 3 at bit 17, M >> 4 at bit 24
    constexpr uint32_t idesc_s = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(FT_BN >> 3) << 17) | ((uint32_t)(FT_BM >> 4) << 24);
    constexpr uint32_t idesc_o = (1u << 4) | (fmt << 7) | (fmt << 10) | (1u << 16) | ((uint32_t)(D >> 3) << 17) | ((uint32_t)(FT_BM >> 4) << 24);
    // (reductions leave their result in uniform registers, where the products take their operands from)
    const uint32_t qb = __reduce_max_sync(0xffffffffu, smem_u32(q_s)), kb = __reduce_max_sync(0xffffffffu, smem_u32(k_s)),
                   v_lo = __reduce_max_sync(0xffffffffu, (smem_u32(v_s) >> 4) | ((p.v_lbo >> 4) << 16)),
                   v_hi = __reduce_max_sync(0xffffffffu, (p.v_sbo >> 4) | (1u << 14) | (2u << 29));
    int scored = 0, done = 0;
    bool ok = ft_wait(q_full, 0, late);
    for (int j = 0; ok && j < nt; j++) {
      const int ph = j & 1;
      ok = ft_wait(k_full, ph, late) && (j == 0 || ft_wait(pv_done, ph ^ 1, late));   // PV_{j-1} has read P out of the S columns S_j is about to overwrite
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int i = 0; i < BOXES; i++) ft_mma_s4(t_s, qb + (uint32_t)(i * BOX), kb + (uint32_t)(i * BOX), idesc_s, i ? 1u : 0u);
      umma_commit_warp(s_full);
      umma_commit_warp(k_empty);
      scored++;
      ok = ft_wait(v_full, ph, late) && (!ragged || j + 1 < nt || ft_wait(v_clean, 0, late)) && ft_wait(p_full, ph, late);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int i = 0; i < 8; i++)     // 16 tokens per MMA: two 8-row groups of 1024 B
        ft_mma_o(t_o, t_p + (uint32_t)(8 * i), v_lo + (uint32_t)(i * 128), v_hi, idesc_o, (j | i) ? 1u : 0u);
      umma_commit_warp(pv_done);
      umma_commit_warp(v_empty);
      done++;
    }
    // no product is in flight when tensor memory is freed
    if (scored > 0) ft_wait(s_full, (scored - 1) & 1, late);
    if (done > 0) ft_wait(pv_done, (done - 1) & 1, late);
  } else {
    // ===================== softmax / correction / epilogue: thread = query row =====================
    const int q4 = warp & 3;
    const int r = q4 * 32 + lane;
    const uint32_t lane_off = (uint32_t)(q4 * 32) << 16;
    const int qg = q0 + r;                                 // row index inside the sequence
    // m_ref is the exponent's reference point, not necessarily the running maximum: it only moves when a row's
    // maximum outgrows it by more than 2^8 (then O and l are rescaled).  The quotient O / l does not depend on the
    // reference, P just lives in [0, 256] instead of [0, 1] — and the O round trip through TMEM, with its wait for the
    // previous PV, almost never happens (with a plain running maximum some row of a warp moves in most tiles).
    float m_ref = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < nt; j++) {
      const int ph = j & 1;
      const uint32_t ts = t_s + lane_off;
      const int kv0 = first + j * FT_BN;
      const int lim = min(p.causal ? qg : len - 1, len - 1) - kv0;                 // columns > lim are masked,
      const int low = WINDOW ? qg - p.window_left - kv0 : 0;                       // and those below low
      ok = ft_wait(s_full, ph, late);
      if (!ok) break;
      tc_fence_after();
      // the whole S row in registers: four loads in flight, one wait
      uint32_t v[128];
      tmem_ld_32x32_nowait(ts, v);
      tmem_ld_32x32_nowait(ts + 32u, v + 32);
      tmem_ld_32x32_nowait(ts + 64u, v + 64);
      tmem_ld_32x32_nowait(ts + 96u, v + 96);
      tmem_ld_wait();
      // only the tiles that the ends of a row's keys fall into are masked: a comparison and a selection for each score in two passes otherwise.
      // Maximum and sum run in four chains (one was 128 dependent steps).  Three prompts of up to 2900 tokens, 32 heads on 8: 291 us (535 TFLOP/s)
      // masked everywhere and in one chain, 225 (691) so.
      const bool whole = __all_sync(0xffffffffu, lim >= FT_BN - 1 && low <= 0);
      if (!whole) {
#pragma unroll
        for (int i = 0; i < 128; i++) v[i] = (i <= lim && i >= low) ? v[i] : 0xff800000u;      // -infinity
      }
      float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 128; i++) m4[i & 3] = fmaxf(m4[i & 3], __uint_as_float(v[i]));
      float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
      mx *= p.scale_log2;                                   // (scale > 0: max commutes with the scaling)
      const bool move = (m_ref == -INFINITY) || (mx > m_ref + p.slack);
      const float m_use = move ? fmaxf(m_ref, mx) : m_ref;
      const float corr = (m_use == m_ref) ? 1.f : ex2_approx(m_ref - m_use);   // (m_ref = -inf: 0, nothing accumulated yet)
      const float msub = (m_use == -INFINITY) ? 0.f : m_use;
      if (j > 0 && __any_sync(0xffffffffu, corr != 1.f)) {
        // (S_j was issued behind the products of the tile before)
#pragma unroll 1
        for (int c0 = 0; c0 < D; c0 += 32) {
          uint32_t o[32];
          tmem_ld_32x32(t_o + lane_off + (uint32_t)c0, o);
#pragma unroll
          for (int i = 0; i < 32; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
          tmem_st_32x32(t_o + lane_off + (uint32_t)c0, o);
        }
      }
      // p = 2^(s * scale - m_use), row sum in f32, P rounded to the activation format, written over the head of S
      float r4[4] = {0.f, 0.f, 0.f, 0.f};
      auto exponentials = [&](auto all) {
#pragma unroll
        for (int c0 = 0; c0 < FT_BN; c0 += 32) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float p0 = ex2_approx(fmaf(__uint_as_float(v[c0 + i]), p.scale_log2, -msub));
            float p1 = ex2_approx(fmaf(__uint_as_float(v[c0 + i + 1]), p.scale_log2, -msub));
            if constexpr (!decltype(all)::value) {
              p0 = c0 + i <= lim && c0 + i >= low ? p0 : 0.f;
              p1 = c0 + i + 1 <= lim && c0 + i + 1 >= low ? p1 : 0.f;
            }
            r4[(i >> 1) & 3] += p0 + p1;
            if constexpr (BF) { const __nv_bfloat162 hh = __floats2bfloat162_rn(p0, p1); pk[i >> 1] = *(const uint32_t *)&hh; }
            else { const __half2 hh = __floats2half2_rn(p0, p1); pk[i >> 1] = *(const uint32_t *)&hh; }
          }
          tmem_st_x16(t_p + lane_off + (uint32_t)(c0 >> 1), pk);
        }
      };
      if (whole) exponentials(std::true_type{});
      else exponentials(std::false_type{});
      l_run = l_run * corr + ((r4[0] + r4[1]) + (r4[2] + r4[3]));
      m_ref = m_use;
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    // epilogue: O / l -> global, one row of D values per thread
    ok = ok && ft_wait(pv_done, (nt - 1) & 1, late);
    tc_fence_after();
    const float inv = (l_run > 0.f) ? 1.f / l_run : 0.f;
    uint8_t *orow = (uint8_t *)p.o + ((int64_t)(seq0 + qg) * p.o_stride + (int64_t)h * D) * 2;
#pragma unroll 1
    for (int c0 = 0; ok && c0 < D; c0 += 32) {
      uint32_t v[32];
      tmem_ld_32x32(t_o + lane_off + (uint32_t)c0, v);
      if (qg < len) {
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          uint4 pk;
          uint32_t *w = (uint32_t *)&pk;
#pragma unroll
          for (int k = 0; k < 4; k++) {
            const float a = __uint_as_float(v[i + 2 * k]) * inv, bq = __uint_as_float(v[i + 2 * k + 1]) * inv;
            if constexpr (BF) { const __nv_bfloat162 hh = __floats2bfloat162_rn(a, bq); w[k] = *(const uint32_t *)&hh; }
            else { const __half2 hh = __floats2half2_rn(a, bq); w[k] = *(const uint32_t *)&hh; }
          }
          *(uint4 *)(orow + (size_t)(c0 + i) * 2) = pk;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, FT_TCOLS);
}

}  // namespace mrs

using namespace mrs;

extern "C" int32_t *mrs_mmq_timeout_flag(void);      // mmq_ts.cu: the device's word for waits that ran out (page-locked host memory)

static uint32_t g_ft_lbo = 16384u, g_ft_sbo = 1024u;
static int g_ft_enable = 1;
// dev knobs: MN-major descriptor strides of V (bytes); enable = 0 keeps mrs_prefill_attention on prefill_attn.cu
extern "C" void mrs_prefill_attn_tc_debug(int32_t enable, uint32_t lbo, uint32_t sbo) {
  g_ft_enable = enable;
  if (lbo) g_ft_lbo = lbo;
  if (sbo) g_ft_sbo = sbo;
}

template <int D, bool BF, bool WINDOW>
static cudaError_t ft_launch_as(const CUtensorMap &tq, const CUtensorMap &tk, const CUtensorMap &tv, const FtParams &p, int batch, int max_len, cudaStream_t st) {
  const int tiles = (max_len + FT_BM - 1) / FT_BM;
  if (tiles > 65535 || batch > 65535) return cudaErrorNotSupported;
  auto kern = prefill_attn_tc_kernel<D, BF, WINDOW>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, ft_smem<D>());
  kern<<<dim3(p.H, batch, tiles), FT_THREADS, ft_smem<D>(), st>>>(tq, tk, tv, p);
  return cudaGetLastError();
}

template <int D, bool BF>
static cudaError_t ft_launch(const CUtensorMap &tq, const CUtensorMap &tk, const CUtensorMap &tv, const FtParams &p, int batch, int max_len, cudaStream_t st) {
  return p.window_left >= 0 ? ft_launch_as<D, BF, true>(tq, tk, tv, p, batch, max_len, st) : ft_launch_as<D, BF, false>(tq, tk, tv, p, batch, max_len, st);
}

// returns cudaErrorNotSupported when the call does not fit this kernel (the caller falls back to prefill_attn.cu)
extern "C" int32_t mrs_prefill_attention_tc(const void *q, const void *k, const void *v, void *out, const int32_t *cu_seqlens,
                                            int32_t batch, int32_t total_tokens, int32_t max_seqlen, int32_t num_heads,
                                            int32_t num_kv_heads, int32_t head_dim, int64_t q_stride, int64_t kv_stride,
                                            int64_t o_stride, float softmax_scale, int32_t causal, int32_t window_left,
                                            float softcap, uint32_t dtype, void *stream) {
  if (!g_ft_enable || (head_dim != 64 && head_dim != 128) || softcap > 0.f || !(softmax_scale > 0.f) || (dtype != 0 && dtype != 1))
    return (int32_t)cudaErrorNotSupported;
  if (total_tokens <= 0) return 0;
  if (num_kv_heads <= 0 || num_heads % num_kv_heads || (q_stride | kv_stride | o_stride) % 8) return (int32_t)cudaErrorNotSupported;
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)out) & 15) return (int32_t)cudaErrorNotSupported;
  if (q_stride < (int64_t)num_heads * head_dim || kv_stride < (int64_t)num_kv_heads * head_dim) return (int32_t)cudaErrorNotSupported;
  PFN_encodeTiled enc = tc_get_encode();
  int32_t *const flag = mrs_mmq_timeout_flag();
  if (enc == nullptr || flag == nullptr) return (int32_t)cudaErrorNotSupported;
  if (*(volatile const int32_t *)flag != 0) return (int32_t)cudaErrorLaunchTimeout;
  const int nb = cu_seqlens ? batch : 1, ml = cu_seqlens ? max_seqlen : total_tokens;
  auto make = [&](CUtensorMap *m, const void *base, int64_t cols, int64_t stride) -> bool {
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)total_tokens};
    const cuuint64_t strides[1] = {(cuuint64_t)stride * 2};
    const cuuint32_t box[2] = {64u, 128u};
    const cuuint32_t estr[2] = {1, 1};
    return enc(m, dtype == 1 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(base), dims,
               strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  CUtensorMap tq, tk, tv;
  if (!make(&tq, q, (int64_t)num_heads * head_dim, q_stride) || !make(&tk, k, (int64_t)num_kv_heads * head_dim, kv_stride) ||
      !make(&tv, v, (int64_t)num_kv_heads * head_dim, kv_stride))
    return (int32_t)cudaErrorNotSupported;
  FtParams p = {};
  p.o = out; p.cu_seqlens = cu_seqlens; p.T = total_tokens; p.H = num_heads; p.KVH = num_kv_heads; p.o_stride = o_stride;
  p.scale_log2 = softmax_scale * 1.4426950408889634f; p.causal = causal; p.window_left = window_left < (1 << 30) ? window_left : 1 << 30;
  // whole prompts of head size 128 let the reference stand, as they always did; head size 64 and windows follow the maximum exactly, as the
  // kernel that they ran on did (a largest probability of 1 has no rounding error: 0.00203 against 0.00208 over 3000 keys in bf16)
  p.slack = head_dim == 128 && window_left < 0 ? 8.0f : 0.0f;
  p.v_lbo = g_ft_lbo; p.v_sbo = g_ft_sbo;
  p.timeouts = flag;
  cudaStream_t st = (cudaStream_t)stream;
  if (head_dim == 128) return (int32_t)(dtype == 0 ? ft_launch<128, false>(tq, tk, tv, p, nb, ml, st) : ft_launch<128, true>(tq, tk, tv, p, nb, ml, st));
  return (int32_t)(dtype == 0 ? ft_launch<64, false>(tq, tk, tv, p, nb, ml, st) : ft_launch<64, true>(tq, tk, tv, p, nb, ml, st));
}
