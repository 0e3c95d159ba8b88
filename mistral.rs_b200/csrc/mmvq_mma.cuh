// mmvq_mma.cuh — streaming GEMV of mmvq.cu for three (Q8_0: five) to eight rows of Q8_1 activations over large matrices: integer products on the tensor
// cores (mma.sync m16n8k32 / m16n8k16, s8).
//
// The vector kernel's dot products, and its reads of the activations from shared memory, grow with the rows: Q4_K 14336 x 4096 took 12 us for
// one row, 19 for four, 30 for eight, 5 of them HBM.  Here sixteen weight rows are the M of a product, the activation rows its N: one
// instruction does the 4096 integer products of a Q8_1 block, and what is left per block (unpacking, scales) does not depend on the rows.
// (Every block of 32 has scales of its own, so its results are needed at once: in registers here, where tcgen05's would be read back from
// tensor memory, behind a product that takes 50 clocks for up to 96 columns.)
// The arithmetic is the vector kernel's (Q8_1 blocks, exact integer dots, f32 scales); only the order of the f32 sums differs.
//
// Same frame: a producer warp streams row segments with cp.async.bulk into a ring, eight consumer warps.  A pass is sixteen rows (eight gate
// and eight up rows for GLU); a warp takes every eighth 256-wide stretch of K of all sixteen, and the eight partial tiles meet in shared
// memory at the end of a pass, in warp order.  Included by mmvq.cu.
#pragma once
#include <type_traits>

namespace mrs {

constexpr int MV_STRETCH = 8;        // stretches of 256 k in a stage: one a warp
template <int T> struct MvFmt { static constexpr bool ok = false; };
template <> struct MvFmt<MRS_Q4_K> { static constexpr bool ok = true; static constexpr int BYTES = 144, PITCH = MV_STRETCH * 144 + 32; };
template <> struct MvFmt<MRS_Q5_K> { static constexpr bool ok = true; static constexpr int BYTES = 176, PITCH = MV_STRETCH * 176 + 32; };
template <> struct MvFmt<MRS_Q6_K> { static constexpr bool ok = true; static constexpr int BYTES = 210, PITCH = MV_STRETCH * 210 + 32 + 96; };
template <> struct MvFmt<MRS_Q8_0> { static constexpr bool ok = true; static constexpr int BYTES = 272, PITCH = MV_STRETCH * 272 + 32 + 64; };
// (pitches: 32 modulo 128 where a lane reads 8 aligned bytes, 16 modulo 32 where it reads words; room for 30 bytes of phase and over-read)
static_assert(MvFmt<MRS_Q4_K>::PITCH % 128 == 32 && MvFmt<MRS_Q5_K>::PITCH % 128 == 32, "bank conflicts");
static_assert(MvFmt<MRS_Q6_K>::PITCH % 16 == 0 && MvFmt<MRS_Q8_0>::PITCH % 16 == 0, "bulk copies");

__device__ __forceinline__ void mv_mma32(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void mv_mma16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b) {
  asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(b), "r"(0));
}
__device__ __forceinline__ uint2 mv_lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ float4 mv_ldsf4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}
// By the whole warp, with a limit.  A wait that runs out is reported, and the warp goes through its part without waiting again (and without a result).
constexpr uint32_t MV_WAIT_LIMIT = 1u << 22;
__device__ __forceinline__ void mv_wait(uint64_t *bar, uint32_t parity, bool &dead, int *timeouts) {
  if (!mbar_wait_warp(bar, parity, dead ? 1u : MV_WAIT_LIMIT)) {
    dead = true;
    *(volatile int *)timeouts = 1;
  }
}
// Copies in flight land before a CTA may end: the last of `n` stages, where a wait has run out.  (Out of line: in the consumers' code it cost launches
// of four rows 1 %.)
__device__ __noinline__ void mv_land(uint64_t *full, int n, int nst, int *timeouts) {
  for (int i = max(0, n - nst); i < n; i++) { bool gone = false; mv_wait(&full[i % nst], (i / nst) & 1, gone, timeouts); }
}
// the word at a 2-byte aligned shared address
__device__ __forceinline__ uint32_t mv_word(uint32_t a) {
  const uint32_t w = a & ~3u;
  return __funnelshift_r(lds32(w), lds32(w + 4u), (a & 2u) * 8u);
}

// Lane (g, t) = (lane / 4, lane % 4) of a product holds rows g and g + 8 of the weights, column g of the activations and columns 2 t, 2 t + 1
// of both rows' results.  Which k stand in which slot is free as long as both operands agree: a lane takes bytes 8 t .. 8 t + 7 of a block of
// 32 (k32), or 4 t .. 4 t + 3 of a block of 16 (k16).
// x: the activations' int8 at column g, k 0 of the stretch; ds: (d, d * sum) of columns 2 t, 2 t + 1 of the stretch's first block, `step` bytes
// a block.  w0, w1: the stretch in rows g and g + 8.  acc[0..3]: (g, 2 t), (g, 2 t + 1), (g + 8, 2 t), (g + 8, 2 t + 1).
template <int T> struct MvStretch;

template <bool FIVE> struct MvK45 {
  __device__ static __forceinline__ void run(uint32_t w0, uint32_t w1, uint32_t x, uint32_t ds, uint32_t step, int t, float (&acc)[4]) {
    const uint4 h0 = lds128(w0), h1 = lds128(w1);
    // six-bit scales and minima of the eight blocks, a byte each
    auto bytes = [](const uint4 &h, uint32_t &s03, uint32_t &s47, uint32_t &m03, uint32_t &m47) {
      s03 = h.y & 0x3F3F3F3Fu; m03 = h.z & 0x3F3F3F3Fu;
      s47 = (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
      m47 = ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
    };
    uint32_t s[2][2], m[2][2];
    bytes(h0, s[0][0], s[0][1], m[0][0], m[0][1]);
    bytes(h1, s[1][0], s[1][1], m[1][0], m[1][1]);
    uint2 q0 = make_uint2(0u, 0u), q1 = q0, f0 = q0, f1 = q0;      // FIVE: the fifth bits
    if constexpr (FIVE) { f0 = mv_lds64(w0 + 16u + 8u * t); f1 = mv_lds64(w1 + 16u + 8u * t); }
    float sum[4] = {0.f, 0.f, 0.f, 0.f}, low[4] = {0.f, 0.f, 0.f, 0.f};
    auto block = [&](auto bc) {
      constexpr int b = decltype(bc)::value, r = b >> 2, e = b & 3;
      if constexpr ((b & 1) == 0) {
        const uint32_t at = (FIVE ? 48u : 16u) + 16u * b + 8u * t;
        q0 = mv_lds64(w0 + at); q1 = mv_lds64(w1 + at);
      }
      constexpr int sh = 4 * (b & 1);
      uint32_t a[4] = {(q0.x >> sh) & 0x0F0F0F0Fu, (q1.x >> sh) & 0x0F0F0F0Fu, (q0.y >> sh) & 0x0F0F0F0Fu, (q1.y >> sh) & 0x0F0F0F0Fu};
      if constexpr (FIVE) {
        constexpr int up = b < 4 ? 4 - b : 0, down = b > 4 ? b - 4 : 0;      // bit b of each byte to bit 4
        a[0] |= ((f0.x << up) >> down) & 0x10101010u; a[1] |= ((f1.x << up) >> down) & 0x10101010u;
        a[2] |= ((f0.y << up) >> down) & 0x10101010u; a[3] |= ((f1.y << up) >> down) & 0x10101010u;
      }
      const uint2 y = mv_lds64(x + 32u * b);
      const float4 d = mv_ldsf4(ds + step * b);
      int c[4];
      mv_mma32(c, a, y.x, y.y);
      const int s0 = (int)((s[0][r] >> 8 * e) & 0xFFu), s1 = (int)((s[1][r] >> 8 * e) & 0xFFu);
      const float m0 = (float)(int)((m[0][r] >> 8 * e) & 0xFFu), m1 = (float)(int)((m[1][r] >> 8 * e) & 0xFFu);
      // (32 x 31 x 128 x 63 < 2^23: exact.  Conversions by additions to 1.5 x 2^23 in their place, which run at a higher rate, were no faster.)
      sum[0] = fmaf(d.x, (float)(c[0] * s0), sum[0]); sum[1] = fmaf(d.z, (float)(c[1] * s0), sum[1]);
      sum[2] = fmaf(d.x, (float)(c[2] * s1), sum[2]); sum[3] = fmaf(d.z, (float)(c[3] * s1), sum[3]);
      low[0] = fmaf(d.y, m0, low[0]); low[1] = fmaf(d.w, m0, low[1]);
      low[2] = fmaf(d.y, m1, low[2]); low[3] = fmaf(d.w, m1, low[3]);
    };
    block(std::integral_constant<int, 0>{}); block(std::integral_constant<int, 1>{}); block(std::integral_constant<int, 2>{});
    block(std::integral_constant<int, 3>{}); block(std::integral_constant<int, 4>{}); block(std::integral_constant<int, 5>{});
    block(std::integral_constant<int, 6>{}); block(std::integral_constant<int, 7>{});
    const float2 e0 = __half22float2(*(const __half2 *)&h0.x), e1 = __half22float2(*(const __half2 *)&h1.x);
    acc[0] += e0.x * sum[0] - e0.y * low[0]; acc[1] += e0.x * sum[1] - e0.y * low[1];
    acc[2] += e1.x * sum[2] - e1.y * low[2]; acc[3] += e1.x * sum[3] - e1.y * low[3];
  }
};
template <> struct MvStretch<MRS_Q4_K> : MvK45<false> {};
template <> struct MvStretch<MRS_Q5_K> : MvK45<true> {};

template <> struct MvStretch<MRS_Q6_K> {   // ql[128] | qh[64] | scales[16] | d
  __device__ static __forceinline__ void run(uint32_t w0, uint32_t w1, uint32_t x, uint32_t ds, uint32_t step, int t, float (&acc)[4]) {
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int n = 0; n < 2; n++) {
      uint32_t hi[2][2], lo[2][2][2];      // [row][sixteen of the 32], and [32 of the 64] before that
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const uint32_t at = 128u + 32u * n + 16u * h + 4u * t;
        hi[0][h] = mv_word(w0 + at); hi[1][h] = mv_word(w1 + at);
#pragma unroll
        for (int k = 0; k < 2; k++) {
          const uint32_t al = 64u * n + 32u * k + 16u * h + 4u * t;
          lo[0][k][h] = mv_word(w0 + al); lo[1][k][h] = mv_word(w1 + al);
        }
      }
      const uint32_t s[2][2] = {{mv_word(w0 + 192u + 8u * n), mv_word(w0 + 196u + 8u * n)}, {mv_word(w1 + 192u + 8u * n), mv_word(w1 + 196u + 8u * n)}};
      auto block = [&](auto qc) {
        constexpr int q = decltype(qc)::value;
        const float4 d = mv_ldsf4(ds + step * (4 * n + q));
        int v[4];
        auto sixteen = [&](auto hc) {
          constexpr int h = decltype(hc)::value;
          uint32_t a[2];
#pragma unroll
          for (int r = 0; r < 2; r++) {
            const uint32_t up = q < 2 ? hi[r][h] << (4 - 2 * q) : hi[r][h] >> (2 * q - 4);      // bits 2 q, 2 q + 1 to bits 4, 5
            const uint32_t u = ((lo[r][q & 1][h] >> (4 * (q >> 1))) & 0x0F0F0F0Fu) | (up & 0x30303030u);
            a[r] = ((u | 0x80808080u) - 0x20202020u) ^ 0x80808080u;                                // u - 32 in each byte
          }
          int c[4];
          mv_mma16(c, a[0], a[1], lds32(x + (uint32_t)(128 * n + 32 * q + 16 * h)));
          constexpr int e = 8 * (2 * (q & 1) + h);
          const int s0 = (int)(int8_t)(s[0][q >> 1] >> e), s1 = (int)(int8_t)(s[1][q >> 1] >> e);
          if constexpr (h == 0) { v[0] = c[0] * s0; v[1] = c[1] * s0; v[2] = c[2] * s1; v[3] = c[3] * s1; }
          else { v[0] += c[0] * s0; v[1] += c[1] * s0; v[2] += c[2] * s1; v[3] += c[3] * s1; }
        };
        sixteen(std::integral_constant<int, 0>{}); sixteen(std::integral_constant<int, 1>{});
        // (2 x 16 x 32 x 127 x 128 < 2^24: exact)
        sum[0] = fmaf(d.x, (float)v[0], sum[0]); sum[1] = fmaf(d.z, (float)v[1], sum[1]);
        sum[2] = fmaf(d.x, (float)v[2], sum[2]); sum[3] = fmaf(d.z, (float)v[3], sum[3]);
      };
      block(std::integral_constant<int, 0>{}); block(std::integral_constant<int, 1>{});
      block(std::integral_constant<int, 2>{}); block(std::integral_constant<int, 3>{});
    }
    const float d0 = half_bits_to_float(lds_u16s(w0 + 208u)), d1 = half_bits_to_float(lds_u16s(w1 + 208u));
    acc[0] += d0 * sum[0]; acc[1] += d0 * sum[1]; acc[2] += d1 * sum[2]; acc[3] += d1 * sum[3];
  }
};

template <> struct MvStretch<MRS_Q8_0> {   // eight blocks of d | qs[32]
  __device__ static __forceinline__ void run(uint32_t w0, uint32_t w1, uint32_t x, uint32_t ds, uint32_t step, int t, float (&acc)[4]) {
#pragma unroll
    for (int b = 0; b < 8; b++) {
      const uint32_t at = 34u * b + 2u + 8u * t;
      uint32_t a[4];
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const uint32_t p = (r ? w1 : w0) + at, w = p & ~3u, sh = (p & 2u) * 8u;
        const uint32_t v0 = lds32(w), v1 = lds32(w + 4u), v2 = lds32(w + 8u);
        a[r] = __funnelshift_r(v0, v1, sh); a[2 + r] = __funnelshift_r(v1, v2, sh);
      }
      const uint2 y = mv_lds64(x + 32u * b);
      const float4 d = mv_ldsf4(ds + step * b);
      int c[4];
      mv_mma32(c, a, y.x, y.y);
      const float d0 = half_bits_to_float(lds_u16s(w0 + 34u * b)), d1 = half_bits_to_float(lds_u16s(w1 + 34u * b));
      acc[0] = fmaf(d0 * d.x, (float)(c[0]), acc[0]); acc[1] = fmaf(d0 * d.z, (float)(c[1]), acc[1]);
      acc[2] = fmaf(d1 * d.x, (float)(c[2]), acc[2]); acc[3] = fmaf(d1 * d.z, (float)(c[3]), acc[3]);
    }
  }
};

// lanes read words 4 t of sixteen (k16) or 8 bytes 8 t of 32 (k32) of a column
template <int T> __device__ __forceinline__ uint32_t mv_x_lane(int t) { return T == MRS_Q6_K ? 4u * t : 8u * t; }

template <int T, int NC>
__global__ void __launch_bounds__(9 * 32, 2) mmvq_mma_kernel(const MmvqParams p) {
  using F = MvFmt<T>;
  constexpr int NCW = 8, SLOTS = 16, PITCH = F::PITCH, STAGE = SLOTS * PITCH;
  extern __shared__ __align__(128) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_st = p.K / 256, nseg = (n_st + MV_STRETCH - 1) / MV_STRETCH, row_bytes = n_st * F::BYTES, nst = p.nstages;
  const int xp = p.K + 32;                                            // bytes of a column
  // [barriers 256 B][columns][(d, d sum) a block and column][partial tiles, two passes][ring]
  uint64_t *full = (uint64_t *)smem, *empty = full + MAX_STAGES;
  uint8_t *xq = smem + 256;
  float2 *xd = (float2 *)(xq + NC * xp);
  float *red = (float *)((uint8_t *)xd + (size_t)p.K / 32 * NC * 8);
  const uint32_t ring = smem_u32(red) + 2u * NCW * 128u * 4u;
  if (tid == 0) {
    for (int i = 0; i < nst; i++) { mbar_init(&full[i], 32); mbar_init(&empty[i], NCW); }
    fence_mbar_init();
  }
  __syncthreads();
  const int vr0 = (int)((long long)p.vrows * blockIdx.x / gridDim.x), vr1 = (int)((long long)p.vrows * (blockIdx.x + 1) / gridDim.x);
  const int P = p.mode == MODE_GLU ? SLOTS / 2 : SLOTS;               // virtual rows of a pass

  if (warp == NCW) {
    // ===================== producer: lane = slot; weights do not wait for the grid before =====================
    if (p.pdl) pdl_launch_dependents();
    int stage = 0, phase = 0, n = 0;
    bool dead = false;
    for (int base = vr0; base < vr1 && !dead; base += P) {
      const uint8_t *rowp = nullptr;
      if (lane < SLOTS) {
        const int vrow = p.mode == MODE_GLU ? base + (lane & 7) : base + lane;
        if (vrow < vr1) {
          int m, row;
          resolve_row(p, vrow, lane >> 3, m, row);
          rowp = p.w[m] + (size_t)row * row_bytes;
        }
      }
      for (int s = 0; s < nseg; s++) {
        // (stages come free once the consumers have their activations: a limit does not count the grids before this one)
        if (p.pdl && n == nst) pdl_wait();
        mv_wait(&empty[stage], phase ^ 1, dead, p.timeouts);
        if (dead) break;
        n++;
        if (rowp != nullptr) {
          const uintptr_t a = (uintptr_t)(rowp + s * (MV_STRETCH * F::BYTES)), a0 = a & ~(uintptr_t)15;
          const int len = min(MV_STRETCH * F::BYTES, row_bytes - s * (MV_STRETCH * F::BYTES));
          const uint32_t bytes = (uint32_t)(((a + len + 15) & ~(uintptr_t)15) - a0);
          mbar_arrive_expect_tx(&full[stage], bytes);
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                           ring + (uint32_t)(stage * STAGE + lane * PITCH)),
                       "l"(a0), "r"(bytes), "r"(smem_u32(&full[stage]))
                       : "memory");
        } else {
          mbar_arrive(&full[stage]);
        }
        if (++stage == nst) { stage = 0; phase ^= 1; }
      }
    }
    if (dead) mv_land(full, n, nst, p.timeouts);      // (otherwise the consumers wait for the last copies, or see to them where their own wait ran out)
    return;
  }

  // ===================== consumers =====================
  if (p.pdl) pdl_wait();
  // Q8_1 rows into columns of int8 and (d, d * sum of the int8)
  {
    const block_q8_1 *y = (const block_q8_1 *)p.x;
    const int nb = p.K / 32;
    for (int i = tid; i < nb * NC; i += NCW * 32) {
      const int col = i / nb, b = i - col * nb;
      uint32_t q[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
      float d = 0.f;
      int n = 0;
      if (col < p.ncols) {
        const block_q8_1 *yb = y + (size_t)col * p.stride_col_y + b;
#pragma unroll
        for (int k = 0; k < 8; k++) { q[k] = *(const uint32_t *)(yb->qs + 4 * k); n = __dp4a((int)q[k], 0x01010101, n); }
        d = __low2float(yb->ds);
      }
      uint4 *to = (uint4 *)(xq + col * xp + 32 * b);
      to[0] = make_uint4(q[0], q[1], q[2], q[3]); to[1] = make_uint4(q[4], q[5], q[6], q[7]);
      xd[b * NC + col] = make_float2(d, d * (float)n);
    }
  }
  asm volatile("bar.sync 1, %0;" ::"n"(NCW * 32));

  const int g = lane >> 2, t = lane & 3;
  // (columns past NC repeat others; their results are not stored)
  const uint32_t xl = smem_u32(xq) + (uint32_t)((g & (NC - 1)) * xp) + mv_x_lane<T>(t), dl = smem_u32(xd) + 16u * (uint32_t)(t & (NC / 2 - 1));
  int stage = 0, phase = 0, buf = 0;
  bool dead = false;
  for (int base = vr0; base < vr1; base += P, buf ^= 1) {
    uint32_t ph[2];                          // where rows g and g + 8 start in their 16-byte aligned copies
#pragma unroll
    for (int r = 0; r < 2; r++) {
      int vrow = p.mode == MODE_GLU ? base + g : base + g + 8 * r, m, row;
      if (vrow >= vr1) vrow = vr1 - 1;
      resolve_row(p, vrow, r, m, row);
      ph[r] = (uint32_t)((uintptr_t)(p.w[m] + (size_t)row * row_bytes) & 15);
    }
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int s = 0; s < nseg; s++) {
      mv_wait(&full[stage], phase, dead, p.timeouts);
      const int k = s * MV_STRETCH + warp;
      if (k < n_st) {
        const uint32_t st = ring + (uint32_t)(stage * STAGE + g * PITCH), sp = (uint32_t)(s * (MV_STRETCH * F::BYTES)) & 15u;
        MvStretch<T>::run(st + ((ph[0] + sp) & 15u) + (uint32_t)(warp * F::BYTES), st + 8u * PITCH + ((ph[1] + sp) & 15u) + (uint32_t)(warp * F::BYTES),
                          xl + 256u * (uint32_t)k, dl + (uint32_t)(k * 8 * NC * 8), NC * 8u, t, acc);
      }
      __syncwarp();
      // (a warp whose wait ran out gives no stage back: its copies may be on their way still, and the producer's own wait ends that part)
      if (lane == 0 && !dead) mbar_arrive(&empty[stage]);
      if (++stage == nst) { stage = 0; phase ^= 1; }
    }
    // partial tiles [warp][row][8 columns]; NaN where a wait ran out, and so in every sum that lacks the tile
    if (dead) acc[0] = acc[1] = acc[2] = acc[3] = __int_as_float(0x7fffffff);
    float *mine = red + (size_t)(buf * NCW + warp) * 128;
    *(float2 *)(mine + g * 8 + 2 * t) = make_float2(acc[0], acc[1]);
    *(float2 *)(mine + (g + 8) * 8 + 2 * t) = make_float2(acc[2], acc[3]);
    asm volatile("bar.sync 1, %0;" ::"n"(NCW * 32));      // (the next pass writes the other buffer: nobody overtakes a reader)
    auto total = [&](int row, int col) {
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < NCW; w++) v += red[(size_t)(buf * NCW + w) * 128 + row * 8 + col];
      return v;
    };
    if (p.mode == MODE_GLU) {
      const int row = tid >> 3, col = tid & 7, vrow = base + row;
      if (row < 8 && col < p.ncols && vrow < vr1) {
        // gate and up rounded to the output type first, activation in f32, product in that type — REF mmvq_gguf.cu:866-870
        const float a = round_act(total(row, col), p.dst_dtype), b = round_act(total(row + 8, col), p.dst_dtype);
        store_act(p.dst[0], (int64_t)col * p.stride_col_dst + vrow, round_act(glu_activation(a, p.activation), p.dst_dtype) * b, p.dst_dtype);
      }
    } else {
      const int row = tid & 15, col = tid >> 4, vrow = base + row;
      if (col < p.ncols && vrow < vr1) {
        int m, r;
        resolve_row(p, vrow, 0, m, r);
        const int64_t at = (int64_t)col * (p.mode == MODE_QKV ? p.nrows[m] : p.stride_col_dst) + r;
        float v = total(row, col);
        if (p.residual != nullptr) v = round_act(v, p.dst_dtype) + load_act(p.residual, at, p.dst_dtype);      // (rounded, then added: as the vector kernel)
        store_act(p.dst[m], at, v, p.dst_dtype);
      }
    }
  }
  if (dead) mv_land(full, (vr1 - vr0 + P - 1) / P * nseg, nst, p.timeouts);
}

}  // namespace mrs
