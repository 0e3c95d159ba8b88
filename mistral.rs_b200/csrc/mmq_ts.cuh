// mmq_ts.cuh — GEMM over ggml quant blocks for more rows than the vector kernels take: swap-AB, A operand in tensor memory.
//
// Y[M,N] = X[M,K] . W[N,K]^T, W in raw ggml blocks of any of the ten types, X / Y 16-bit, f32 accumulate (replaces REF
// mistralrs-quant/src/gguf/fast_mmq.rs:762-826 `fast_mmq::plain`).  The WEIGHT rows are the UMMA M dimension (128 rows = 128 TMEM
// lanes), the tokens the N dimension (16 .. 256): the dequantised tile is the A operand, which tcgen05.mma reads from tensor
// memory, so nothing of it passes through shared memory.  One CTA per SM, 24 warps:
//   warp 0 (and 3)  raw blocks -> shared memory, one span of 256 k of 128 rows per stage: one TMA box where rows are multiples of
//                   16 bytes, else 16-byte cp.async of both warps (a TMA row stride has to be a multiple of 16 bytes)
//   warp 2          X tiles [tokens x 64 k] by TMA, SWIZZLE_128B
//   warps 4..19     dequantisers: thread = (weight row, 64 consecutive k of the span): the thread reads its blocks' bytes once,
//                   16 bytes at a time, and writes 16-bit pairs with tcgen05.st (lane = row, two consecutive k per 32-bit column)
//   warp 1          MMA issuer: 16 x tcgen05.mma M=128 N=tokens K=16 per span, accumulators and two A stages in tensor memory
//   warps 20..23    epilogue, beside the products of the CTA's next tile
// Two modes: K whole (persistent CTAs walk the output tiles, row tiles innermost: the CTAs that run at one time read the same X tile), or K split
// over a cluster of 2 .. 8 CTAs whose partial tiles meet through distributed shared memory: each CTA sums a share of the tokens, in
// rank order, so results do not depend on timing.  ts_plan chooses mode, token tile and split.
//
// Numerics: every weight is dequantised with the reference's f32 formula and rounded once to the activation format; activations are
// used as they are; f32 accumulation in tensor memory, in k order (K whole: bit for bit csrc/mmq_tc.cu).
// What bounds it: the dequantisers' issue slots (some 5300 warp instructions a span for Q4_K, 4400 for Q8_0) up to about 130 tokens a tile,
// then the tensor pipe and the power limit.  The issuer must not be the bound: with its operands in ordinary registers sixteen products took
// 1900 clocks beside the dequantisers, with a warp index that the compiler knows to be uniform 500.  Measured on one B200, us before and
// after (before: one kernel for Q8_0, Q4_K and Q6_K with 128 or 256 tokens a tile and K whole, per-element decoding for the other types,
// a kernel with 8 dequantising warps for int4): Q4_K 14336 x 4096, 24 tokens 29.3 / 18.4; Q5_K 4096 x 4096, 200 tokens 2517 / 18.5; Q8_0
// 14336 x 4096, 4096 tokens 475 / 418; int4 14336 x 4096, 32 tokens 21.9 / 16.5; int4 with zero points 4096 x 14336, 500 tokens 170 / 61.5.
// Every wait has a limit; one that runs out ends the CTA and sets a word in host memory, after which the entry points refuse every call
// on that device with cudaErrorLaunchTimeout (the word itself: mrs_mmq_timeout_flag, mrs_mmq_timeouts).  That launch's output is not valid:
// a tile may be missing, or with K split lack a rank's part (telling the other ranks cost every split launch 1 to 6 %).  What a limit counts is this grid's
// own work: in a programmatic-dependent-launch chain a warp passes pdl_wait before its first wait that the activations hold up.
#pragma once
#include "dequant.cuh"
#include "tc_common.cuh"

#include <stdio.h>
#include <type_traits>

namespace mrs {

constexpr int TS_BM = 128;                 // weight rows per tile (UMMA M, TMEM lanes)
constexpr int TS_SPAN_K = 256;             // k per raw stage and per A stage
constexpr int TS_XK = 64;                  // k per X tile (one SWIZZLE_128B atom row)
constexpr int TS_AS = 2;                   // A stages in tensor memory, 128 columns each, behind 256 accumulator columns
constexpr int TS_RS_MAX = 12, TS_XS_MAX = 8;
constexpr int TS_DQ_WARPS = 16, TS_EPI_WARPS = 4;
constexpr int TS_THREADS = 32 * (4 + TS_DQ_WARPS + TS_EPI_WARPS);
constexpr int TS_N_BARS = 2 * TS_RS_MAX + 2 * TS_XS_MAX + 2 * TS_AS + 4 + 1;
constexpr int TS_SMEM_MAX = 226 * 1024;
constexpr uint32_t TS_WAIT_LIMIT = 1u << 22;

struct TsParams {
  const uint8_t *w;
  void *y;
  int *timeouts;
  int M, N, K, row_bytes;
  int nt, tiles_m, tiles_n;   // tokens per tile (multiple of 16), tiles
  int ksplit;                 // CTAs of a cluster that share K
  int rs, xs, xb;             // depths of the raw and the X ring; 64-k tiles of an X stage
  // int4 checkpoints: w in tiles [K/64][N][32 B] (csrc/w4a16.cu), scales [K/group][N]
  const uint8_t *scales;
  const uint8_t *qzeros;      // AWQ [K/group][N/8] words, or null: zero point 8
  int group32, group_shift;   // weights of a group / 32, and its logarithm or -1
  int scale_perm;             // columns 0 plain, 1 / 2 Marlin-permuted 64 / 32 wide
  int pdl;                    // link of a programmatic-dependent-launch chain: x comes from, y may be read by, the grid before
};
// (eight bytes more, and every launch took the host 0.3 us longer)
static_assert(sizeof(TsParams) <= 104, "parameters of a launch");

// block types of int4 checkpoints: scales in the activation format, and in the other 16-bit format (f16 scales of bf16 rows, bf16 scales of f16 rows),
// rounded as they are read (4096 x 14336, 500 tokens: 54.6 us behind a launch that casts them, 50.5 so).  A type of its own: asked for at run time in the
// inner loop the format cost every int4 call up to 1 % (14336 x 4096 at 32 tokens 15.31 us, 15.21 without; 4096 x 14336 at 500 49.5, 49.0).
constexpr int TS_INT4 = 200, TS_INT4_OTHER = 201;
constexpr bool ts_is_int4(int type) { return type == TS_INT4 || type == TS_INT4_OTHER; }
// SPAN: bytes of 256 weights of a row; PITCH: of a row in a raw stage, an odd multiple of 16 (16-byte reads of 8 consecutive rows
// then fall on distinct banks) that also holds the bytes in front of and behind an unaligned span
template <int TYPE> struct TsFmt;
template <> struct TsFmt<MRS_Q4_0> { static constexpr int SPAN = 144, PITCH = 176; };
template <> struct TsFmt<MRS_Q4_1> { static constexpr int SPAN = 160, PITCH = 176; };
template <> struct TsFmt<MRS_Q5_0> { static constexpr int SPAN = 176, PITCH = 208; };
template <> struct TsFmt<MRS_Q5_1> { static constexpr int SPAN = 192, PITCH = 208; };
template <> struct TsFmt<MRS_Q8_0> { static constexpr int SPAN = 272, PITCH = 304; };
template <> struct TsFmt<MRS_Q2_K> { static constexpr int SPAN = 84, PITCH = 112; };
template <> struct TsFmt<MRS_Q3_K> { static constexpr int SPAN = 110, PITCH = 144; };
template <> struct TsFmt<MRS_Q4_K> { static constexpr int SPAN = 144, PITCH = 144; };
template <> struct TsFmt<MRS_Q5_K> { static constexpr int SPAN = 176, PITCH = 176; };
template <> struct TsFmt<MRS_Q6_K> { static constexpr int SPAN = 210, PITCH = 240; };
// where rows and spans are multiples of 16 bytes nothing lies in front of a span, so a shorter pitch serves
template <int TYPE, bool ALIGNED> struct TsPitch { static constexpr int value = TsFmt<TYPE>::PITCH; };
template <> struct TsPitch<MRS_Q4_0, true> { static constexpr int value = 144; };
template <> struct TsPitch<MRS_Q5_0, true> { static constexpr int value = 176; };
template <> struct TsPitch<MRS_Q8_0, true> { static constexpr int value = 272; };
// int4 tiles: four chunks of [128 rows][32 B], then up to 8 rows of 128 scales (groups of 32 at least) and 8 of 16 zero-point words
template <> struct TsFmt<TS_INT4> { static constexpr int SPAN = 0, PITCH = 32; };
template <> struct TsFmt<TS_INT4_OTHER> : TsFmt<TS_INT4> {};
constexpr int TS_I4_CHUNK = TS_BM * 32, TS_I4_SCALES = 4 * TS_I4_CHUNK, TS_I4_ZEROS = TS_I4_SCALES + 8 * TS_BM * 2, TS_I4_STAGE = TS_I4_ZEROS + 8 * 64;
template <int TYPE, bool ALIGNED> struct TsStage { static constexpr int BYTES = TS_BM * TsPitch<TYPE, ALIGNED>::value; };
template <> struct TsStage<TS_INT4, true> { static constexpr int BYTES = TS_I4_STAGE; };
template <> struct TsStage<TS_INT4_OTHER, true> : TsStage<TS_INT4, true> {};

// By the whole warp.  False when the phase did not complete within the limit: the caller then ends its part of the CTA.  (The issuer and the producers
// pass several waits in a span: 2 to 5 % of a launch lies between this loop and one that leaves PTX to vote in each round: Q5_K 4096 x 4096, 200
// tokens in a graph 17.5 us and 18.3, int4 14336 x 4096, 32 tokens 15.3 and 16.1.)
__device__ __forceinline__ bool ts_wait(uint64_t *bar, uint32_t parity, int *timeouts) {
  if (mbar_wait_warp(bar, parity, TS_WAIT_LIMIT)) return true;
  *(volatile int *)timeouts = 1;
  return false;
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}
__device__ __forceinline__ float ts_h2f(uint32_t bits) { return __half2float(__ushort_as_half((unsigned short)bits)); }
template <bool BF> __device__ __forceinline__ uint32_t ts_pack(float lo, float hi) {
  if constexpr (BF) { const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi); return *(const uint32_t *)&h; }
  else { const __half2 h = __floats2half2_rn(lo, hi); return *(const uint32_t *)&h; }
}
// a = v.lo * d + c, b = v.hi * d + c: f16 times f16 (the low half of d) plus f32, rounded once
__device__ __forceinline__ void ts_mix(uint32_t v, uint32_t d, float c, float &a, float &b) {
  asm("{\n\t.reg .f16 lo, hi, s, t;\n\tmov.b32 {lo, hi}, %2;\n\tmov.b32 {s, t}, %3;\n\t"
      "fma.rn.f32.f16 %0, lo, s, %4;\n\tfma.rn.f32.f16 %1, hi, s, %4;\n\t}" : "=f"(a), "=f"(b) : "r"(v), "r"(d), "f"(c));
}
__device__ __forceinline__ uint32_t ts_hfma2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ uint32_t ts_hsub2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t ts_hmul2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// integer as f16, in both halves
__device__ __forceinline__ uint32_t ts_int2(int v) { return (uint32_t)__half_as_ushort(__int2half_rn(v)) * 0x00010001u; }
// (w & MASK) | 0x6400 0x6400: fields of up to ten bits on 1024 as f16, one instruction
template <uint32_t MASK> __device__ __forceinline__ uint32_t ts_field(uint32_t w) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, 0x64006400, 0xea;" : "=r"(d) : "r"(w), "n"(MASK));
  return d;
}
__device__ __forceinline__ uint32_t ts_or_masked(uint32_t w, uint32_t mask, uint32_t acc) {   // (w & mask) | acc
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xea;" : "=r"(d) : "r"(w), "r"(mask), "r"(acc));
  return d;
}

// Four weights from the f16 pairs e02 = 1024 + (q0, q2), e13 = 1024 + (q1, q3), rounded once to 16 bits as the f32 formula is: what
// has to be exact in f16 or f32 on the way is.  Byte permutations, conversions, logic and shifts run at 64 lanes a clock, f16 x f16 +
// f32 at 128: taking two quants a logic operation and converting them inside the product leaves about 1.1 of the slow kind a weight,
// where a permutation, a subtraction and a conversion each took 1.75.
//
// d * (sc * q) + c, sc * q an f16 (sc q < 2048, and 1024 sc an f16): sc2 and off2 = -1024 sc in both halves
template <bool BF> __device__ __forceinline__ void ts_scaled4(uint32_t e02, uint32_t e13, uint32_t sc2, uint32_t off2, uint32_t d, float c, uint32_t *o) {
  float v0, v1, v2, v3;
  ts_mix(ts_hfma2(e02, sc2, off2), d, c, v0, v2);
  ts_mix(ts_hfma2(e13, sc2, off2), d, c, v1, v3);
  o[0] = ts_pack<BF>(v0, v1); o[1] = ts_pack<BF>(v2, v3);
}
// d * (1024 + q) + c = d (q - OFF) exactly (c = -(1024 + OFF) d), then times the integer sc in f32: rounds as (d sc) * (q - OFF) does
template <bool BF> __device__ __forceinline__ void ts_times4(uint32_t e02, uint32_t e13, uint32_t d, float c, float sc, uint32_t *o) {
  float v0, v1, v2, v3;
  ts_mix(e02, d, c, v0, v2);
  ts_mix(e13, d, c, v1, v3);
  o[0] = ts_pack<BF>(v0 * sc, v1 * sc); o[1] = ts_pack<BF>(v2 * sc, v3 * sc);
}
// bytes of t (quants on OFF) as consecutive pairs: d * (q - OFF), c = -(1024 + OFF) d.  f16 results take two f16 instructions:
// 1024 + q is an f16, so is q - OFF, and an integer of 8 bits times 11 bits rounds once, as the f32 product rounded to f16 does
template <int OFF, bool BF> __device__ __forceinline__ void ts_bytes4(uint32_t t, uint32_t d, float c, uint32_t *o) {
  const uint32_t p = prmt(t, 0x64646464u, 0x4140u), q = prmt(t, 0x64646464u, 0x4342u);
  if constexpr (BF) {
    float v0, v1, v2, v3;
    ts_mix(p, d, c, v0, v1);
    ts_mix(q, d, c, v2, v3);
    o[0] = ts_pack<BF>(v0, v1); o[1] = ts_pack<BF>(v2, v3);
  } else {
    const uint32_t off = 0x64006400u + (uint32_t)OFF * 0x00010001u, d2 = d * 0x00010001u;
    o[0] = ts_hmul2(ts_hsub2(p, off), d2);
    o[1] = ts_hmul2(ts_hsub2(q, off), d2);
  }
}
// bytes of t (quants) as consecutive pairs: d * q + m
template <bool BF> __device__ __forceinline__ void ts_affine4(uint32_t t, uint32_t d, float m, uint32_t *o) {
  const uint32_t p = ts_hsub2(prmt(t, 0x64646464u, 0x4140u), 0x64006400u), q = ts_hsub2(prmt(t, 0x64646464u, 0x4342u), 0x64006400u);
  float v0, v1, v2, v3;
  ts_mix(p, d, m, v0, v1);
  ts_mix(q, d, m, v2, v3);
  o[0] = ts_pack<BF>(v0, v1); o[1] = ts_pack<BF>(v2, v3);
}

// NW words from the 2-byte aligned shared address a: aligned 16-byte reads, a word shift by the address, a funnel shift by half a word.
// UNIFORM: the low address bits are the same in all lanes (the shift is a branch), else they are not (selects).
template <int NW, bool UNIFORM>
__device__ __forceinline__ void ts_run(uint32_t a, uint32_t *W) {
  constexpr int NV = (NW * 4 + 14 + 15) / 16, NX = NV * 4;
  const uint32_t a0 = a & ~15u, ph = a & 15u, sh = (ph & 2u) * 8u;
  uint32_t x[NX];
#pragma unroll
  for (int i = 0; i < NV; i++) {
    const uint4 v = lds128(a0 + 16u * i);
    x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
  }
  auto at = [&](int i) { return i < NX ? x[i] : 0u; };      // (what lies past the reads is only ever shifted out)
  if constexpr (UNIFORM) {
    switch (ph >> 2) {
    case 0:
#pragma unroll
      for (int i = 0; i < NW; i++) W[i] = __funnelshift_r(at(i), at(i + 1), sh);
      break;
    case 1:
#pragma unroll
      for (int i = 0; i < NW; i++) W[i] = __funnelshift_r(at(i + 1), at(i + 2), sh);
      break;
    case 2:
#pragma unroll
      for (int i = 0; i < NW; i++) W[i] = __funnelshift_r(at(i + 2), at(i + 3), sh);
      break;
    default:
#pragma unroll
      for (int i = 0; i < NW; i++) W[i] = __funnelshift_r(at(i + 3), at(i + 4), sh);
      break;
    }
  } else {
    const bool by2 = ph & 8u, by1 = ph & 4u;
#pragma unroll
    for (int i = 0; i < NW + 2; i++) x[i] = by2 ? at(i + 2) : x[i];
#pragma unroll
    for (int i = 0; i < NW + 1; i++) x[i] = by1 ? at(i + 1) : x[i];
#pragma unroll
    for (int i = 0; i < NW; i++) W[i] = __funnelshift_r(x[i], at(i + 1), sh);
  }
}

// four high bits of a 5-bit type, starting at bit i of qh, at bit 4 of four bytes
__device__ __forceinline__ uint32_t ts_high4(uint32_t qh, int i) { return (((qh >> i) & 15u) * 0x02040810u) & 0x10101010u; }

// ---- a thread's 64 weights: elements 64 p .. 64 p + 63 of the row's span of 256.  `row` is the shared address of the span.  load
// reads the bytes, half<h> turns 32 of the weights into 16 packed pairs.  Formulas: dequant.cuh (oracle unpack_block). ----
template <int TYPE, bool UNIFORM, bool BF> struct TsUnit;

template <bool UNIFORM, bool BF> struct TsUnit<MRS_Q4_K, UNIFORM, BF> {   // d, dmin | scales[12] | qs[128]
  uint32_t q[8], d, sc, m;                 // low byte of sc, m: sub-block 2 p, next byte: 2 p + 1
  float dmin;
  __device__ __forceinline__ void scales(const uint4 &hdr, int p) {
    d = hdr.x & 0xFFFFu; dmin = ts_h2f(hdr.x >> 16);
    const int sh = 16 * (p & 1);
    const uint32_t A = hdr.y >> sh, B = hdr.z >> sh, C = hdr.w >> sh;
    if (p < 2) { sc = A & 0x3F3Fu; m = B & 0x3F3Fu; }
    else { sc = (C & 0x0F0Fu) | ((A & 0xC0C0u) >> 2); m = ((C >> 4) & 0x0F0Fu) | ((B & 0xC0C0u) >> 2); }
  }
  template <int H> __device__ __forceinline__ int scale() const { return (int)(H ? sc >> 8 : sc & 0xFFu); }
  template <int H> __device__ __forceinline__ float minimum() const { return -(dmin * (float)(H ? m >> 8 : m & 0xFFu)); }
  __device__ __forceinline__ void load(uint32_t row, int p) {
    const uint4 hdr = lds128(row), a = lds128(row + 16u + 32u * p), b = lds128(row + 32u + 32u * p);
    q[0] = a.x; q[1] = a.y; q[2] = a.z; q[3] = a.w; q[4] = b.x; q[5] = b.y; q[6] = b.z; q[7] = b.w;
    scales(hdr, p);
  }
  template <int H> __device__ __forceinline__ void half(int, uint32_t *o) const {
    // the high nibbles stay in place: 1024 + 16 q, times sc / 16, minus 64 sc
    const uint32_t off2 = ts_int2(-(H ? 64 : 1024) * scale<H>());
    const uint32_t sc2 = H ? ts_hmul2(ts_int2(scale<H>()), 0x2C002C00u) : ts_int2(scale<H>());
    const float c = minimum<H>();
#pragma unroll
    for (int i = 0; i < 8; i++)
      ts_scaled4<BF>(ts_field<H ? 0x00F000F0u : 0x000F000Fu>(q[i]), ts_field<H ? 0x00F000F0u : 0x000F000Fu>(q[i] >> 8), sc2, off2, d, c, o + 2 * i);
  }
};

template <bool UNIFORM, bool BF> struct TsUnit<MRS_Q5_K, UNIFORM, BF> : TsUnit<MRS_Q4_K, UNIFORM, BF> {   // d, dmin | scales[12] | qh[32] | qs[128]
  uint32_t h[8];
  __device__ __forceinline__ void load(uint32_t row, int p) {
    const uint4 hdr = lds128(row), a = lds128(row + 48u + 32u * p), b = lds128(row + 64u + 32u * p), c = lds128(row + 16u), e = lds128(row + 32u);
    uint32_t *q = this->q;
    q[0] = a.x; q[1] = a.y; q[2] = a.z; q[3] = a.w; q[4] = b.x; q[5] = b.y; q[6] = b.z; q[7] = b.w;
    h[0] = c.x; h[1] = c.y; h[2] = c.z; h[3] = c.w; h[4] = e.x; h[5] = e.y; h[6] = e.z; h[7] = e.w;
    this->scales(hdr, p);
  }
  template <int H> __device__ __forceinline__ void half(int p, uint32_t *o) const {
    const uint32_t sc2 = ts_int2(this->template scale<H>()), off2 = ts_int2(-1024 * this->template scale<H>());
    const float c = this->template minimum<H>();
    const int at = 4 - 2 * p - H;          // bit 2 p + H of each byte to bit 4 (the shifts stay inside the byte's word)
    const int l = at > 0 ? at : 0, r = at < 0 ? -at : 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint32_t w = H ? this->q[i] >> 4 : this->q[i], x = (h[i] << l) >> r;
      ts_scaled4<BF>(ts_or_masked(x, 0x00100010u, ts_field<0x000F000Fu>(w)), ts_or_masked(x >> 8, 0x00100010u, ts_field<0x000F000Fu>(w >> 8)), sc2,
                     off2, this->d, c, o + 2 * i);
    }
  }
};

template <bool UNIFORM, bool BF> struct TsUnit<MRS_Q6_K, UNIFORM, BF> {   // ql[128] | qh[64] | scales[16] | d
  uint32_t l[16], h[8], sc, d;
  __device__ __forceinline__ void load(uint32_t row, int p) {
    const uint32_t n = (uint32_t)p >> 1, hi = (uint32_t)p & 1u;
    ts_run<16, UNIFORM>(row + 64u * n, l);
    ts_run<8, UNIFORM>(row + 128u + 32u * n, h);
    const uint32_t s = row + 192u + 8u * n + 4u * hi;
    sc = lds_u16s(s) | (lds_u16s(s + 2u) << 16);
    d = lds_u16s(row + 208u);
  }
  template <int H> __device__ __forceinline__ void half(int p, uint32_t *o) const {
    const int hi = p & 1, at = 4 - 4 * hi - 2 * H;       // bits 4 hi + 2 H, + 1 of each byte of qh to bits 4, 5
    const int lsh = at > 0 ? at : 0, rsh = at < 0 ? -at : 0, nib = 4 * hi;
    const float s0 = (float)(int8_t)((sc >> (16 * H)) & 0xFFu), s1 = (float)(int8_t)((sc >> (16 * H + 8)) & 0xFFu), c = -1056.0f * ts_h2f(d);
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint32_t w = l[8 * H + i] >> nib, x = (h[i] << lsh) >> rsh;
      ts_times4<BF>(ts_or_masked(x, 0x00300030u, ts_field<0x000F000Fu>(w)), ts_or_masked(x >> 8, 0x00300030u, ts_field<0x000F000Fu>(w >> 8)), d, c,
                    i < 4 ? s0 : s1, o + 2 * i);
    }
  }
};

template <bool UNIFORM, bool BF> struct TsUnit<MRS_Q2_K, UNIFORM, BF> {   // scales[16] | qs[64] | d, dmin
  uint32_t q[8], sc, dm;
  __device__ __forceinline__ void load(uint32_t row, int p) {
    ts_run<8, UNIFORM>(row + 16u + 32u * ((uint32_t)p >> 1), q);
    sc = lds32(row + 4u * (uint32_t)p);    // spans start on a multiple of 4 bytes
    dm = lds32(row + 80u);
  }
  template <int H> __device__ __forceinline__ void half(int p, uint32_t *o) const {
    const int sh = 4 * (p & 1) + 2 * H;
    const float dmin = ts_h2f(dm >> 16);
#pragma unroll
    for (int g = 0; g < 2; g++) {          // 16 weights share a scale
      const int s = (int)((sc >> (16 * H + 8 * g)) & 0xFFu);
      const uint32_t sc2 = ts_int2(s & 15), off2 = ts_int2(-1024 * (s & 15));
      const float c = -(dmin * (float)(s >> 4));
#pragma unroll
      for (int i = 4 * g; i < 4 * g + 4; i++) {
        const uint32_t w = q[i] >> sh;
        ts_scaled4<BF>(ts_field<0x00030003u>(w), ts_field<0x00030003u>(w >> 8), sc2, off2, dm & 0xFFFFu, c, o + 2 * i);
      }
    }
  }
};

template <bool UNIFORM, bool BF> struct TsUnit<MRS_Q3_K, UNIFORM, BF> {   // hmask[32] | qs[64] | scales[12] | d
  uint32_t q[8], m[8], sc, d;
  __device__ __forceinline__ void load(uint32_t row, int p) {
    const uint32_t n = (uint32_t)p >> 1, jj = (uint32_t)p & 1u;
    ts_run<8, UNIFORM>(row + 32u + 32u * n, q);
    ts_run<8, UNIFORM>(row, m);
    const uint32_t s = row + 96u;
    const uint32_t lo = lds_u16s(s + 4u * jj) | (lds_u16s(s + 4u * jj + 2u) << 16), hi = lds_u16s(s + 8u) | (lds_u16s(s + 10u) << 16);
    sc = ((lo >> (4u * n)) & 0x0F0F0F0Fu) | (((hi >> (2u * (2u * n + jj))) & 0x03030303u) << 4);
    d = lds_u16s(row + 108u);
  }
  template <int H> __device__ __forceinline__ void half(int p, uint32_t *o) const {
    const int n = p >> 1, j = 2 * (p & 1) + H, at = 2 - (4 * n + j);     // bit 4 n + j of the mask to bit 2
    const int l = at > 0 ? at : 0, r = at < 0 ? -at : 0;
#pragma unroll
    for (int g = 0; g < 2; g++) {
      const int s = (int)((sc >> (16 * H + 8 * g)) & 0xFFu) - 32;
      const uint32_t sc2 = ts_int2(s), off2 = ts_int2(-1024 * s);
      const float c = ts_h2f(d) * (float)(-4 * s);        // exact, and so is d (sc q) - 4 d sc
#pragma unroll
      for (int i = 4 * g; i < 4 * g + 4; i++) {
        const uint32_t w = q[i] >> (2 * j), x = (m[i] << l) >> r;
        ts_scaled4<BF>(ts_or_masked(x, 0x00040004u, ts_field<0x00030003u>(w)), ts_or_masked(x >> 8, 0x00040004u, ts_field<0x00030003u>(w >> 8)), sc2,
                       off2, d, c, o + 2 * i);
      }
    }
  }
};

// 32-wide types: two blocks, one run of 2 x BYTES bytes (spans start on a multiple of 4 bytes)
template <bool UNIFORM, bool BF> struct TsUnit<MRS_Q4_0, UNIFORM, BF> {   // d | qs[16]
  uint32_t w[9];
  __device__ __forceinline__ void load(uint32_t row, int p) { ts_run<9, UNIFORM>(row + 36u * (uint32_t)p, w); }
  template <int H> __device__ __forceinline__ void half(int, uint32_t *o) const {
    const uint32_t d = H ? w[4] >> 16 : w[0] & 0xFFFFu;
    const float c = -1032.0f * ts_h2f(d);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t q = H ? w[5 + i] : __funnelshift_r(w[i], w[i + 1], 16);
      ts_bytes4<8, BF>(q & 0x0F0F0F0Fu, d, c, o + 2 * i);
      ts_bytes4<8, BF>((q >> 4) & 0x0F0F0F0Fu, d, c, o + 8 + 2 * i);
    }
  }
};

template <bool UNIFORM, bool BF> struct TsUnit<MRS_Q4_1, UNIFORM, BF> {   // d, m | qs[16]
  uint32_t w[10];
  __device__ __forceinline__ void load(uint32_t row, int p) { ts_run<10, UNIFORM>(row + 40u * (uint32_t)p, w); }
  template <int H> __device__ __forceinline__ void half(int, uint32_t *o) const {
    const uint32_t d = w[5 * H] & 0xFFFFu;
    const float m = ts_h2f(w[5 * H] >> 16);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t q = w[5 * H + 1 + i];
      ts_affine4<BF>(q & 0x0F0F0F0Fu, d, m, o + 2 * i);
      ts_affine4<BF>((q >> 4) & 0x0F0F0F0Fu, d, m, o + 8 + 2 * i);
    }
  }
};

template <bool UNIFORM, bool BF> struct TsUnit<MRS_Q5_0, UNIFORM, BF> {   // d | qh[4] | qs[16]
  uint32_t w[11];
  __device__ __forceinline__ void load(uint32_t row, int p) { ts_run<11, UNIFORM>(row + 44u * (uint32_t)p, w); }
  template <int H> __device__ __forceinline__ void half(int, uint32_t *o) const {
    const uint32_t d = H ? w[5] >> 16 : w[0] & 0xFFFFu, qh = H ? w[6] : __funnelshift_r(w[0], w[1], 16);
    const float c = -1040.0f * ts_h2f(d);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t q = H ? w[7 + i] : __funnelshift_r(w[1 + i], w[2 + i], 16);
      ts_bytes4<16, BF>(ts_or_masked(q, 0x0F0F0F0Fu, ts_high4(qh, 4 * i)), d, c, o + 2 * i);
      ts_bytes4<16, BF>(ts_or_masked(q >> 4, 0x0F0F0F0Fu, ts_high4(qh, 16 + 4 * i)), d, c, o + 8 + 2 * i);
    }
  }
};

template <bool UNIFORM, bool BF> struct TsUnit<MRS_Q5_1, UNIFORM, BF> {   // d, m | qh[4] | qs[16]
  uint32_t w[12];
  __device__ __forceinline__ void load(uint32_t row, int p) { ts_run<12, UNIFORM>(row + 48u * (uint32_t)p, w); }
  template <int H> __device__ __forceinline__ void half(int, uint32_t *o) const {
    const uint32_t d = w[6 * H] & 0xFFFFu;
    const float m = ts_h2f(w[6 * H] >> 16);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t q = w[6 * H + 2 + i];
      ts_affine4<BF>(ts_or_masked(q, 0x0F0F0F0Fu, ts_high4(w[6 * H + 1], 4 * i)), d, m, o + 2 * i);
      ts_affine4<BF>(ts_or_masked(q >> 4, 0x0F0F0F0Fu, ts_high4(w[6 * H + 1], 16 + 4 * i)), d, m, o + 8 + 2 * i);
    }
  }
};

template <bool UNIFORM, bool BF> struct TsUnit<MRS_Q8_0, UNIFORM, BF> {   // d | qs[32]
  uint32_t w[17];
  __device__ __forceinline__ void load(uint32_t row, int p) { ts_run<17, UNIFORM>(row + 68u * (uint32_t)p, w); }
  template <int H> __device__ __forceinline__ void half(int, uint32_t *o) const {
    const uint32_t d = H ? w[8] >> 16 : w[0] & 0xFFFFu;
    const float c = -1152.0f * ts_h2f(d);
#pragma unroll
    for (int i = 0; i < 8; i++)            // q + 128
      ts_bytes4<128, BF>((H ? w[9 + i] : __funnelshift_r(w[i], w[i + 1], 16)) ^ 0x80808080u, d, c, o + 2 * i);
  }
};

// int4 checkpoints.  The word order of the tiles puts (k, k + 1) in the nibbles at bits 0 and 16: (q & 0xf) | 0x6400 is 1024 + q as f16,
// | 0x4300 is 128 + q as bf16 (7 bits of mantissa hold the nibble); q - z is exact, times the scale rounds once (REF marlin dequant).
template <bool BF> struct TsInt4 {
  uint4 a, b;
  uint32_t s[2], z[2];
  template <int H> __device__ __forceinline__ void half(uint32_t *o) const {
    const uint32_t s2 = s[H] * 0x00010001u, w[4] = {H ? b.x : a.x, H ? b.y : a.y, H ? b.z : a.z, H ? b.w : a.w};
#pragma unroll
    for (int c = 0; c < 4; c++) {
      if constexpr (BF) {
        const uint32_t sub = 0x43004300u + z[H] * 0x00010001u;
#pragma unroll
        for (int j = 0; j < 4; j++) {
          uint32_t v;
          asm("lop3.b32 %0, %1, 0x000f000f, 0x43004300, 0xea;" : "=r"(v) : "r"(w[c] >> (4 * j)));
          const __nv_bfloat162 r = __hmul2(__hsub2(*(const __nv_bfloat162 *)&v, *(const __nv_bfloat162 *)&sub), *(const __nv_bfloat162 *)&s2);
          o[4 * c + j] = *(const uint32_t *)&r;
        }
      } else {
        // bits 4 .. 7 in place: 1024 + 16 q, times 1/16, minus 64 + z — exact
        const uint32_t lo = 0x64006400u + z[H] * 0x00010001u, hi = (0xD400u + (z[H] << 4)) * 0x00010001u;
#pragma unroll
        for (int j = 0; j < 2; j++) {
          const uint32_t q = w[c] >> (8 * j);
          o[4 * c + 2 * j] = ts_hmul2(ts_hsub2(ts_field<0x000F000Fu>(q), lo), s2);
          o[4 * c + 2 * j + 1] = ts_hmul2(ts_hfma2(ts_field<0x00F000F0u>(q), 0x2C002C00u, hi), s2);
        }
      }
    }
  }
};

__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t *r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::
          "r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// 32 lanes x 8 columns of accumulators
__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, uint32_t *r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void ts_cp_async16(uint32_t dst, const void *src, uint32_t bytes) {   // bytes < 16: the rest are zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// Four products over 64 k by the whole warp, one elected lane issuing: A at the TMEM address a (8 columns each), B at the shared
// address b (32 bytes on inside the SWIZZLE_128B atom each); descriptor fields as in umma_desc_sw128.  Behind them, where `bar` is not 0,
// the arrival on it of all products issued so far.
__device__ __forceinline__ void ts_mma4(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t accumulate, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred e, p, q;\n\t.reg .b32 l, t;\n\t.reg .b64 x;\n\t"
      "elect.sync _|e, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.eq.b32 q, %3, %3;\n\t"
      "shr.u32 l, %2, 4;\n\tor.b32 l, l, 0x10000;\n\tmov.b64 x, {l, %5};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], x, %3, p;\n\t"
      "add.u32 l, l, 2;\n\tadd.u32 t, %1, 8;\n\tmov.b64 x, {l, %5};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [t], x, %3, q;\n\t"
      "add.u32 l, l, 2;\n\tadd.u32 t, t, 8;\n\tmov.b64 x, {l, %5};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [t], x, %3, q;\n\t"
      "add.u32 l, l, 2;\n\tadd.u32 t, t, 8;\n\tmov.b64 x, {l, %5};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [t], x, %3, q;\n\t"
      "setp.ne.and.b32 p, %6, 0, e;\n\t"
      "@p tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%6];\n\t}" ::"r"(d), "r"(a), "r"(b), "r"(idesc), "r"(accumulate),
      "n"((1024 >> 4) | (1 << 14) | (2 << 29)), "r"(bar)
      : "memory");
}

// the sixteen products of a span, XB tiles of X a wait
template <int XB>
__device__ __forceinline__ bool ts_issue_span(uint32_t acc, uint32_t a, uint32_t more, uint32_t idesc, uint64_t *x_full, uint32_t x0, uint32_t xe0, int x_bytes,
                                              int XS, int &xs, int &xph, int *late) {
#pragma unroll
  for (int h = 0; h < 4; h += XB) {
    if (!ts_wait(x_full + xs, xph, late)) return false;
    tc_fence_after();
    const uint32_t b = x0 + (uint32_t)(xs * XB * x_bytes);
#pragma unroll
    for (int e = 0; e < XB; e++)
      ts_mma4(acc, a + 32u * (uint32_t)(h + e), b + (uint32_t)(e * x_bytes), idesc, h + e ? 1u : more, e == XB - 1 ? xe0 + 8u * (uint32_t)xs : 0u);
    if (++xs == XS) { xs = 0; xph ^= 1; }
  }
  return true;
}

// Up to three matrices of a type that read the same activations, as one grid: their row tiles follow one another (p.N, p.y and the map of the launch are the
// first one's).  Alone each pays for its start, its drain and its last wave: q, k and v of an 8B model (Q4_K, 4096 + 1024 + 1024 rows) at 300 tokens.
struct TsMore {
  CUtensorMap w[2];
  void *y[2];
  int n[2], first[2];                    // rows, and the first row tile, of the second and the third matrix
};

// of row `r` of row tile tn: the row in its matrix, the matrix's rows and results
__device__ __forceinline__ void ts_place(const TsMore *more, int tn, int r, int &nrow, int &N, void *&out) {
  if (tn < more->first[0]) return;
  const int k = tn >= more->first[1] ? 1 : 0;
  nrow = (tn - more->first[k]) * TS_BM + r;
  N = more->n[k];
  out = more->y[k];
}

template <int TYPE, bool ALIGNED, bool BF, bool MULTI>
__device__ __forceinline__ void ts_grid(const CUtensorMap &tmap_w, const CUtensorMap &tmap_x, const TsParams &p, const TsMore *more) {
  using F = TsFmt<TYPE>;
  constexpr int PITCH = TsPitch<TYPE, ALIGNED>::value, RAW_BYTES = TsStage<TYPE, ALIGNED>::BYTES;
  constexpr int LOADERS = ALIGNED ? 1 : 64;           // arrivals that fill a raw stage
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int x_bytes = p.nt * 128, RS = p.rs, XS = p.xs, XB = p.xb;
  uint8_t *x_ring = smem, *r_ring = smem + (size_t)XS * XB * x_bytes;
  uint64_t *bars = (uint64_t *)(r_ring + (size_t)RS * RAW_BYTES);
  uint64_t *raw_full = bars, *raw_empty = raw_full + TS_RS_MAX, *x_full = raw_empty + TS_RS_MAX, *x_empty = x_full + TS_XS_MAX,
           *a_full = x_empty + TS_XS_MAX, *a_empty = a_full + TS_AS, *acc_full = a_empty + TS_AS, *acc_empty = acc_full + 2, *drain = acc_empty + 2;
  uint32_t *tmem_slot = (uint32_t *)(bars + TS_N_BARS);
  int *const late = p.timeouts;

  // (taken from lane 0: the compiler then knows that the warp's branches are uniform and keeps their operands in uniform registers)
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (p.pdl && tid == 96) pdl_launch_dependents();
  const int n_spans = (p.K + TS_SPAN_K - 1) / TS_SPAN_K, n_tiles = p.tiles_m * p.tiles_n;
  const int rank = (int)blockIdx.x, first = (int)blockIdx.y, step = (int)gridDim.y;      // a cluster is one row of the grid
  int s0 = 0, s1 = n_spans;
  if (p.ksplit > 1) { s0 = n_spans * rank / p.ksplit; s1 = n_spans * (rank + 1) / p.ksplit; }
  const int n_acc = p.nt <= 128 ? 2 : 1;              // accumulators that fit in front of the A stages

  // Set-up, split so that both streams start at once: the producers initialise their own rings' barriers and signal the CTA barrier
  // without waiting for it; it orders their initialisation before any consumer's first wait.
  uint32_t tmem_base = 0u;
  if (warp == 0 || warp == 2) {
    if (warp == 0) {
      if (lane < 2 * TS_RS_MAX) mbar_init(&raw_full[lane], lane < TS_RS_MAX ? (uint32_t)LOADERS : (uint32_t)TS_DQ_WARPS);
    } else if (lane < 2 * TS_XS_MAX) {
      mbar_init(&x_full[lane], 1u);
    }
    fence_mbar_init();
    __syncwarp();
    asm volatile("bar.arrive 1, %0;" ::"n"(TS_THREADS) : "memory");
  } else {
    if (warp == 1) {
      if (lane < 2 * TS_AS + 5)
        mbar_init(&a_full[lane], lane < TS_AS ? (uint32_t)TS_DQ_WARPS : lane >= 2 * TS_AS + 2 && lane < 2 * TS_AS + 4 ? (uint32_t)TS_EPI_WARPS : 1u);
      fence_mbar_init();
      __syncwarp();
      tmem_alloc(tmem_slot, 512);
    }
    tc_fence_before();
    asm volatile("bar.sync 1, %0;" ::"n"(TS_THREADS) : "memory");
    tc_fence_after();
    tmem_base = __reduce_max_sync(0xffffffffu, *tmem_slot);                 // uniform register
  }
  const uint32_t tmem_a = tmem_base + 256u;

  if (warp == 0 || (warp == 3 && !ALIGNED)) {
    // ===================== raw producer =====================
    int it = 0, st = 0, ph = 0;
    bool ok = true;
    for (int t = first; ok && t < n_tiles; t += step) {
      int n0 = (t % p.tiles_n) * TS_BM;
      const CUtensorMap *map = &tmap_w;
      if constexpr (MULTI) {
        const int tn = t % p.tiles_n, k = tn >= more->first[1] ? 1 : 0;
        if (tn >= more->first[0]) { n0 = (tn - more->first[k]) * TS_BM; map = &more->w[k]; }
      }
      for (int s = s0; s < s1; s++, it++) {
        if (p.pdl && it == RS) pdl_wait();             // the ring is full: from here on its stages are freed at the grid before's pace
        ok = ts_wait(raw_empty + st, ph ^ 1, late);
        if (!ok) break;
        if constexpr (ts_is_int4(TYPE)) {
          const int k0 = s * TS_SPAN_K, rows = min(TS_BM, p.N - n0), chunks = min(4, (p.K - k0) >> 6), g0 = (k0 >> 5) / p.group32;
          const int groups = ((k0 + 64 * chunks - 1) >> 5) / p.group32 - g0 + 1;                // that the span's k touch
          const uint32_t dst = smem_u32(r_ring) + (uint32_t)st * RAW_BYTES, bar = smem_u32(raw_full + st);
          const uint32_t zero_bytes = p.qzeros != nullptr ? (uint32_t)rows / 2u : 0u;
          mbar_arrive_expect_tx_warp(raw_full + st, (uint32_t)(chunks * rows * 32) + (uint32_t)groups * ((uint32_t)rows * 2u + zero_bytes));
          const uint8_t *src = p.w + ((size_t)(k0 >> 6) * p.N + n0) * 32;
          for (int c = 0; c < chunks; c++) bulk_g2s_warp(dst + (uint32_t)(c * TS_I4_CHUNK), src + (size_t)c * p.N * 32, (uint32_t)rows * 32u, bar, 1u);
          for (int g = 0; g < groups; g++) {
            bulk_g2s_warp(dst + (uint32_t)(TS_I4_SCALES + g * TS_BM * 2), p.scales + ((size_t)(g0 + g) * p.N + n0) * 2, (uint32_t)rows * 2u, bar, 1u);
            if (zero_bytes) bulk_g2s_warp(dst + (uint32_t)(TS_I4_ZEROS + g * 64), p.qzeros + ((size_t)(g0 + g) * (p.N >> 3) + (n0 >> 3)) * 4, zero_bytes, bar, 1u);
          }
        } else if constexpr (ALIGNED) {
          // (a box starts on a 16-byte boundary: the aligned address below the span; the dequantisers read from the phase on)
          mbar_arrive_expect_tx_warp(raw_full + st, RAW_BYTES);
          tma_load_2d_warp(r_ring + (size_t)st * RAW_BYTES, map, ((s * F::SPAN) & ~15) / 2, n0, raw_full + st);
        } else {
          constexpr int CH = (F::SPAN + 14 + 15) / 16;                     // 16-byte chunks that cover a span at any phase
          const uint32_t dst = smem_u32(r_ring) + (uint32_t)st * RAW_BYTES;
          const long long total = (long long)p.N * p.row_bytes;
#pragma unroll 4
          for (int i = (warp ? 32 : 0) + lane; i < TS_BM * CH; i += 64) {
            const int r = i / CH, c = i % CH;
            const long long row = (long long)(n0 + r) * p.row_bytes, at = ((row + (long long)s * F::SPAN) & ~15ll) + 16 * c;
            // a chunk is read while it starts inside its row; past the end of the matrix it is zeros
            const bool in = n0 + r < p.N && at < row + p.row_bytes;
            ts_cp_async16(dst + (uint32_t)(r * PITCH + 16 * c), p.w + (in ? at : 0), in ? (uint32_t)min(16ll, total - at) : 0u);
          }
          asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(raw_full + st)) : "memory");
        }
        if (++st == RS) { st = 0; ph ^= 1; }
      }
    }
    // copies in flight land before the CTA may end
    if constexpr (ALIGNED) { for (int i = max(0, it - RS); i < it; i++) ts_wait(raw_full + i % RS, (i / RS) & 1, late); }
    else asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp == 2) {
    // ===================== X producer: XB tiles of [tokens x 64 k] a stage (zeros past M and K) =====================
    if (p.pdl) pdl_wait();                   // the activations are the grid's before (the weight stream does not wait)
    int it = 0, st = 0, ph = 0;
    bool ok = true;
    for (int t = first; ok && t < n_tiles; t += step) {
      const int m0 = (t / p.tiles_n) * p.nt;
      for (int s = 4 * s0; s < 4 * s1; s += XB, it++) {
        ok = ts_wait(x_empty + st, ph ^ 1, late);
        if (!ok) break;
        mbar_arrive_expect_tx_warp(x_full + st, (uint32_t)(XB * x_bytes));
        for (int h = 0; h < XB; h++)
          tma_load_2d_warp(x_ring + (size_t)(st * XB + h) * x_bytes, &tmap_x, (s + h) * TS_XK, m0, x_full + st);
        if (++st == XS) { st = 0; ph ^= 1; }
      }
    }
    for (int i = max(0, it - XS); i < it; i++) ts_wait(x_full + i % XS, (i / XS) & 1, late);
  } else if (warp == 1) {
    // ===================== MMA issuer: D[128 rows, tokens] += A[tmem] . X[smem]^T =====================
    const uint32_t fmt = BF ? 1u : 0u;
    const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(p.nt >> 3) << 17) | ((uint32_t)(TS_BM >> 4) << 24);
    // (reductions leave their result in uniform registers, where the products take their operands from)
    const uint32_t x0 = __reduce_max_sync(0xffffffffu, smem_u32(x_ring)), xe0 = __reduce_max_sync(0xffffffffu, smem_u32(x_empty));
    int it = 0, xs = 0, xph = 0, j = 0;
    bool ok = true;
    if (p.pdl) pdl_wait();                   // (x_full completes behind it)
    for (int t = first; ok && t < n_tiles; t += step, j++) {
      const int b = j % n_acc;
      const uint32_t acc = tmem_base + (uint32_t)b * 128u;
      ok = ts_wait(acc_empty + b, ((j / n_acc) & 1) ^ 1, late);
      if (!ok) break;
      tc_fence_after();
      for (int s = s0; s < s1; s++, it++) {
        const int as = it % TS_AS;
        ok = ts_wait(a_full + as, (it / TS_AS) & 1, late);
        if (!ok) break;
        const uint32_t ta = tmem_a + (uint32_t)as * 128u;
        const uint32_t more = s > s0 ? 1u : 0u;
        if (XB == 4) ok = ts_issue_span<4>(acc, ta, more, idesc, x_full, x0, xe0, x_bytes, XS, xs, xph, late);
        else if (XB == 2) ok = ts_issue_span<2>(acc, ta, more, idesc, x_full, x0, xe0, x_bytes, XS, xs, xph, late);
        else ok = ts_issue_span<1>(acc, ta, more, idesc, x_full, x0, xe0, x_bytes, XS, xs, xph, late);
        if (!ok) break;
        umma_commit_warp(a_empty + as);
      }
      if (ok) umma_commit_warp(acc_full + b);
    }
    if (it > 0) {                            // no product is in flight when tensor memory is freed
      umma_commit_warp(drain);
      ts_wait(drain, 0, late);
    }
  } else if (warp >= 4 && warp < 4 + TS_DQ_WARPS) {
    // ===================== dequantisers: warp -> (TMEM lane quarter, 64 k of the span) =====================
    const int q4 = warp & 3, part = (warp - 4) >> 2;
    const int r = q4 * 32 + lane;                      // weight row in the tile == TMEM lane
    const uint32_t row0 = smem_u32(r_ring) + (uint32_t)(r * PITCH);
    const uint32_t ta0 = tmem_a + ((uint32_t)(q4 * 32) << 16) + (uint32_t)(part * 32);
    uint32_t scale0 = 0u, zero0 = 0u;                  // int4: this row's first scale and zero-point word
    int zero_shift = 0;
    if constexpr (ts_is_int4(TYPE)) {
      // inverses of the reference's scale-column permutations (REF gptq_cuda.rs:530-540 get_scale_perms), which stay inside a tile:
      // 64 wide perm[8 i + j] = i + 8 j, 32 wide perm[8 i + j] = 2 i + {0, 1, 8, 9, 16, 17, 24, 25}[j]
      const int c = p.scale_perm == 1 ? (r & ~63) + 8 * (r & 7) + ((r & 63) >> 3)
                  : p.scale_perm == 2 ? (r & ~31) + 8 * ((r & 7) >> 1) + 2 * ((r & 31) >> 3) + (r & 1) : r;
      scale0 = smem_u32(r_ring) + (uint32_t)(TS_I4_SCALES + 2 * c);
      zero0 = smem_u32(r_ring) + (uint32_t)(TS_I4_ZEROS + 4 * (r >> 3));
      zero_shift = 4 * ((r & 1) ? 4 + ((r & 7) >> 1) : (r & 7) >> 1);        // nibble i of a word is column {0, 2, 4, 6, 1, 3, 5, 7}[i]
    }
    int it = 0, st = 0, ph = 0;
    bool ok = true;
    for (int t = first; ok && t < n_tiles; t += step) {
      const int n0 = (t % p.tiles_n) * TS_BM;
      for (int s = s0; s < s1; s++, it++) {
        const int as = it % TS_AS;
        uint32_t phase;                                // of the span inside its 16-byte aligned copy
        if constexpr (ts_is_int4(TYPE)) phase = 0u;
        else if constexpr (ALIGNED) phase = (uint32_t)(s * F::SPAN) & 15u;
        else phase = ((uint32_t)(n0 + r) * (uint32_t)p.row_bytes + (uint32_t)s * (uint32_t)F::SPAN) & 15u;
        ok = ts_wait(raw_full + st, ph, late);
        if (!ok) break;
        const bool live = s * TS_SPAN_K + 64 * part < p.K;   // the last span of a 32-wide type may be ragged
        uint32_t o[16];
        const uint32_t stage = (uint32_t)st * RAW_BYTES;
        typename std::conditional<ts_is_int4(TYPE), TsInt4<BF>, TsUnit<TYPE, ALIGNED, BF>>::type u;
        if constexpr (ts_is_int4(TYPE)) {
          u.a = lds128(row0 + stage + (uint32_t)(part * TS_I4_CHUNK)); u.b = lds128(row0 + stage + (uint32_t)(part * TS_I4_CHUNK) + 16u);
          // each 32 weights' group, counted from the span's first (uniform); in units of 32 weights, by shifts where a group is a power of two
          const uint32_t u0 = (uint32_t)(s * (TS_SPAN_K / 32)), u1 = u0 + 2u * (uint32_t)part;
          const uint32_t g0 = p.group_shift >= 0 ? u0 >> p.group_shift : u0 / (uint32_t)p.group32;
#pragma unroll
          for (uint32_t h = 0; h < 2; h++) {
            const uint32_t g = (p.group_shift >= 0 ? (u1 + h) >> p.group_shift : (u1 + h) / (uint32_t)p.group32) - g0;
            u.s[h] = lds_u16s(scale0 + stage + g * (TS_BM * 2));
            if constexpr (TYPE == TS_INT4_OTHER) {
              if constexpr (BF) u.s[h] = __bfloat16_as_ushort(__float2bfloat16_rn(ts_h2f(u.s[h])));
              else u.s[h] = __half_as_ushort(__float2half_rn(__uint_as_float(u.s[h] << 16)));
            }
            u.z[h] = p.qzeros != nullptr ? (lds32(zero0 + stage + g * 64u) >> zero_shift) & 0xFu : 8u;
          }
          u.template half<0>(o);
        } else {
          u.load(row0 + stage + phase, part);
          u.template half<0>(part, o);
        }
        if (p.pdl && it == TS_AS) pdl_wait();          // (a stage is freed by products, which need x)
        ok = ts_wait(a_empty + as, ((it / TS_AS) & 1) ^ 1, late);   // the MMAs that read this A stage have retired
        if (!ok) break;
        tc_fence_after();
        const uint32_t ta = ta0 + (uint32_t)as * 128u;
        if (!live) {
#pragma unroll
          for (int i = 0; i < 16; i++) o[i] = 0u;
        }
        tmem_st_32x16(ta, o);
        if constexpr (ts_is_int4(TYPE)) u.template half<1>(o);
        else u.template half<1>(part, o);
        if (!live) {
#pragma unroll
          for (int i = 0; i < 16; i++) o[i] = 0u;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(raw_empty + st);    // the span's bytes are in registers (and past them)
        tmem_st_32x16(ta + 16u, o);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(a_full + as);
        if (++st == RS) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp >= 4 + TS_DQ_WARPS && p.ksplit == 1) {
    // ===================== epilogue, K whole: TMEM -> registers -> y[token][row] =====================
    const int q4 = warp & 3;
    if (p.pdl) pdl_wait();                   // y may still be read by the grid before
    int j = 0;
    for (int t = first; t < n_tiles; t += step, j++) {
      const int b = j % n_acc, m0 = (t / p.tiles_n) * p.nt;
      int nrow = (t % p.tiles_n) * TS_BM + q4 * 32 + lane, N = p.N;
      void *out = p.y;
      if constexpr (MULTI) ts_place(more, t % p.tiles_n, q4 * 32 + lane, nrow, N, out);
      if (!ts_wait(acc_full + b, (j / n_acc) & 1, late)) break;
      tc_fence_after();
      const int cols = min(p.nt, p.M - m0);
#pragma unroll 1
      for (int c0 = 0; c0 < cols; c0 += 32) {
        uint32_t acc[32];
        tmem_ld_32x32(tmem_base + (uint32_t)b * 128u + ((uint32_t)(q4 * 32) << 16) + (uint32_t)c0, acc);
        if (c0 + 32 >= cols) {                         // the last columns are in registers: the next tile's products may start
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc_empty + b);
        }
        if (nrow < N) {
          uint16_t *y = (uint16_t *)out + (size_t)(m0 + c0) * N + nrow;
#pragma unroll
          for (int c = 0; c < 32; c++) {
            if (c0 + c < cols) {
              const float v = __uint_as_float(acc[c]);
              if constexpr (BF) *(__nv_bfloat16 *)y = __float2bfloat16_rn(v);
              else *(__half *)y = __float2half_rn(v);
            }
            y += N;
          }
        }
      }
    }
  }
  if (p.ksplit > 1) {
    // ===================== epilogue, K split: partial tiles meet in shared memory =====================
    // Rank r sums tokens [r C, r C + C): every CTA writes its partial columns to their owner's rings, which are free once all CTAs of
    // the cluster have left their products behind.  One tile per cluster.
    const int C = ((p.nt + p.ksplit - 1) / p.ksplit + 7) & ~7;
    const int q4 = warp & 3, g = (warp - 4) >> 2, row = q4 * 32 + lane;      // five warps share a lane quarter
    constexpr int G = (TS_DQ_WARPS + TS_EPI_WARPS) / 4;
    float *red = (float *)smem;                        // [rank][C][128 rows]
    __syncwarp();
    if (p.pdl) pdl_wait();
    bool ok = true;
    if (warp >= 4) {
      ok = ts_wait(acc_full, 0, late);
      tc_fence_after();
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (warp >= 4) {
      for (int c0 = 8 * g; c0 < p.nt; c0 += 8 * G) {
        uint32_t v[8];
        tmem_ld_32x8(tmem_base + ((uint32_t)(q4 * 32) << 16) + (uint32_t)c0, v);
        const uint32_t owner = (uint32_t)(c0 / C);
        uint32_t to;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(smem_u32(red + (rank * C + c0 - (int)owner * C) * TS_BM + row)), "r"(owner));
#pragma unroll
        for (int i = 0; i < 8; i++) asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(to + (uint32_t)i * (TS_BM * 4)), "r"(v[i]) : "memory");
      }
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int m0 = (first / p.tiles_n) * p.nt + rank * C;
    int nrow = (first % p.tiles_n) * TS_BM + row, N = p.N;
    void *out = p.y;
    if constexpr (MULTI) ts_place(more, first % p.tiles_n, row, nrow, N, out);
    if (warp >= 4 && ok && nrow < N) {
      const int cols = min(min(C, p.nt - rank * C), p.M - m0);
      for (int c = g; c < cols; c += G) {
        float v = red[(size_t)c * TS_BM + row];
        for (int s = 1; s < p.ksplit; s++) v += red[((size_t)s * C + c) * TS_BM + row];
        const size_t at = (size_t)(m0 + c) * N + nrow;
        if constexpr (BF) ((__nv_bfloat16 *)out)[at] = __float2bfloat16_rn(v);
        else ((__half *)out)[at] = __float2half_rn(v);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}
template <int TYPE, bool ALIGNED, bool BF>
__global__ void __launch_bounds__(TS_THREADS, 1)
mmq_ts_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const TsParams p) {
  ts_grid<TYPE, ALIGNED, BF, false>(tmap_w, tmap_x, p, nullptr);
}
template <int TYPE, bool BF>
__global__ void __launch_bounds__(TS_THREADS, 1)
mmq_ts_multi_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const TsParams p, const __grid_constant__ TsMore more) {
  ts_grid<TYPE, true, BF, true>(tmap_w, tmap_x, p, &more);
}

// ---- host ---------------------------------------------------------------------------------------
struct TsCall {
  const void *w, *x;
  void *y;
  int M, N, K, row_bytes, dtype;      // dtype: 0 f16, 1 bf16 (activations, outputs and the dequantised weights)
  int nt, tiles_m, ksplit, sms;       // the plan
  int *timeouts;
  cudaStream_t stream;
  const void *scales, *qzeros;        // int4
  int group, scale_perm, pdl;
  int matrices;                       // more than one: w, y and N are the first's
  const void *w2[2];
  void *y2[2];
  int n2[2];
};

template <int TYPE> static bool ts_map_weights(CUtensorMap *map, const void *w, int N, int row_bytes) {
  const cuuint64_t dims[2] = {(cuuint64_t)(row_bytes / 2), (cuuint64_t)N};
  const cuuint64_t strides[1] = {(cuuint64_t)row_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)(TsPitch<TYPE, true>::value / 2), (cuuint32_t)TS_BM};
  const cuuint32_t estr[2] = {1, 1};
  return tc_get_encode()(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void *>(w), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
template <int TYPE, bool ALIGNED> static cudaError_t ts_launch_as(const TsCall &c) {
  constexpr int RAW_BYTES = TsStage<TYPE, ALIGNED>::BYTES;
  // types that files hold side by side: q, k and v, gate and up
  constexpr bool GROUPS = ALIGNED && (TYPE == MRS_Q4_K || TYPE == MRS_Q5_K || TYPE == MRS_Q6_K || TYPE == MRS_Q8_0);
  if (c.matrices > 1 && !GROUPS) return cudaErrorNotSupported;
  if (tc_get_encode() == nullptr) return cudaErrorNotSupported;
  CUtensorMap tw, tx;
  if (!tc_make_map_2d(&tx, c.x, (uint64_t)c.M, (uint64_t)c.K, TS_XK, (uint32_t)c.nt, c.dtype)) return cudaErrorInvalidValue;
  if (ALIGNED && !ts_is_int4(TYPE)) {
    if (!ts_map_weights<TYPE>(&tw, c.w, c.N, c.row_bytes)) return cudaErrorInvalidValue;
  } else {
    tw = tx;                          // not read
  }
  TsParams p = {};
  p.w = (const uint8_t *)c.w; p.y = c.y; p.timeouts = c.timeouts; p.M = c.M; p.N = c.N; p.K = c.K; p.row_bytes = c.row_bytes;
  p.scales = (const uint8_t *)c.scales; p.qzeros = (const uint8_t *)c.qzeros; p.scale_perm = c.scale_perm; p.pdl = c.pdl;
  p.group32 = c.group / 32; p.group_shift = -1;
  for (int i = 0; i < 26; i++) if (p.group32 == 1 << i) p.group_shift = i;
  p.nt = c.nt; p.tiles_m = c.tiles_m; p.tiles_n = (c.N + TS_BM - 1) / TS_BM; p.ksplit = c.ksplit;
  // Fewer and larger X stages where the tokens are few: each costs the issuer a wait and a commit.  Three raw stages (two where three do
  // not fit), the rest of the memory first to X up to its limit: a stage's round trip (products retire, copy from L2) takes some 2500
  // clocks, so with four stages of 64 k a span of 160 tokens took 3000 clocks where its products take 1280.
  constexpr int BUDGET = TS_SMEM_MAX - 2048;
  p.xb = c.nt > 176 ? 1 : c.nt > 64 ? 2 : 4;
  const int stage = p.xb * c.nt * 128;
  p.xs = (BUDGET - 3 * RAW_BYTES) / stage;
  if (p.xs < 4) p.xs = (BUDGET - 2 * RAW_BYTES) / stage;
  if (p.xs > TS_XS_MAX) p.xs = TS_XS_MAX;
  if (p.xb == 4 && p.xs > 4) p.xs = 4;
  p.rs = (BUDGET - p.xs * stage) / RAW_BYTES;
  if (p.rs > TS_RS_MAX) p.rs = TS_RS_MAX;
  TsMore more;
  if (c.matrices > 1) {
    for (int i = 0; i < 2; i++) {
      const bool there = i + 1 < c.matrices;
      if (there && !ts_map_weights<TYPE>(&more.w[i], c.w2[i], c.n2[i], c.row_bytes)) return cudaErrorInvalidValue;
      more.first[i] = there ? p.tiles_n : 1 << 30;
      more.n[i] = there ? c.n2[i] : 0;
      more.y[i] = there ? c.y2[i] : nullptr;
      if (!there) more.w[i] = tx;     // not read
      if (there) p.tiles_n += (c.n2[i] + TS_BM - 1) / TS_BM;
    }
  }
  const int tiles = p.tiles_m * p.tiles_n;
  auto kern = c.dtype == 1 ? mmq_ts_kernel<TYPE, ALIGNED, true> : mmq_ts_kernel<TYPE, ALIGNED, false>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = p.ksplit > 1 ? dim3(p.ksplit, tiles) : dim3(1, tiles < c.sms ? tiles : c.sms);
  cfg.blockDim = dim3(TS_THREADS);
  cfg.dynamicSmemBytes = (size_t)(2048 + p.xs * stage + p.rs * RAW_BYTES);
  cfg.stream = c.stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (p.ksplit > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = p.ksplit; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = 1;
    na++;
  }
  if (p.pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    na++;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  if constexpr (GROUPS) {
    if (c.matrices > 1) {
      auto multi = c.dtype == 1 ? mmq_ts_multi_kernel<TYPE, true> : mmq_ts_multi_kernel<TYPE, false>;
      cudaFuncSetAttribute(multi, cudaFuncAttributeMaxDynamicSharedMemorySize, TS_SMEM_MAX);
      return cudaLaunchKernelEx(&cfg, multi, tw, tx, p, more);
    }
  }
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TS_SMEM_MAX);
  return cudaLaunchKernelEx(&cfg, kern, tw, tx, p);
}

template <int TYPE> cudaError_t ts_launch(const TsCall &c) {
  if (ts_is_int4(TYPE) || c.row_bytes % 16 == 0) return ts_launch_as<TYPE, true>(c);
  // superblocks of 144 and 176 bytes make every row a multiple of 16
  if constexpr (ts_is_int4(TYPE) || TYPE == MRS_Q4_K || TYPE == MRS_Q5_K) return cudaErrorNotSupported;
  else return ts_launch_as<TYPE, false>(c);
}

// what a plan is made for and from: the current device, and the choice of token tile and split (mmq_ts.cu)
struct TsDevice { int sms, clusters[9]; int *timeouts; int32_t *flag; };   // the timeout word as the device and as the host address it
const TsDevice &ts_device();
// cudaErrorLaunchTimeout once a wait has run out on the device, cudaErrorNotSupported when there is no word to report it in
cudaError_t ts_refused(const TsDevice &d);
struct TsPlan { int nt, tiles_m, ksplit, waves; double cost; };
TsPlan ts_plan(int M, int N, int K, int span_bytes, int dequant_clocks, int split_min_rows, const TsDevice &d);

// clusters of n CTAs of this kernel that the device holds at once, n = 2 .. 8 (every type's kernel takes a whole SM)
void ts_count_clusters(int *out);    // mmq_ts_k4.cu

}  // namespace mrs
