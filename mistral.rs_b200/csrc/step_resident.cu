// step_resident.cu — one decode step of one sequence (all layers and the head) as ONE resident grid: a CTA per SM that stays for the whole step.
//
// What bounds a step as a chain of launches is not the weight stream (Llama-3-8B Q4_K_M: 131 MB a layer, 20 us of HBM) but its links: every GEMV
// starts with an empty ring, so each launch pays for its hand-off, its prologue and its ring's fill one after another (56 us a layer).  Here the
// producer warps walk through the weights of the whole step without regard to where the activations are: while the grid meets at a barrier and
// quantises the next input, the rings (200 KB a CTA, 30 MB over the GPU, 4.5 us of HBM) fill with the matrices that come next.
//
//   warps 0..15   consumers: rows of the products, two at a time (GLU: a gate row and its up row); between the products the small parts of the layer:
//                 RMSNorm and quantisation (every CTA for itself), RoPE, attention over the paged cache (a CTA per (KV head, tile of the step's plan))
//   warps 16..19  producers, one for four consumers: lane = (consumer warp, row of its pair), one cp.async.bulk a row segment into the group's ring
//
// A layer has five grid barriers: q / k / v, attention, o_proj, gate and up, down.  The grid is launched as a cooperative one, so all its CTAs run at
// the same time.  Every wait has a limit; one that runs out ends the grid (each CTA sees its copies land first), leaves NaN in the logits of each CTA that
// it stopped and sets the device's word (mrs_mmq_timeout_flag), after which steps are launched as a chain again.  The grid's own word of arrivals then
// stays RS_DEAD: a later launch with the same scratch (a replay passes no host code) leaves at its first meeting, its logits NaN, and sets the device's word
// again.  A runner's replay and mmq.check_timeouts look at that word.
//
// Every operation is the chain's, in its order, so the bits of logits and caches are the chain's too.  (They have to be: the 8-bit quants of a layer's five
// products blow up any difference, f32 sums in another order left eight layers' logits as far from the chain's as from exact ones.)
//
// One B200, bf16, us a step in a graph, chain / resident: eight layers 4096 x 14336 with a 32000 head, Q4_K_M, 500 tokens of context 535 / 439; 32 layers
// with a 128256 head 1878 / 1624; two layers at 100, 1000, 4000, 16000 tokens 164 / 151, 182 / 152, 195 / 170, 236 / 213, Q8_0 178 / 174, 197 / 179, 209 / 192,
// 249 / 234; four layers 3072 x 8192 at 20, 500, 3000 tokens 221 / 200, 235 / 205, 270 / 225.
// A layer of the first takes 91000 clocks (v and down in Q6_K: 102000), by stamps of each CTA: products until its last warp is done 55000 (65000), that is
// q / k / v 10100 (11600), o_proj 7200, gate and up 24700 (5.3 TB/s with what the ring held), down 12700 (21500); attention and the meetings on both sides
// of it 15500, a chain of loads in 56 of the CTAs that the others wait for; quantising the four inputs 14000 (1900 to 5200 each), in every CTA; the other
// meetings 6700.
// Tried: one producer warp for all rings (a copy took it 110 clocks: 713 us); consumers that ask for their own segments (480); vectors as words with tags
// instead of barriers (all CTAs polling the same lines took L2 from the weights: 530); rows brought into L2 ahead of the ring (nothing).
#include "mma_common.cuh"
#include "mmvq_types.cuh"
#include "mrs_b200_model.h"
#include "rope_common.cuh"

#include <stdio.h>
#include <string.h>
#include <type_traits>

extern "C" int32_t *mrs_mmq_timeout_flag(void);      // mmq_ts.cu: the device's word for waits that ran out

namespace mrs {

constexpr int RS_WARPS = 16, RS_CT = RS_WARPS * 32, RS_GROUP = 4, RS_PRODUCERS = RS_WARPS / RS_GROUP, RS_THREADS = RS_CT + 32 * RS_PRODUCERS;
constexpr int RS_LAYERS = 32;            // layers of a launch (its parameters hold their pointers); longer models take several
constexpr int RS_DEPTH = 8;              // stages of a group's ring in flight
constexpr int RS_TILES = 64;             // most tiles of a KV head
constexpr int RS_HEADER = 1024;          // barriers, offsets, small exchanges
// Narrower models: the meetings take longer than the chain's links (four layers 2048 wide at 20 tokens 155 us, 160 so).  Long tiles: their steps of 64 tokens
// are copied one at a time, two in the chain's kernel, so where KV heads leave a tile many tokens the chain is faster (two layers, chain / resident: 16 KV heads,
// 451 tokens a tile 183 / 176, Q8_0 195 / 196; 1784 tokens 257 / 261; 32 KV heads, 58 tokens 155 / 149, Q8_0 164 / 167, 268 tokens 176 / 182, 2016 tokens
// 263 / 281; 8 KV heads, 892 tokens 236 / 213).  Heads of 64: half the bytes a step for the same chain of loads, so half the tile (8 KV heads, three layers, resident /
// chain: 500 tokens a tile 0.99 at 2560 x 6912, 0.97 at 2560 x 10240 and 0.94 at 4096 x 14336, 778 tokens 1.03, 1.00 and 0.95, 1000 tokens 1.04, 1.02 and 0.96;
// Q8_0 0.03 to 0.06 above).  Close to the line Q8_0 may lose a few in a hundred: 2560 x 6912, 32 heads of 64 on 8, 1.00 to 1.05 at any length, and where the whole
// context is two tiles 1.02 to 1.08 up to 2816 wide or with heads of 64; 20 heads of 128 on 4 0.78 to 0.97.
constexpr int RS_MIN_HIDDEN = 2560, RS_MAX_KV_HEADS = 16, RS_MAX_TILE = 64;      // tile: tokens x KV heads for each element of a head
constexpr uint32_t RS_COPY_LIMIT = 1u << 22, RS_GRID_LIMIT = 1u << 22;      // polls (seconds)
constexpr uint32_t RS_DEAD = 1u << 31;   // in the word of arrivals: a wait of this step ran out, now or in a launch before (arrivals stay far below)

struct RsLayer {
  const uint8_t *w[7];                   // q, k, v, o, gate, up, down
  const void *attn_norm, *ffn_norm;
  void *kc, *vc;
  uint8_t type[5];                       // of the five products: q and k, v, o, gate and up, down
};
struct RsParams {
  RsLayer L[RS_LAYERS];
  const uint8_t *head;                   // null: a later launch has it
  const void *final_norm, *rope_cos, *rope_sin;
  const int32_t *positions;
  const int64_t *slots;
  const int32_t *kv_indptr, *kv_indices, *last_page, *tile_ends, *tile_size;
  void *x, *x2, *q, *k, *v, *attn, *act, *logits;
  float *part;                           // [tiles][heads][D], then two words a tile and head
  uint32_t *sync;                        // arrivals (or RS_DEAD), CTAs that are done, tiles of each KV head: zero between launches
  int *timeouts;
  float eps, scale_log2;
  int layers, hidden, inter, nq, nkv, heads, kv_heads, page_size, page_shift, vocab, head_type, interleaved, tiles;
  int x_bytes, ring;                     // bytes of the activation area, of a group's ring
};
static_assert(sizeof(RsParams) <= 4096, "parameters of a launch");

// What a lane multiplies of a segment, and the image of the activations for it.  Lanes, units of 32 weights and the order of the f32 operations are the
// vector kernel's (QT::dot behind Geo's map: lane = (block of eight, t), first unit t, then unit 4 + t of the block), so a row's bits are too; the integers
// are got at for less (both units' 6-bit scales unpacked together, quants used as they are stored, no conversions).
//   WORDS  16-byte words of activations of a lane      AUX  bytes of scales and sums behind them
//   place  where the 8 activations at element e (multiple of 8) of a block go: t, word, half of the word
//   side   what they add to the scales: d the block's scale, isum16 the sum of the 16 that they belong to
//
// Integers as f32 without conversions (which run at 4 lanes a clock and scheduler): sums start at 1.5 x 2^23 as f32 and stay within 2^22 of it; bytes on 2^23
constexpr int RS_MAGIC = 0x4B400000;
__device__ __forceinline__ float rs_sum(int v) { return __int_as_float(v) - 12582912.0f; }
template <int B> __device__ __forceinline__ float rs_byte(uint32_t v, float off = 8388608.0f) { return __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7440 + B)) - off; }
template <int T> struct RsUnit;
template <> struct RsUnit<MRS_Q4_K> {                               // d, dmin | scales[12] | qs[128]
  static constexpr int WORDS = 4, AUX = 32;
  struct X { int4 q[4]; float4 a[2]; };                             // of a unit: scales of its two Q8_1 blocks (the second / 16), scale times sum of its 16 of each
  __device__ static __forceinline__ void place(int e, int &t, int &word, int &half) {
    const int r = e & 63, c = 2 * (e >> 6) + ((r >> 4) & 1);
    t = c & 3; word = 2 * (c >> 2) + (r >> 5); half = (r >> 3) & 1;
  }
  __device__ static __forceinline__ void side(int e, float d, int isum16, uint8_t *aux, int npos, int pos) {
    const int hi = (e >> 5) & 1;
    float *const a = (float *)(aux + (e >> 7) * 16 * npos) + 4 * pos;
    if ((e & 15) == 0) { a[hi] = hi ? d * 0.0625f : d; a[2 + hi] = d * (float)isum16; }
  }
  __device__ static __forceinline__ void read(const uint8_t *aux, int npos, int pos, X &x) {
    x.a[0] = ((const float4 *)aux)[pos];
    x.a[1] = ((const float4 *)(aux + 16 * npos))[pos];
  }
  // (the products are integers below 2^24: exact, as the vector kernel's conversions of integer products are)
  __device__ static __forceinline__ float unit(const uint4 &q, const int4 &xl, const int4 &xh, const float4 &xa, uint32_t sc, uint32_t m, const float2 &dm) {
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
    const int l[4] = {xl.x, xl.y, xl.z, xl.w}, h[4] = {xh.x, xh.y, xh.z, xh.w};
    int lo = RS_MAGIC, hi = RS_MAGIC;                               // (the high nibbles stay in place: 16 times)
#pragma unroll
    for (int i = 0; i < 4; i++) {
      lo = __dp4a((int)(w[i] & 0x0F0F0F0Fu), l[i], lo);
      hi = dp4a_us(w[i] & 0xF0F0F0F0u, h[i], hi);
    }
    const float pl = __fmul_rn(rs_sum(lo), rs_byte<0>(sc)), ph = __fmul_rn(rs_sum(hi), rs_byte<1>(sc));
    const float sd = xa.x * pl + xa.y * ph;
    const float sm = xa.z * rs_byte<0>(m) + xa.w * rs_byte<1>(m);
    return dm.x * sd - dm.y * sm;
  }
  __device__ static __forceinline__ void add(float &acc, const uint8_t *blk, int t, const X &x) {
    const uint4 h = *(const uint4 *)blk, a = *(const uint4 *)(blk + 16 + 16 * t), b = *(const uint4 *)(blk + 80 + 16 * t);
    const int sh = 8 * (t & 2);
    const uint32_t A = h.y >> sh, B = h.z >> sh, C = h.w >> sh;
    const float2 dm = __half22float2(*(const __half2 *)&h.x);
    acc += unit(a, x.q[0], x.q[1], x.a[0], A & 0x3F3Fu, B & 0x3F3Fu, dm);
    acc += unit(b, x.q[2], x.q[3], x.a[1], (C & 0x0F0Fu) | ((A >> 2) & 0x3030u), ((C >> 4) & 0x0F0Fu) | ((B >> 2) & 0x3030u), dm);
  }
};
template <> struct RsUnit<MRS_Q6_K> {                               // ql[128] | qh[64] | int8 scales[16] | d
  static constexpr int WORDS = 4, AUX = 32;
  struct X { int4 q[4]; int4 off; float4 d; };                      // -32 times the sums of the units' 16s: the quants are used as they are stored
  __device__ static __forceinline__ void place(int e, int &t, int &word, int &half) {
    const int r = e & 127, r2 = r & 63;
    t = 2 * (r2 >> 5) + ((r2 >> 4) & 1); word = 2 * (e >> 7) + (r >> 6); half = (r2 >> 3) & 1;
  }
  __device__ static __forceinline__ void side(int e, float d, int isum16, uint8_t *aux, int npos, int pos) {
    const int i = 4 * pos + 2 * (e >> 7) + ((e >> 6) & 1);
    if ((e & 15) == 0) { ((int *)aux)[i] = RS_MAGIC - 32 * isum16; ((float *)(aux + 16 * npos))[i] = d; }
  }
  __device__ static __forceinline__ void read(const uint8_t *aux, int npos, int pos, X &x) {
    x.off = ((const int4 *)aux)[pos];
    x.d = ((const float4 *)(aux + 16 * npos))[pos];
  }
  __device__ static __forceinline__ float unit(const uint8_t *blk, int n, int t, const int4 &xl, const int4 &xh, int offl, int offh, float dl, float dh, float d) {
    uint32_t l[4], h[4];
    lds_words_unaligned<4>(blk + 64 * n + 16 * t, l);
    lds_words_unaligned<4>(blk + 128 + 32 * n + 16 * (t & 1), h);
    const uint8_t *const sc = blk + 192 + 8 * n + t;
    const int x0[4] = {xl.x, xl.y, xl.z, xl.w}, x1[4] = {xh.x, xh.y, xh.z, xh.w};
    // nibbles and the two bits above them apart: four masks a word instead of shifts and merges
    int lo = offl, lo2 = 0, hi = offh, hi16 = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t w = h[i] >> (t & 2);
      lo = __dp4a((int)(l[i] & 0x0F0F0F0Fu), x0[i], lo);
      lo2 = __dp4a((int)(w & 0x03030303u), x0[i], lo2);
      hi16 = dp4a_us(l[i] & 0xF0F0F0F0u, x1[i], hi16);
      hi = __dp4a((int)(w & 0x30303030u), x1[i], hi);
    }
    // (integers below 2^24: exact; scale bytes are signed, 128 up)
    const float a = __fmul_rn(rs_sum(lo + 16 * lo2), rs_byte<0>((uint32_t)sc[0] ^ 0x80u, 8388736.0f));
    const float b = __fmul_rn(rs_sum(hi + (hi16 >> 4)), rs_byte<0>((uint32_t)sc[4] ^ 0x80u, 8388736.0f));
    return d * (dl * a + dh * b);
  }
  __device__ static __forceinline__ void add(float &acc, const uint8_t *blk, int t, const X &x) {
    const float d = half_bits_to_float(lds_u16(blk + 208));
    acc += unit(blk, 0, t, x.q[0], x.q[1], x.off.x, x.off.y, x.d.x, x.d.y, d);
    acc += unit(blk, 1, t, x.q[2], x.q[3], x.off.z, x.off.w, x.d.z, x.d.w, d);
  }
};
template <> struct RsUnit<MRS_Q8_0> {                               // d | int8 qs[32]; lane = block
  static constexpr int WORDS = 2, AUX = 4;
  struct X { int4 q[2]; float d; };
  __device__ static __forceinline__ void place(int e, int &t, int &word, int &half) { t = 0; word = e >> 4; half = (e >> 3) & 1; }
  __device__ static __forceinline__ void side(int e, float d, int, uint8_t *aux, int, int pos) { if (e == 0) ((float *)aux)[pos] = d; }
  __device__ static __forceinline__ void read(const uint8_t *aux, int, int pos, X &x) { x.d = ((const float *)aux)[pos]; }
  __device__ static __forceinline__ void add(float &acc, const uint8_t *blk, int, const X &x) {
    uint32_t q[8];
    lds_words_unaligned<8>(blk + 2, q);
    const int *xq = (const int *)&x.q[0];
    int s = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) s = __dp4a((int)q[i], xq[i], s);
    acc += (float)s * half_bits_to_float(lds_u16(blk)) * x.d;
  }
};

// geometry of a type's row segments
template <int T> struct RsGeo {
  using Q = QT<T>;
  using U = RsUnit<T>;
  static constexpr int SEG_BLOCKS = Q::UPB == 1 ? 32 : 8, SEG_BYTES = SEG_BLOCKS * Q::BYTES;
  static constexpr bool ALIGNED = Q::WALIGN == 16;                  // rows start on 16-byte boundaries
  static constexpr int SLOT = ALIGNED ? SEG_BYTES : (SEG_BYTES + 30 + 15) & ~15;
  __host__ __device__ static constexpr int npos(int K) { return ((K / Q::QK + SEG_BLOCKS - 1) / SEG_BLOCKS) * 32; }
  __host__ __device__ static constexpr int image(int K) { return npos(K) * (16 * U::WORDS + U::AUX); }
  __device__ static __forceinline__ int pos(int blk, int t) { return 32 * (blk / SEG_BLOCKS) + blk % SEG_BLOCKS + 8 * t; }
};
#define RS_TYPES(F) F(MRS_Q4_K) F(MRS_Q6_K) F(MRS_Q8_0)
__host__ __device__ inline bool rs_type_ok(int t) { return t == MRS_Q4_K || t == MRS_Q6_K || t == MRS_Q8_0; }
struct RsType { int seg, slot, block, weights; };      // bytes of a segment, of its slot, of a block; weights of a block
__host__ __device__ inline RsType rs_type(int t) {
  switch (t) {
#define RS_CASE(T) case T: return RsType{RsGeo<T>::SEG_BYTES, RsGeo<T>::SLOT, QT<T>::BYTES, QT<T>::QK};
    RS_TYPES(RS_CASE)
#undef RS_CASE
  default: return RsType{16, 16, 16, 32};
  }
}
__host__ __device__ inline int rs_image(int t, int K) {
  switch (t) {
#define RS_CASE(T) case T: return RsGeo<T>::image(K);
    RS_TYPES(RS_CASE)
#undef RS_CASE
  default: return 0;
  }
}

enum { RS_QK = 0, RS_V = 1, RS_O = 2, RS_GU = 3, RS_DOWN = 4, RS_HEAD = 5 };

// Product `i` of the launch: five a layer, then the head.  A CTA's share is a range of pairs of rows.
struct RsOp {
  const uint8_t *w0, *w1;
  int kind, type, K, n0, n1, first, count, turn;      // rows of w0 and w1; pairs [first, first + count); the warp that takes the first
};
__device__ __forceinline__ RsOp rs_op(const RsParams &p, int i) {
  RsOp o;
  const int l = i / 5, k = i - 5 * l, cta = (int)blockIdx.x, n = (int)gridDim.x;
  o.w1 = nullptr; o.n1 = 0; o.turn = 0; o.K = p.hidden;
  if (l == p.layers) { o.kind = RS_HEAD; o.type = p.head_type; o.w0 = p.head; o.n0 = p.vocab; }
  else {
    const RsLayer &L = p.L[l];
    o.kind = k; o.type = L.type[k];
    switch (k) {
    case RS_QK: o.w0 = L.w[0]; o.w1 = L.w[1]; o.n0 = p.nq; o.n1 = p.nkv; break;
    case RS_V: {
      const int pairs = (p.nq + p.nkv) >> 1;          // (of q and k: the warps take v's in turn behind them)
      o.w0 = L.w[2]; o.n0 = p.nkv; o.turn = (int)((uint32_t)(pairs * (cta + 1)) / (uint32_t)n - (uint32_t)(pairs * cta) / (uint32_t)n) % RS_WARPS;
      break;
    }
    case RS_O: o.w0 = L.w[3]; o.n0 = p.hidden; o.K = p.nq; break;
    case RS_GU: o.w0 = L.w[4]; o.w1 = L.w[5]; o.n0 = p.inter; break;
    default: o.w0 = L.w[6]; o.n0 = p.hidden; o.K = p.inter; break;
    }
  }
  const int pairs = o.kind == RS_GU ? o.n0 : (o.n0 + o.n1 + 1) >> 1;
  o.first = (int)((uint32_t)(pairs * cta) / (uint32_t)n);       // (the host checks that the products fit)
  o.count = (int)((uint32_t)(pairs * (cta + 1)) / (uint32_t)n) - o.first;
  return o;
}
// row r (0, 1) of pair i, or null where the last pair has one row
__device__ __forceinline__ const uint8_t *rs_row(const RsOp &o, int i, int r, int row_bytes) {
  if (o.kind == RS_GU) return (r ? o.w1 : o.w0) + (size_t)i * row_bytes;
  const int row = 2 * i + r;
  if (row < o.n0) return o.w0 + (size_t)row * row_bytes;
  return row - o.n0 < o.n1 ? o.w1 + (size_t)(row - o.n0) * row_bytes : nullptr;
}

struct RsShared {
  uint64_t full[RS_PRODUCERS][RS_DEPTH], empty[RS_PRODUCERS][RS_DEPTH];
  uint32_t ends[RS_PRODUCERS][RS_DEPTH];      // of the stages in flight, for their producer
  float red[8];
  int stop;                              // a wait ran out
  int last;                              // this CTA is the last one with a split of its head
  int go;                                // what thread 0 found at the last barrier of the grid
};
static_assert(sizeof(RsShared) <= RS_HEADER, "header");


// ---------------------------------------------------------------- producers
// A group is a producer warp and four consumer warps.  In a round of a product each of the four takes a pair of rows (or none, at the end of the CTA's
// share); a stage is a segment of all of the round's rows, and the group's stages go round in a ring of bytes.
struct RsStage { uint32_t pos, seq; };      // end of the last stage, stages so far
__device__ __forceinline__ uint32_t rs_place(const RsStage &r, uint32_t size, int ring) { return r.pos + size > (uint32_t)ring ? 0u : r.pos; }
__device__ __forceinline__ int rs_rounds(const RsOp &o, int group) {      // (the warp whose turn is first takes the share's first pair)
  int first = RS_WARPS;                    // the group's earliest place in the order of the warps
#pragma unroll
  for (int i = 0; i < RS_GROUP; i++) first = min(first, (RS_GROUP * group + i - o.turn) & (RS_WARPS - 1));
  return o.count > first ? (o.count - first + RS_WARPS - 1) / RS_WARPS : 0;
}
__device__ __forceinline__ void rs_produce(const RsParams &p, RsShared &sh, uint8_t *ring, int group, int lane) {
  const int w = RS_GROUP * group + (lane & (RS_GROUP - 1)), r = (lane / RS_GROUP) & 1, ops = 5 * p.layers + (p.head != nullptr ? 1 : 0);
  RsStage head = {0u, 0u}, tail = {0u, 0u};          // newest stage; oldest stages that were released, by their ends
  uint32_t *const ends = sh.ends[group];
  bool dead = false;
  int tries = 0;
  for (int op = 0; op < ops; op++) {
    const RsOp o = rs_op(p, op);
    const RsType t = rs_type(o.type);
    const int row_bytes = o.K / t.weights * t.block, rounds = rs_rounds(o, group), mine = (w - o.turn) & (RS_WARPS - 1);
    const uint32_t size = 2u * RS_GROUP * (uint32_t)t.slot;
    for (int j = 0; j < rounds; j++) {
      const int at_pair = mine + RS_WARPS * j;
      const uint8_t *row = lane < 2 * RS_GROUP && at_pair < o.count ? rs_row(o, o.first + at_pair, r, row_bytes) : nullptr;
      for (int off = 0; off < row_bytes; off += t.seg) {
        const uint32_t at = rs_place(head, size, p.ring);
        // free is what lies behind the newest stage, up to the end of the last one that was released (in the ring's order)
        while (!dead) {
          const uint32_t held = head.seq - tail.seq;
          if (held == 0 || (held < RS_DEPTH && (head.pos > tail.pos ? (at == head.pos || size <= tail.pos) : (at == head.pos && head.pos + size <= tail.pos)))) break;
          const bool free = mbar_wait_warp(&sh.empty[group][tail.seq & (RS_DEPTH - 1)], (tail.seq / RS_DEPTH) & 1, RS_COPY_LIMIT / 256);
          if (!__all_sync(0xffffffffu, free)) {
            if (++tries == 256 || *(volatile int *)&sh.stop) dead = true;
            continue;
          }
          tries = 0;
          tail.pos = ends[tail.seq & (RS_DEPTH - 1)]; tail.seq++;
        }
        dead = __any_sync(0xffffffffu, dead || *(volatile int *)&sh.stop);
        if (dead) break;
        const int slot = (int)(head.seq & (RS_DEPTH - 1)), n = min(t.seg, row_bytes - off);
        if (lane < 2 * RS_GROUP) {
          if (row != nullptr) {
            const uintptr_t a = (uintptr_t)(row + off), a0 = a & ~(uintptr_t)15;
            const uint32_t bytes = (uint32_t)(((a + n + 15) & ~(uintptr_t)15) - a0);
            mbar_arrive_expect_tx(&sh.full[group][slot], bytes);
            bulk_g2s(ring + at + (2 * (lane & (RS_GROUP - 1)) + r) * t.slot, (const void *)a0, bytes, &sh.full[group][slot]);
          } else mbar_arrive(&sh.full[group][slot]);
        }
        head.pos = at + size;
        if (lane == 0) ends[slot] = head.pos;
        __syncwarp();
        head.seq++;
      }
      if (dead) break;
    }
    if (dead) break;
  }
  // no CTA ends before its copies have landed
  for (tail.seq = head.seq > RS_DEPTH ? head.seq - RS_DEPTH : 0u; tail.seq != head.seq; tail.seq++) mbar_wait_warp(&sh.full[group][tail.seq & (RS_DEPTH - 1)], (tail.seq / RS_DEPTH) & 1, RS_COPY_LIMIT);
}

// ---------------------------------------------------------------- consumers
struct RsRing { RsStage at; uint32_t polls; bool gives; };      // where the warp reads; its waits' limit; the lane gives stages back (the first, until a wait ran out)

__device__ __forceinline__ void rs_bar() { asm volatile("bar.sync 1, %0;" ::"n"(RS_CT) : "memory"); }

// Everything that the grid's CTAs wrote before their arrival is seen behind the wait.  Between the two a CTA may start on what no other CTA writes.
__device__ __forceinline__ void rs_arrive(const RsParams &p, int tid) {
  rs_bar();
  if (tid == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p.sync) : "memory");
}
__device__ __forceinline__ bool rs_meet(const RsParams &p, RsShared &sh, uint32_t &round, int tid) {
  round += gridDim.x;
  if (tid == 0) {
    uint32_t n = *(volatile int *)&sh.stop ? RS_GRID_LIMIT : 0u, seen;
    for (;; n++) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(p.sync) : "memory");
      if (n >= RS_GRID_LIMIT || (seen & RS_DEAD) || seen >= round) break;
    }
    sh.go = n < RS_GRID_LIMIT && !(seen & RS_DEAD);          // (one thread's finding: all of the CTA's threads leave, or none)
  }
  rs_bar();
  return *(volatile int *)&sh.go != 0;
}

// The CTA leaves a step that is lost: its own copies have landed (the producers see to theirs), its rows of the logits are NaN, and the word of arrivals
// sends the other CTAs, and launches to come, the same way.  A lost step is not counted as done, so nothing makes the word zero again.
__device__ __forceinline__ void rs_lost(const RsParams &p, RsShared &sh, int dt, int tid) {
  if (tid == 0) {
    *(volatile int *)&sh.stop = 1;
    *(volatile int *)p.timeouts = 1;
    atomicExch(p.sync, RS_DEAD);
  }
  cp_async_wait<0>();
  if (p.head == nullptr) return;         // (the launch behind this one has the head)
  const RsOp o = rs_op(p, 5 * p.layers);
  for (int row = 2 * o.first + tid; row < min(2 * (o.first + o.count), p.vocab); row += RS_CT) store_act(p.logits, row, __int_as_float(0x7FC00000), dt);
}

template <typename T> __device__ __forceinline__ void rs_unpack8(const uint4 &v, float *f) {
  unpack_act8(v, std::is_same<T, __half>::value ? MRS_F16 : MRS_BF16, f);
}
template <typename T> __device__ __forceinline__ uint32_t rs_one_bits(const void *p, int64_t i) { return __ldcg((const unsigned short *)p + i); }
template <typename T> __device__ __forceinline__ float rs_one(uint32_t bits) {
  const unsigned short b = (unsigned short)bits;
  T t;
  memcpy(&t, &b, 2);
  return (float)t;
}

// one 8-element chunk (four neighbouring lanes are a Q8_1 block) into the activation image of a type: mmvq.cu's fused prologue
template <int TYPE> __device__ __forceinline__ void rs_store_chunk(uint8_t *img, int K, int e0, const uint32_t (&wq)[2], float d, int isum16) {
  using U = RsUnit<TYPE>;
  using G = RsGeo<TYPE>;
  const int npos = G::npos(K), blk = e0 / QT<TYPE>::QK, e = e0 - blk * QT<TYPE>::QK;
  int t, word, half;
  U::place(e, t, word, half);
  const int pos = G::pos(blk, t);
  *((int2 *)(img + (size_t)(word * npos + pos) * 16) + half) = make_int2((int)wq[0], (int)wq[1]);
  U::side(e, d, isum16, img + (size_t)npos * 16 * U::WORDS, npos, pos);
}

// (a lane whose wait ran out gives no stage back from then on: copies may be on their way still, and the producer waits for them at its end)
__device__ __forceinline__ void rs_landed(RsShared &sh, RsRing &rr, int group, int slot) {
  if (!mbar_wait_warp(&sh.full[group][slot], (rr.at.seq / RS_DEPTH) & 1, rr.polls)) {
    rr.polls = 1u;
    rr.gives = false;
    *(volatile int *)&sh.stop = 1;
  }
}
// A pair of rows after another of the CTA's share of a product.
template <int TYPE, typename T>
__device__ __forceinline__ void rs_gemv(const RsParams &p, const RsOp &o, RsShared &sh, const uint8_t *img, const uint8_t *ring, RsRing &rr, int warp, int lane) {
  using Q = QT<TYPE>;
  using U = RsUnit<TYPE>;
  using G = RsGeo<TYPE>;
  constexpr int DT = std::is_same<T, __half>::value ? MRS_F16 : MRS_BF16;
  const int nblocks = o.K / Q::QK, nseg = (nblocks + G::SEG_BLOCKS - 1) / G::SEG_BLOCKS, npos = G::npos(o.K), row_bytes = nblocks * Q::BYTES;
  const int4 *xq = (const int4 *)img;
  const uint8_t *aux = img + (size_t)npos * 16 * U::WORDS;
  const int lblk = lane % G::SEG_BLOCKS, t = lane / G::SEG_BLOCKS;
  const void *residual = o.kind == RS_O ? p.x : o.kind == RS_DOWN ? p.x2 : nullptr;
  const int group = warp / RS_GROUP, rounds = rs_rounds(o, group), mine = (warp - o.turn) & (RS_WARPS - 1);
  const uint32_t size = 2u * RS_GROUP * G::SLOT;
  for (int j = 0; j < rounds; j++) {
    const int pair = o.first + mine + RS_WARPS * j;
    if (mine + RS_WARPS * j >= o.count) {        // a round without rows for this warp
      for (int s = 0; s < nseg; s++) {
        const int slot = (int)(rr.at.seq & (RS_DEPTH - 1));
        rs_landed(sh, rr, group, slot);
        if (rr.gives) mbar_arrive(&sh.empty[group][slot]);
        rr.at.pos = rs_place(rr.at, size, p.ring) + size; rr.at.seq++;
      }
      continue;
    }
    uint32_t res = 0;
    if (residual != nullptr && lane < 2 && 2 * pair + lane < o.n0) res = rs_one_bits<T>(residual, 2 * pair + lane);
    uint32_t ph0 = 0, ph1 = 0;
    if constexpr (!G::ALIGNED) {
      ph0 = (uint32_t)(uintptr_t)rs_row(o, pair, 0, row_bytes);
      ph1 = (uint32_t)(uintptr_t)rs_row(o, pair, 1, row_bytes);      // (of a row that is not there: its results are not stored)
    }
    float acc0 = 0.f, acc1 = 0.f;
    const uint32_t rows_at = 2u * (uint32_t)(warp & (RS_GROUP - 1)) * G::SLOT + (uint32_t)(lblk * Q::BYTES);
    for (int s = 0; s < nseg; s++) {
      const int slot = (int)(rr.at.seq & (RS_DEPTH - 1));
      const uint32_t at = rs_place(rr.at, size, p.ring), sp = (uint32_t)(s * G::SEG_BYTES);
      rs_landed(sh, rr, group, slot);
      const uint8_t *wp0 = ring + at + rows_at + (G::ALIGNED ? 0u : ((ph0 + sp) & 15u));
      const uint8_t *wp1 = ring + at + rows_at + G::SLOT + (G::ALIGNED ? 0u : ((ph1 + sp) & 15u));
      if (s * G::SEG_BLOCKS + lblk < nblocks) {
        const int pos = 32 * s + lane;
        typename U::X x;
#pragma unroll
        for (int i = 0; i < U::WORDS; i++) x.q[i] = xq[i * npos + pos];
        U::read(aux, npos, pos, x);
        U::add(acc0, wp0, t, x);
        U::add(acc1, wp1, t, x);
      }
      __syncwarp();
      if (rr.gives) mbar_arrive(&sh.empty[group][slot]);
      rr.at.pos = at + size; rr.at.seq++;
    }
    // both rows' sums in one butterfly: lanes 0..15 the first's, 16..31 the second's
    float v = (lane & 16 ? acc1 : acc0) + __shfl_xor_sync(0xffffffffu, lane & 16 ? acc0 : acc1, 16);
#pragma unroll
    for (int m = 8; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
    const float other = __shfl_xor_sync(0xffffffffu, v, 16);
    if (o.kind == RS_GU) {
      if (lane == 0) {
        const float g = round_act(v, DT), up = round_act(other, DT);
        store_act(p.act, pair, round_act(glu_activation(g, 0), DT) * up, DT);
      }
    } else if (lane < 2) {
      const int row = 2 * pair + lane;
      if (lane) v = other;
      if (residual != nullptr) v = round_act(v, DT) + rs_one<T>(res);
      if (row < o.n0) store_act(o.kind == RS_QK ? p.q : o.kind == RS_V ? p.v : o.kind == RS_O ? p.x2 : o.kind == RS_DOWN ? p.x : p.logits, row, v, DT);
      else if (row - o.n0 < o.n1) store_act(p.k, row - o.n0, v, DT);
    }
  }
}

// The input of a product, with its RMSNorm, quantised into the images of the types that read it (two where attn_v has a type of its own).  The norm's sums
// in the order of mmvq.cu's fused prologue.
constexpr int RS_OWN = 4;                  // chunks of eight that a thread holds: all on their way before the first is needed
template <typename T>
__device__ __forceinline__ void rs_quantise(const RsParams &p, const RsOp &o, RsShared &sh, int type2, const void *norm_w, const uint4 &nw0,
                                            uint8_t *img, int tid, int warp, int lane) {
  constexpr int DT = std::is_same<T, __half>::value ? MRS_F16 : MRS_BF16;
  const int K = o.K, nchunks = K >> 3, nchunks_w = (nchunks + 31) & ~31;
  const uint4 *x = (const uint4 *)(o.kind == RS_O ? p.attn : o.kind == RS_GU ? p.x2 : o.kind == RS_DOWN ? p.act : p.x);
  float inv_rms = 1.0f;
  uint4 own[RS_OWN];
#pragma unroll
  for (int i = 0; i < RS_OWN; i++) {
    own[i] = make_uint4(0u, 0u, 0u, 0u);
    if (tid + i * RS_CT < nchunks) own[i] = __ldcg(x + tid + i * RS_CT);
  }
  if (norm_w != nullptr) {
    if (tid < 256) {
      const bool two = tid + 256 < nchunks;
      uint4 next = make_uint4(0u, 0u, 0u, 0u);
      if (two) next = __ldcg(x + tid + 256);
      float ss = 0.f, v[8];
      rs_unpack8<T>(own[0], v);
#pragma unroll
      for (int e = 0; e < 8; e++) ss = fmaf(v[e], v[e], ss);
      rs_unpack8<T>(next, v);
#pragma unroll
      for (int e = 0; e < 8; e++) ss = fmaf(v[e], v[e], ss);
      for (int i = tid + 512; i < nchunks; i += 256) {
        rs_unpack8<T>(__ldcg(x + i), v);
#pragma unroll
        for (int e = 0; e < 8; e++) ss = fmaf(v[e], v[e], ss);
      }
      ss = warp_sum(ss);
      if (lane == 0) sh.red[warp] = ss;
    }
    rs_bar();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) tot += sh.red[i];
    inv_rms = rsqrtf(tot / (float)K + p.eps);
  }
  uint8_t *const img2 = img + rs_image(o.type, K);
#pragma unroll 1
  for (int ch = tid; ch < nchunks_w; ch += RS_CT) {
    const bool ok = ch < nchunks;
    const uint4 now = own[0];
#pragma unroll
    for (int i = 0; i + 1 < RS_OWN; i++) own[i] = own[i + 1];
    own[RS_OWN - 1] = make_uint4(0u, 0u, 0u, 0u);
    if (ch + RS_OWN * RS_CT < nchunks) own[RS_OWN - 1] = __ldcg(x + ch + RS_OWN * RS_CT);
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = 0.f;
    if (ok) {
      rs_unpack8<T>(now, v);
      if (norm_w != nullptr) {
        float wv[8];
        rs_unpack8<T>(ch == tid ? nw0 : __ldg((const uint4 *)norm_w + ch), wv);
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = round_act(v[i] * inv_rms * wv[i], DT);
      }
    }
    float am = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) am = fmaxf(am, fabsf(v[i]));
    am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 1));
    am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 2));
    const float d = __fdividef(am, 127.0f);
    uint32_t qi[8], wq[2];
#pragma unroll
    for (int i = 0; i < 8; i++) {           // (half away from zero: adding a half towards zero crosses no integer that the sum itself does not reach)
      const float t = __fdividef(v[i], d);
      qi[i] = am == 0.0f ? 0u : (uint32_t)(int)__fadd_rz(t, copysignf(0.5f, t));
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
      wq[i] = __byte_perm(__byte_perm(qi[4 * i], qi[4 * i + 1], 0x0040), __byte_perm(qi[4 * i + 2], qi[4 * i + 3], 0x0040), 0x5410);
    const int isum8 = __dp4a((int)wq[0], 0x01010101, __dp4a((int)wq[1], 0x01010101, 0));
    const int isum16 = isum8 + __shfl_xor_sync(0xffffffffu, isum8, 1);
    if (ok) {
      const float dr = __half2float(__float2half_rn(d));
      uint8_t *to = img;
      for (int type = o.type;; type = type2, to = img2) {
        switch (type) {
#define RS_CASE(TY) case TY: rs_store_chunk<TY>(to, K, 8 * ch, wq, dr, isum16); break;
          RS_TYPES(RS_CASE)
#undef RS_CASE
        }
        if (to == img2 || type2 == o.type) break;
      }
    }
  }
  rs_bar();
}

// Attention of the CTA's (KV head, tile): the decode attention kernel's arithmetic (paged_attn_mma.cuh, FUSED), operation for operation.  Of a step of 64
// tokens, warps w and w + 4 have tokens 16 w .. and, for all of them, the scores, each for half of the head's dimensions the sums: the accumulators of a
// whole head do not fit beside what the step's other parts keep.  The tiles' states meet in memory: the last CTA of a head adds them up, in tile order, as the
// kernel's cluster does (up to PM_CL_MAX tiles), or its last tile (more).  The cache rows of the first 64 tokens are asked for before the barrier that brings
// q.  Returns false where the barrier ran out.
template <int D> constexpr int rs_attend_bytes() { return 2 * 64 * D * 2 + 3 * 16 * D * 2 + 2 * 64 * 4; }
template <typename T, int D>
__device__ __forceinline__ bool rs_attend(const RsParams &p, const RsLayer &L, RsShared &sh, uint8_t *area, uint32_t &round, int tiles, int chunk, int kv_len,
                                          int page0, int tid, int warp, int lane) {
  constexpr int DT = std::is_same<T, __half>::value ? MRS_F16 : MRS_BF16;
  constexpr int KSTEPS = D / 16, LPT = D / 8, CPR = D / 8, HT = D / 16;      // HT: 8-wide output columns of half a head
  uint8_t *const sk = area, *const sv = sk + 64 * D * 2, *const sq = sv + 64 * D * 2, *const snk = sq + 16 * D * 2, *const snv = snk + 16 * D * 2;
  float *const mm = (float *)(snv + 16 * D * 2), *const ml = mm + 64;        // [4 warps][16 rows]
  const int kvh = (int)blockIdx.x % p.kv_heads, tile = (int)blockIdx.x / p.kv_heads, G = p.heads / p.kv_heads, h0 = kvh * G;
  const bool mine = tile < tiles;
  const int t_begin = tile * chunk, t_end = min(kv_len, t_begin + chunk);
  const bool owns_new = mine && kv_len - 1 >= t_begin && kv_len - 1 < t_end;
  const int t_cache = owns_new ? kv_len - 1 : t_end, steps = mine && t_cache > t_begin ? (t_cache - t_begin + 63) / 64 : 0;
  const int64_t row = (int64_t)p.page_size * D, block = row * p.kv_heads;
  const T *const kc = (const T *)L.kc + kvh * row, *const vc = (const T *)L.vc + kvh * row;
  auto ask = [&](int it) {
#pragma unroll
    for (int i = tid; i < 64 * CPR; i += RS_CT) {
      const int r = i / CPR, ch = i % CPR, t = t_begin + 64 * it + r;
      const bool ok = t < t_cache;
      int64_t at = 0;
      if (ok) {
        const int pg = p.page_shift >= 0 ? t >> p.page_shift : t / p.page_size, in = p.page_shift >= 0 ? t & (p.page_size - 1) : t - pg * p.page_size;
        at = (int64_t)__ldg(p.kv_indices + page0 + pg) * block + (int64_t)in * D + ch * 8;
      }
      cp_async16(sk + tile_off<D>(r, ch), kc + at, ok);
      cp_async16(sv + tile_off<D>(r, ch), vc + at, ok);
    }
    cp_async_commit();
  };
  int slot = -1;
  const T *cosp = nullptr, *sinp = nullptr;
  if (mine) {
    if (steps > 0) ask(0);
    for (int i = tid; i < 2 * 16 * D * 2 / 16; i += RS_CT) ((uint4 *)snk)[i] = make_uint4(0u, 0u, 0u, 0u);
    const int64_t pos = __ldg(p.positions);
    cosp = (const T *)p.rope_cos + pos * (D / 2);
    sinp = (const T *)p.rope_sin + pos * (D / 2);
    slot = (int)__ldg((const int32_t *)p.slots);          // (low word: no cache of 2^31 rows fits the GPU)
  }
  if (!rs_meet(p, sh, round, tid)) return false;
  if (!mine) return true;

  if (tid < 16 * LPT) {                               // (whole warps) rows = heads of the group
    const int g = tid / LPT, gl = tid % LPT;
    float x[8];
#pragma unroll
    for (int i = 0; i < 8; i++) x[i] = 0.f;
    if (g < G) rs_unpack8<T>(__ldcg((const uint4 *)((const T *)p.q + (int64_t)(h0 + g) * D) + gl), x);
    rope_any<T, D>(x, cosp, sinp, gl, p.interleaved != 0);
    Vec8<T>::store((T *)(sq + tile_off<D>(g, gl)), x);
  } else if (owns_new && warp == RS_WARPS - 1) {      // the new token: attended from shared memory, its cache rows written on the side
    const int gl = lane % LPT;
    float kn[8], vn[8];
    rs_unpack8<T>(__ldcg((const uint4 *)((const T *)p.k + kvh * D) + gl), kn);
    rs_unpack8<T>(__ldcg((const uint4 *)((const T *)p.v + kvh * D) + gl), vn);
    rope_any<T, D>(kn, cosp, sinp, gl, p.interleaved != 0);
    if (lane < LPT) {
      Vec8<T>::store((T *)(snk + tile_off<D>(0, gl)), kn);
      Vec8<T>::store((T *)(snv + tile_off<D>(0, gl)), vn);
      if (slot >= 0) {
        const int pg = p.page_shift >= 0 ? slot >> p.page_shift : slot / p.page_size;
        const int64_t at = pg * block + kvh * row + (int64_t)(slot - pg * p.page_size) * D + gl * 8;
        Vec8<T>::store((T *)L.kc + at, kn);
        Vec8<T>::store((T *)L.vc + at, vn);
      }
    }
  }
  float oacc[HT][4];
#pragma unroll
  for (int i = 0; i < HT; i++) { oacc[i][0] = oacc[i][1] = oacc[i][2] = oacc[i][3] = 0.f; }
  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
  const int w4 = warp & 3, dhalf = (warp >> 2) & 1;
  // 16 tokens in rows row0 .. of (kt, vt), token of row j t_first + j, live below t_hi
  auto step16 = [&](const uint8_t *kt, const uint8_t *vt, int row0, int t_first, int t_hi) {
    float sacc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ks++) {
      uint32_t qa[4], b0, b1, b2, b3;
      ldsm_x4(smem_u32(sq + tile_off<D>(lane & 15, 2 * ks + (lane >> 4))), qa[0], qa[1], qa[2], qa[3]);
      ldsm_x4(smem_u32(kt + tile_off<D>(row0 + (lane & 7) + ((lane >> 4) << 3), 2 * ks + ((lane >> 3) & 1))), b0, b1, b2, b3);
      mma16816<T>(sacc[0], qa, b0, b1);
      mma16816<T>(sacc[1], qa, b2, b3);
    }
    float mx[2] = {m_run[0], m_run[1]};
#pragma unroll
    for (int j = 0; j < 2; j++) {
#pragma unroll
      for (int e = 0; e < 4; e++) {
        float s = sacc[j][e];
        s *= p.scale_log2;
        const int t = t_first + 8 * j + 2 * (lane & 3) + (e & 1);
        if (t >= t_hi) s = -INFINITY;
        sacc[j][e] = s;
        mx[e >> 1] = fmaxf(mx[e >> 1], s);
      }
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
    }
    float corr[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
      corr[r] = (mx[r] == -INFINITY) ? 1.f : exp2f(m_run[r] - mx[r]);
      m_run[r] = mx[r];
    }
    uint32_t pa[4];
    float rs[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const float p0 = (mx[0] == -INFINITY) ? 0.f : exp2f(sacc[j][0] - mx[0]);
      const float p1 = (mx[0] == -INFINITY) ? 0.f : exp2f(sacc[j][1] - mx[0]);
      const float p2 = (mx[1] == -INFINITY) ? 0.f : exp2f(sacc[j][2] - mx[1]);
      const float p3 = (mx[1] == -INFINITY) ? 0.f : exp2f(sacc[j][3] - mx[1]);
      rs[0] += p0 + p1; rs[1] += p2 + p3;
      pa[2 * j] = pack2<T>(p0, p1);
      pa[2 * j + 1] = pack2<T>(p2, p3);
    }
#pragma unroll
    for (int r = 0; r < 2; r++) l_run[r] = l_run[r] * corr[r] + rs[r];
#pragma unroll
    for (int i = 0; i < HT; i++) { oacc[i][0] *= corr[0]; oacc[i][1] *= corr[0]; oacc[i][2] *= corr[1]; oacc[i][3] *= corr[1]; }
#pragma unroll
    for (int dp = 0; dp < HT / 2; dp++) {
      uint32_t b0, b1, b2, b3;
      ldsm_x4_t(smem_u32(vt + tile_off<D>(row0 + (lane & 7) + (((lane >> 3) & 1) << 3), HT * dhalf + 2 * dp + (lane >> 4))), b0, b1, b2, b3);
      mma16816<T>(oacc[2 * dp], pa, b0, b1);
      mma16816<T>(oacc[2 * dp + 1], pa, b2, b3);
    }
  };
#pragma unroll 1
  for (int it = 0; it < steps; it++) {
    if (it > 0) {
      rs_bar();                                       // the rows of the last step have been read
      ask(it);
    }
    cp_async_wait<0>();
    rs_bar();
    const int tw = t_begin + 64 * it + 16 * w4;
    if (warp < 8 && tw < t_cache) step16(sk, sv, 16 * w4, tw, t_cache);
  }
  if (steps == 0) rs_bar();                           // the new token and q are there
  if (owns_new && warp < 8 && w4 == 0) step16(snk, snv, 0, kv_len - 1, kv_len);
#pragma unroll
  for (int r = 0; r < 2; r++) {
    l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 1);
    l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 2);
  }
  rs_bar();                                           // the warps' states go where the rows were
  float *const mo = (float *)area;                    // [4 warps][16][D]
  if (warp < 8) {
    const int r0 = lane >> 2;
#pragma unroll
    for (int i = 0; i < HT; i++) {
      const int col = D / 2 * dhalf + 8 * i + 2 * (lane & 3);
      *(float2 *)(mo + ((size_t)w4 * 16 + r0) * D + col) = make_float2(oacc[i][0], oacc[i][1]);
      *(float2 *)(mo + ((size_t)w4 * 16 + r0 + 8) * D + col) = make_float2(oacc[i][2], oacc[i][3]);
    }
    if (dhalf == 0 && (lane & 3) == 0) {
      mm[w4 * 16 + r0] = m_run[0]; mm[w4 * 16 + r0 + 8] = m_run[1];
      ml[w4 * 16 + r0] = l_run[0]; ml[w4 * 16 + r0 + 8] = l_run[1];
    }
  }
  rs_bar();
  // what a tile leaves: up to PM_CL_MAX tiles sums, maximum and sum of probabilities (base 2), beyond results as tensors hold them and a natural logarithm
  float2 *const state = (float2 *)(p.part + (size_t)p.tiles * p.heads * D);
  const bool whole = p.tiles <= PM_CL_MAX;
  for (int idx = tid; idx < G * D; idx += RS_CT) {
    const int g = idx / D, d = idx % D;
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; w++) M = fmaxf(M, mm[w * 16 + g]);
    float Ls = 0.f, acc = 0.f;
    if (M > -INFINITY) {
#pragma unroll
      for (int w = 0; w < 4; w++) {
        const float c = exp2f(mm[w * 16 + g] - M);
        Ls += ml[w * 16 + g] * c;
        acc += mo[((size_t)w * 16 + g) * D + d] * c;
      }
    }
    float *const to = p.part + ((size_t)tile * p.heads + h0 + g) * D + d;
    if (p.tiles > 1 && whole) {
      *to = acc;
      if (d == 0) state[(size_t)tile * p.heads + h0 + g] = make_float2(M, Ls);
    } else {
      const float val = (Ls > 0.f) ? acc / Ls : 0.f;
      if (p.tiles > 1) {
        *to = round_act(val, DT);
        if (d == 0) state[(size_t)tile * p.heads + h0 + g] = make_float2((Ls > 0.f) ? (M + log2f(Ls)) * 0.6931471805599453f : -INFINITY, 0.f);
      } else store_act(p.attn, (h0 + g) * D + d, val, DT);
    }
  }
  if (p.tiles == 1) return true;
  rs_bar();
  if (tid == 0) {
    uint32_t before;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(p.sync + 2 + kvh) : "memory");
    sh.last = before == (uint32_t)tiles - 1;
    if (sh.last) p.sync[2 + kvh] = 0u;
  }
  rs_bar();
  if (sh.last)
    for (int idx = tid; idx < G * D; idx += RS_CT) {          // (a warp's outputs are of one head: lane = tile for its maximum and its weight)
      const int head = h0 + idx / D;
      const float *const from = p.part + (size_t)h0 * D + idx;
      float2 st[2];
      float M = -INFINITY;
#pragma unroll
      for (int i = 0; i < 2; i++) {
        st[i] = make_float2(-INFINITY, 0.f);
        if (lane + 32 * i < tiles) st[i] = __ldcg(&state[(size_t)(lane + 32 * i) * p.heads + head]);
        M = fmaxf(M, st[i].x);
      }
      M = warp_max(M);
      float W = 0.f, acc = 0.f;
      if (M > -INFINITY) {
        float c[2];
#pragma unroll
        for (int i = 0; i < 2; i++) c[i] = whole ? exp2f(st[i].x - M) : __expf(st[i].x - M);
#pragma unroll 1
        for (int r0 = 0; r0 < tiles; r0 += 8) {
          float x[8];
#pragma unroll
          for (int i = 0; i < 8; i++) x[i] = r0 + i < tiles ? __ldcg(from + (size_t)(r0 + i) * p.heads * D) : 0.f;
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const int r = r0 + i;
            const float w = __shfl_sync(0xffffffffu, r0 < 32 ? c[0] : c[1], r & 31), l = __shfl_sync(0xffffffffu, r0 < 32 ? st[0].y : st[1].y, r & 31);
            if (r < tiles) {
              if (whole) W += l * w;
              else W += w;
              if (whole) acc += x[i] * w;
              else acc += w * x[i];
            }
          }
        }
      }
      store_act(p.attn, h0 * D + idx, (W > 0.f) ? acc / W : 0.f, DT);
    }
  return true;
}

template <typename T, int D>
__global__ void __launch_bounds__(RS_THREADS, 1) step_resident_kernel(const __grid_constant__ RsParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  RsShared &sh = *(RsShared *)smem;
  uint8_t *const img = smem + RS_HEADER, *const rings = img + p.x_bytes;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (tid < RS_PRODUCERS * RS_DEPTH) {
    mbar_init(&sh.full[0][0] + tid, 2 * RS_GROUP);
    mbar_init(&sh.empty[0][0] + tid, RS_GROUP);
    fence_mbar_init();
  }
  if (tid == 0) sh.stop = 0;
  __syncthreads();
  if (warp >= RS_WARPS) {
    rs_produce(p, sh, rings + (size_t)(warp - RS_WARPS) * p.ring, warp - RS_WARPS, lane);
    return;
  }
  const uint8_t *const ring = rings + (size_t)(warp / RS_GROUP) * p.ring;
  const int page0 = p.kv_indptr[0], kv_len = (p.kv_indptr[1] - page0 - 1) * p.page_size + p.last_page[0];
  // the tiles of the step's plan
  const int tiles = p.tiles > 1 ? p.tile_ends[1] : 1, chunk = p.tiles > 1 ? *p.tile_size : kv_len;
  RsRing rr = {{0u, 0u}, RS_COPY_LIMIT, lane == 0};
  uint32_t round = 0;
  const int ops = 5 * p.layers + (p.head != nullptr ? 1 : 0);
  constexpr int DT = std::is_same<T, __half>::value ? MRS_F16 : MRS_BF16;
  for (int i = 0; i < ops; i++) {
    const RsOp o = rs_op(p, i);
    const RsLayer &L = p.L[min(i / 5, p.layers - 1)];
    const uint8_t *from = img;
    if (o.kind == RS_V) {
      if (o.type != L.type[RS_QK]) from += rs_image(L.type[RS_QK], o.K);
    } else {
      const void *norm_w = o.kind == RS_QK ? L.attn_norm : o.kind == RS_GU ? L.ffn_norm : o.kind == RS_HEAD ? p.final_norm : nullptr;
      uint4 nw0 = make_uint4(0u, 0u, 0u, 0u);
      if (norm_w != nullptr && tid < (o.K >> 3)) nw0 = __ldg((const uint4 *)norm_w + tid);
      if (o.kind == RS_O) {
        if (!rs_attend<T, D>(p, L, sh, img, round, tiles, chunk, kv_len, page0, tid, warp, lane)) return rs_lost(p, sh, DT, tid);
        rs_arrive(p, tid);
      }
      if (i > 0 && !rs_meet(p, sh, round, tid)) return rs_lost(p, sh, DT, tid);
      rs_quantise<T>(p, o, sh, o.kind == RS_QK ? L.type[RS_V] : o.type, norm_w, nw0, img, tid, warp, lane);
    }
    switch (o.type) {
#define RS_CASE(TY) case TY: rs_gemv<TY, T>(p, o, sh, from, ring, rr, warp, lane); break;
      RS_TYPES(RS_CASE)
#undef RS_CASE
    }
    if (o.kind != RS_QK && i + 1 < ops) rs_arrive(p, tid);
  }
  // the last CTA leaves the words as it found them
  rs_bar();
  if (*(volatile int *)&sh.stop) return rs_lost(p, sh, DT, tid);
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(p.sync + 1, 1u) == gridDim.x - 1) { p.sync[0] = 0u; p.sync[1] = 0u; }
  }
}

// ---------------------------------------------------------------- host side
template <typename T, int D> static cudaError_t rs_launch(const RsParams &p, int grid, size_t smem, cudaStream_t stream) {
  auto kern = step_resident_kernel<T, D>;
  int per_sm = 0;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, RS_THREADS, smem);
  if (e != cudaSuccess || per_sm < 1) { cudaGetLastError(); return cudaErrorNotSupported; }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid); cfg.blockDim = dim3(RS_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, p);
}

}  // namespace mrs

using namespace mrs;

extern "C" int64_t mrs_llama_resident_bytes(int32_t heads, int32_t head_dim, int32_t padded_tiles) {
  return 256 + (int64_t)padded_tiles * heads * (head_dim + 2) * 4;
}

// The launch's parameters but for the layers, its CTAs and their shared memory; false where the step is not of the kind described above.
static bool rs_plan(const mrs_llama_step *s, RsParams &p, int &sms, size_t &smem) {
  const int D = s->head_dim, dt = s->act_dtype;
  if (s->extension != MRS_LLAMA_STEP_RESIDENT || s->resident == nullptr || ((uintptr_t)s->resident & 15) || s->batch != 1 || s->skip_mask != 0 ||
      !s->fused_attention || s->tp != nullptr || s->all_reduce != nullptr || (D != 64 && D != 128) || (dt != MRS_F16 && dt != MRS_BF16) || s->n_layers < 1)
    return false;
  if (s->n_kv_heads < 1 || s->n_heads % s->n_kv_heads != 0 || s->n_heads / s->n_kv_heads > 8 || s->n_kv_heads > RS_MAX_KV_HEADS ||
      s->hidden % 256 != 0 || s->hidden < RS_MIN_HIDDEN || s->block_size < 1 || s->vocab < 1 ||
      s->padded_tiles < 1 || s->padded_tiles > RS_TILES || s->tmp_v == nullptr || s->resident_bytes < mrs_llama_resident_bytes(s->n_heads, D, s->padded_tiles))
    return false;
  if ((int64_t)s->max_blocks_per_seq * s->block_size / s->padded_tiles * s->n_kv_heads > (int64_t)RS_MAX_TILE * D) return false;
  int dev = 0, most = 0, coop = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  int32_t *const timeouts = mrs_mmq_timeout_flag();
  if (!coop || (int64_t)s->padded_tiles * s->n_kv_heads > sms || timeouts == nullptr || *(volatile const int32_t *)timeouts != 0) return false;

  const int nq = s->n_heads * D, nkv = s->n_kv_heads * D, inter = s->layers[0].w_down.cols;
  p = {};
  p.x_bytes = D == 64 ? rs_attend_bytes<64>() : rs_attend_bytes<128>();
  int widest = 0;
  auto usable = [&](const mrs_qweight &w, int rows, int K) {
    if (!rs_type_ok(w.ggml_type) || w.rows != rows || w.cols != K || K % 256 != 0 || (int64_t)(rows + 1) * sms > 0x7fffffff) return false;
    if (w.ggml_type == MRS_Q4_K && ((uintptr_t)w.data & 15)) return false;
    if ((uintptr_t)w.data & 1) return false;
    const int slot = rs_type(w.ggml_type).slot;
    if (slot > widest) widest = slot;
    return true;
  };
  auto image = [&](int bytes) { if (bytes > p.x_bytes) p.x_bytes = bytes; };
  const void *aligned[] = {s->x, s->x2, s->q, s->k, s->v, s->attn_out, s->act, s->final_norm, s->rope_cos, s->rope_sin};
  for (const void *a : aligned) if (a == nullptr || ((uintptr_t)a & 15)) return false;
  for (int l = 0; l < s->n_layers; l++) {
    const mrs_llama_layer &L = s->layers[l];
    if (!usable(L.wq, nq, s->hidden) || !usable(L.wk, nkv, s->hidden) || !usable(L.wv, nkv, s->hidden) || !usable(L.wo, s->hidden, nq) ||
        !usable(L.w_gate, inter, s->hidden) || !usable(L.w_up, inter, s->hidden) || !usable(L.w_down, s->hidden, inter) ||
        L.wq.ggml_type != L.wk.ggml_type || L.w_gate.ggml_type != L.w_up.ggml_type)
      return false;
    const void *ptrs[] = {L.attn_norm, L.ffn_norm, L.k_cache, L.v_cache};
    for (const void *a : ptrs) if (a == nullptr || ((uintptr_t)a & 15)) return false;
    image(rs_image(L.wq.ggml_type, s->hidden) + (L.wv.ggml_type != L.wq.ggml_type ? rs_image(L.wv.ggml_type, s->hidden) : 0));
    image(rs_image(L.wo.ggml_type, nq));
    image(rs_image(L.w_gate.ggml_type, s->hidden));
    image(rs_image(L.w_down.ggml_type, inter));
  }
  if (!usable(s->lm_head, s->vocab, s->hidden)) return false;
  image(rs_image(s->lm_head.ggml_type, s->hidden));
  p.x_bytes = (p.x_bytes + 127) & ~127;
  p.ring = (most - RS_HEADER - p.x_bytes) / RS_PRODUCERS & ~15;
  if (p.ring < 4 * RS_GROUP * widest) return false;                 // two stages at least

  p.final_norm = s->final_norm; p.rope_cos = s->rope_cos; p.rope_sin = s->rope_sin;
  p.positions = s->positions; p.slots = s->slot_mapping;
  p.kv_indptr = s->kv_indptr; p.kv_indices = s->kv_indices; p.last_page = s->kv_last_page_len;
  p.tile_ends = s->o_indptr; p.tile_size = s->kv_chunk_size; p.tiles = s->padded_tiles;
  p.x = s->x; p.x2 = s->x2; p.q = s->q; p.k = s->k; p.v = s->v; p.attn = s->attn_out; p.act = s->act; p.logits = s->logits;
  p.sync = (uint32_t *)s->resident;
  p.part = (float *)((uint8_t *)s->resident + 256);
  p.timeouts = timeouts;
  p.eps = s->rms_eps; p.scale_log2 = s->sm_scale * 1.4426950408889634f;
  p.hidden = s->hidden; p.inter = inter; p.nq = nq; p.nkv = nkv; p.heads = s->n_heads; p.kv_heads = s->n_kv_heads;
  p.page_size = s->block_size;
  p.page_shift = -1;
  for (int i = 0; i < 31; i++) if (s->block_size == 1 << i) p.page_shift = i;
  p.vocab = s->vocab; p.head_type = s->lm_head.ggml_type; p.interleaved = s->rope_neox ? 0 : 1;
  smem = RS_HEADER + p.x_bytes + (size_t)RS_PRODUCERS * p.ring;
  return true;
}

// 1 where mrs_llama_decode_step would run this step as a resident grid.
extern "C" int32_t mrs_llama_step_is_resident(const mrs_llama_step *s) {
  RsParams p;
  int sms = 0;
  size_t smem = 0;
  return rs_plan(s, p, sms, smem) ? 1 : 0;
}

// Layers and head of a step, its first hidden state in s->x.  cudaErrorNotSupported, and nothing launched, where the step is not of the kind described
// above: the caller launches its chain.
extern "C" int32_t mrs_llama_step_resident(const mrs_llama_step *s, void *stream) {
  const int no = (int)cudaErrorNotSupported, D = s->head_dim, dt = s->act_dtype;
  RsParams p;
  int sms = 0;
  size_t smem = 0;
  if (!rs_plan(s, p, sms, smem)) return no;
  for (int l0 = 0; l0 < s->n_layers; l0 += RS_LAYERS) {
    p.layers = s->n_layers - l0 < RS_LAYERS ? s->n_layers - l0 : RS_LAYERS;
    p.head = l0 + p.layers == s->n_layers ? (const uint8_t *)s->lm_head.data : nullptr;
    for (int l = 0; l < p.layers; l++) {
      const mrs_llama_layer &L = s->layers[l0 + l];
      RsLayer &to = p.L[l];
      const mrs_qweight *w[7] = {&L.wq, &L.wk, &L.wv, &L.wo, &L.w_gate, &L.w_up, &L.w_down};
      for (int i = 0; i < 7; i++) to.w[i] = (const uint8_t *)w[i]->data;
      to.attn_norm = L.attn_norm; to.ffn_norm = L.ffn_norm; to.kc = L.k_cache; to.vc = L.v_cache;
      to.type[RS_QK] = (uint8_t)L.wq.ggml_type; to.type[RS_V] = (uint8_t)L.wv.ggml_type; to.type[RS_O] = (uint8_t)L.wo.ggml_type;
      to.type[RS_GU] = (uint8_t)L.w_gate.ggml_type; to.type[RS_DOWN] = (uint8_t)L.w_down.ggml_type;
    }
    const cudaError_t e = dt == MRS_F16 ? (D == 64 ? rs_launch<__half, 64>(p, sms, smem, (cudaStream_t)stream) : rs_launch<__half, 128>(p, sms, smem, (cudaStream_t)stream))
                                        : (D == 64 ? rs_launch<__nv_bfloat16, 64>(p, sms, smem, (cudaStream_t)stream)
                                                   : rs_launch<__nv_bfloat16, 128>(p, sms, smem, (cudaStream_t)stream));
    if (e == cudaErrorCooperativeLaunchTooLarge && l0 == 0) { cudaGetLastError(); return no; }      // (fewer SMs than the device has: a part of it)
    if (e != cudaSuccess) return (int32_t)e;
  }
  return 0;
}
