// mmq_ts.cu — plan and entry point of the dequant-GEMM of mmq_ts.cuh (its kernels: mmq_ts_*.cu, two block types each).
#include "mmq_ts.cuh"

#include <atomic>
#include <mutex>
#include <string.h>

namespace mrs {

#define MRS_TS_TYPES(X) X(MRS_Q4_0) X(MRS_Q4_1) X(MRS_Q5_0) X(MRS_Q5_1) X(MRS_Q8_0) X(MRS_Q2_K) X(MRS_Q3_K) X(MRS_Q4_K) X(MRS_Q5_K) X(MRS_Q6_K)
#define MRS_TS_EXTERN(T) extern template cudaError_t ts_launch<T>(const TsCall &);
MRS_TS_TYPES(MRS_TS_EXTERN)

// A word a device that a kernel sets when a wait runs out: page-locked memory, so that the host sees it without waiting for anything.
// Allocated once for the process (the first call may be inside a capture, which forbids allocations in its own mode).
constexpr int TS_MAX_DEVICES = 64;
static int32_t *ts_flags() {
  static std::once_flag once;
  static int32_t *flags = nullptr;
  std::call_once(once, [] {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    const bool relaxed = cudaThreadExchangeStreamCaptureMode(&mode) == cudaSuccess;
    void *p = nullptr;
    if (cudaHostAlloc(&p, TS_MAX_DEVICES * sizeof(int32_t), cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) {
      memset(p, 0, TS_MAX_DEVICES * sizeof(int32_t));
      flags = (int32_t *)p;
    } else {
      (void)cudaGetLastError();
    }
    if (relaxed) cudaThreadExchangeStreamCaptureMode(&mode);
  });
  return flags;
}

const TsDevice &ts_device() {
  static TsDevice devs[TS_MAX_DEVICES] = {};
  static std::once_flag once[TS_MAX_DEVICES];
  static std::atomic<bool> known[TS_MAX_DEVICES];      // (a call_once that has nothing to do is a call all the same)
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= TS_MAX_DEVICES) dev = 0;
  TsDevice &d = devs[dev];
  if (known[dev].load(std::memory_order_acquire)) return d;
  std::call_once(once[dev], [&d, dev] {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    d.sms = sms > 0 ? sms : 148;
    ts_count_clusters(d.clusters);
    if (int32_t *flags = ts_flags()) {
      void *seen = nullptr;
      if (cudaHostGetDevicePointer(&seen, flags + dev, 0) == cudaSuccess) { d.timeouts = (int *)seen; d.flag = flags + dev; }
      else (void)cudaGetLastError();
    }
    known[dev].store(true, std::memory_order_release);
  });
  return d;
}

cudaError_t ts_refused(const TsDevice &d) {
  if (d.flag == nullptr) return cudaErrorNotSupported;
  return *(volatile const int32_t *)d.flag != 0 ? cudaErrorLaunchTimeout : cudaSuccess;
}

// ggml matrices of fewer rows are not split: results then stay bit for bit those of csrc/mmq_tc.cu, and so small a product is short
// either way.  (Where K is split, how depends on the number of tokens too: the bits of a token's results may depend on how many
// tokens are beside it.)
constexpr int TS_SPLIT_MIN_ROWS = 1024;

// Token tile and split of K by an estimate in clocks.  A span (256 k) of a tile takes the longest of: the tensor pipe (8 clocks a token),
// the dequantisers, and the weight stream at its share of the memory's rate; a CTA adds what it spends before the first product and after
// the last.  K whole: persistent CTAs, so the tiles of one share the start.
// The weights rank plans and are no measured clocks: the dequantisers' 800 to 1500 (the callers') stand for spans that take 1300 by issue alone
// (Q4_K) and up to 3300 in a kernel (Q6_K at 24 tokens).  What they are worth, against the fastest of all plans on one B200: ten block types at
// five matrices and 9 to 512 tokens, 1.1 % slower on average and more than 5 % in 27 of 350 (2048 x 2048 at 300 and 512 tokens, up to 37 %;
// 4096 x 4096 at 200 and 512, up to 12 %); int4 at eleven matrices, 1.9 % on average and more than 5 % in 22 of 154 (matrices 1024 columns
// wide from 64 tokens on, up to 24 %; 4096 columns and more at 300 and 500 tokens, up to 10 %).
TsPlan ts_plan(int M, int N, int K, int span_bytes, int dequant_clocks, int split_min_rows, const TsDevice &d) {
  constexpr int START = 4500, TILE_END = 1200, SPLIT_END = 2600;     // clocks
  const int tiles_n = (N + TS_BM - 1) / TS_BM, spans = (K + TS_SPAN_K - 1) / TS_SPAN_K;
  TsPlan best = {};
  double best_cost = 1e30;
  const int least = (M + 255) / 256;
  for (int tm = least; tm <= least + 2; tm++) {
    const int nt = ((M + tm - 1) / tm + 15) & ~15;
    if (nt > 256 || (tm > least && nt * (tm - 1) >= M)) continue;
    const long long tiles = (long long)tiles_n * tm;
    for (int ks = 1; ks <= 8; ks++) {
      if (ks > 1 && (N < split_min_rows || d.clusters[ks] < 1 || spans < 2 * ks || tiles > 65535)) continue;
      const int room = ks > 1 ? d.clusters[ks] : d.sms;
      const double waves = (double)((tiles + room - 1) / room);
      const double busy = (double)(tiles < room ? tiles : room) * ks;
      const double stream = span_bytes * 128.0 * busy / 3000.0;       // bytes a clock that the memory gives to all SMs
      double span = 8.0 * nt;
      if (span < dequant_clocks) span = dequant_clocks;
      if (span < stream) span = stream;
      const double each = ((spans + ks - 1) / ks) * span;
      const double cost = ks > 1 ? waves * (START + each + SPLIT_END + 8.0 * nt) : START + waves * (each + TILE_END) + 8.0 * nt;
      if (cost < best_cost) { best_cost = cost; best = {nt, tm, ks, (int)waves, cost}; }
    }
  }
  return best;
}

}  // namespace mrs

using namespace mrs;

// 0: take this kernel whenever the shape allows (default); 1: never (mmq_tc.cu for everything) — A/B and tests
static int g_mmq_path = 0;
extern "C" void mrs_mmq_set_path(int32_t path) { g_mmq_path = path; }

// non-zero when a wait inside a kernel ever ran out on the current device (synchronises)
extern "C" int32_t mrs_mmq_timeouts(void) {
  const cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return -(int32_t)e;
  const TsDevice &d = ts_device();
  return d.flag != nullptr ? *(volatile const int32_t *)d.flag : -(int32_t)cudaErrorNotSupported;
}
// the word behind it, for callers that know the stream to be done (null without a device)
extern "C" int32_t *mrs_mmq_timeout_flag(void) { return ts_device().flag; }

// returns cudaErrorNotSupported when the launch does not fit this kernel (the caller falls back to mmq_tc.cu)
static int32_t gguf_ts(int32_t ggml_type, const void *w, const void *x, void *y, int32_t M, int32_t N, int32_t K, int32_t dtype, int pdl, void *stream) {
  if (g_mmq_path == 1) return (int32_t)cudaErrorNotSupported;
  const int elems = blk_elems(ggml_type), bytes = blk_bytes(ggml_type);
  if (bytes == 0 || M <= 0 || N <= 0 || K <= 0 || K % elems != 0 || K % 64 != 0 || (dtype != 0 && dtype != 1)) return (int32_t)cudaErrorNotSupported;
  if (((uintptr_t)w & 15) || ((uintptr_t)x & 15) || ((uintptr_t)y & 1)) return (int32_t)cudaErrorNotSupported;
  // results off a 16-byte boundary: taken where they always were (csrc/mmq_tc.cu refuses them)
  const bool common = ggml_type == MRS_Q8_0 || ggml_type == MRS_Q4_K || ggml_type == MRS_Q6_K;
  if (((uintptr_t)y & 15) && !(common && K % TS_SPAN_K == 0 && (K / elems * bytes) % 16 == 0)) return (int32_t)cudaErrorNotSupported;
  const TsDevice &d = ts_device();
  const cudaError_t refused = ts_refused(d);
  if (refused != cudaSuccess) return (int32_t)refused;
  // the dequantisers' weight in the plan's estimate
  const int clocks = ggml_type == MRS_Q6_K ? 1500 : ggml_type == MRS_Q5_K || ggml_type == MRS_Q3_K || ggml_type == MRS_Q5_0 || ggml_type == MRS_Q5_1 ? 1350 : 1150;
  const TsPlan plan = ts_plan(M, N, K, bytes * (256 / elems), clocks, TS_SPLIT_MIN_ROWS, d);
  const TsCall c = {w, x, y, M, N, K, K / elems * bytes, dtype, plan.nt, plan.tiles_m, plan.ksplit, d.sms, d.timeouts, (cudaStream_t)stream, nullptr, nullptr, 0, 0, pdl, 1, {}, {}, {}};
  switch (ggml_type) {
#define MRS_TS_CASE(T) case T: return (int32_t)ts_launch<T>(c);
  MRS_TS_TYPES(MRS_TS_CASE)
  default: return (int32_t)cudaErrorNotSupported;
  }
}

extern "C" int32_t mrs_mmq_gguf_ts(int32_t ggml_type, const void *w, const void *x, void *y, int32_t M, int32_t N, int32_t K,
                                   int32_t dtype, void *stream) {
  return gguf_ts(ggml_type, w, x, y, M, N, K, dtype, 0, stream);
}

namespace mrs { bool mmq_format_is_forced(); }      // mmq_tc.cu
extern "C" int32_t mrs_mmq_gguf(int32_t ggml_type, const void *w, const void *x, void *y, int32_t M, int32_t N, int32_t K, int32_t dtype, void *stream);

// A link of a programmatic-dependent-launch chain: begins on the weights while the launch before it runs.  A layer of a prompt call is ten
// launches of 5 to 50 us, whose starts (tensor memory, first weights, 2 to 3 us) and ends were paid one after the other: eight layers of
// 4096 x 14336, 300 tokens, 1716 to 1765 us so, 1622 with the products, the GLU and the norms as links.
extern "C" int32_t mrs_mmq_gguf_chained(int32_t ggml_type, const void *w, const void *x, void *y, int32_t M, int32_t N, int32_t K, int32_t dtype, void *stream) {
  if (M > 0 && N > 0 && !mmq_format_is_forced()) {
    const int32_t e = gguf_ts(ggml_type, w, x, y, M, N, K, dtype, 1, stream);
    if (e != (int32_t)cudaErrorNotSupported) return e;
  }
  return mrs_mmq_gguf(ggml_type, w, x, y, M, N, K, dtype, stream);
}

// y_i = x . w_i^T for two or three matrices of a type and as many columns (n2 = 0: two), as one launch.  cudaErrorNotSupported, and nothing launched,
// where that does not fit this kernel: the caller launches them one by one.
static int32_t gguf_multi(int32_t ggml_type, const void *w0, const void *w1, const void *w2, const void *x, void *y0, void *y1, void *y2, int32_t M, int32_t n0,
                          int32_t n1, int32_t n2, int32_t K, int32_t dtype, int pdl, void *stream) {
  if (g_mmq_path == 1 || mmq_format_is_forced()) return (int32_t)cudaErrorNotSupported;
  if (ggml_type != MRS_Q4_K && ggml_type != MRS_Q5_K && ggml_type != MRS_Q6_K && ggml_type != MRS_Q8_0) return (int32_t)cudaErrorNotSupported;
  const int elems = blk_elems(ggml_type), bytes = blk_bytes(ggml_type);
  if (M <= 0 || n0 <= 0 || n1 <= 0 || n2 < 0 || K <= 0 || K % elems != 0 || K % 64 != 0 || (K / elems * bytes) % 16 != 0 || (dtype != 0 && dtype != 1))
    return (int32_t)cudaErrorNotSupported;
  const void *const ptrs[] = {w0, w1, n2 > 0 ? w2 : w1, x, y0, y1, n2 > 0 ? y2 : y1};
  for (const void *q : ptrs) if (q == nullptr || ((uintptr_t)q & 15)) return (int32_t)cudaErrorNotSupported;
  if ((int64_t)n0 + n1 + n2 > 0x7fffff00) return (int32_t)cudaErrorNotSupported;
  const TsDevice &d = ts_device();
  const cudaError_t refused = ts_refused(d);
  if (refused != cudaSuccess) return (int32_t)refused;
  const int clocks = ggml_type == MRS_Q6_K ? 1500 : ggml_type == MRS_Q5_K ? 1350 : 1150, pad = TS_BM - 1;
  const int rows = (n0 + pad) / TS_BM * TS_BM + (n1 + pad) / TS_BM * TS_BM + (n2 + pad) / TS_BM * TS_BM;
  const bool split = n0 >= TS_SPLIT_MIN_ROWS && n1 >= TS_SPLIT_MIN_ROWS && (n2 == 0 || n2 >= TS_SPLIT_MIN_ROWS);      // (as each alone)
  const TsPlan plan = ts_plan(M, rows, K, bytes * (256 / elems), clocks, split ? TS_SPLIT_MIN_ROWS : 0x7fffffff, d);
  // Where one launch is worth it, by the plan's estimate: it saves a start and a drain a matrix, and waves where matrices leave SMs idle.  For many tokens only
  // saved waves count: a wave that fills the GPU takes a tenth longer than one that does not.  One B200, us alone / together: Q4_K 4096 + 1024 + 1024 of 4096 at
  // 24, 300, 1000 tokens 23.5 / 12.2, 43.1 / 19.2, 63.2 / 39.1; 2 x 14336 at 24, 200 tokens 34.5 / 30.7, 46.1 / 42.7, and with Q8_0 at 300, 1000 (left alone)
  // 78.5 / 81.1, 195 / 213; Q6_K 2 x 14336 at 512 (alone) 112 / 130; 3 x 4096 at 1000 (alone) 90 / 101; 2 x 5632 of 2048 at 1000 60.2 / 45.8.
  // A plan with more waves than the matrices have alone (finer token tiles, a split K) pays in dequantising, which the estimate makes little of, so it has to
  // promise more, alone / together: 2 x 11008 of 4096 at 256 tokens Q5_K (0.91 of the estimate alone) 54.6 / 65.2, Q4_K (0.79) 53.5 / 48.7, at 224 tokens (0.89) 48.6 / 48.2; 2 x
  // 13824 of 5120 at 256 Q8_0 76.5 / 84.0.
  double alone = 0.0;
  int waves = 0;
  const int each[] = {n0, n1, n2};
  for (int n : each) {
    if (n == 0) continue;
    const TsPlan one = ts_plan(M, n, K, bytes * (256 / elems), clocks, TS_SPLIT_MIN_ROWS, d);
    alone += one.cost;
    waves += one.waves;
  }
  if (plan.cost > (plan.waves > waves ? 0.85 : 0.92) * alone || (M > 320 && plan.waves >= waves)) return (int32_t)cudaErrorNotSupported;
  const TsCall c = {w0, x, y0, M, n0, K, K / elems * bytes, dtype, plan.nt, plan.tiles_m, plan.ksplit, d.sms, d.timeouts, (cudaStream_t)stream, nullptr, nullptr, 0, 0, pdl,
                    n2 > 0 ? 3 : 2, {w1, w2}, {y1, y2}, {n1, n2}};
  switch (ggml_type) {
  case MRS_Q4_K: return (int32_t)ts_launch<MRS_Q4_K>(c);
  case MRS_Q5_K: return (int32_t)ts_launch<MRS_Q5_K>(c);
  case MRS_Q6_K: return (int32_t)ts_launch<MRS_Q6_K>(c);
  case MRS_Q8_0: return (int32_t)ts_launch<MRS_Q8_0>(c);
  default: return (int32_t)cudaErrorNotSupported;
  }
}

extern "C" int32_t mrs_mmq_gguf_multi(int32_t ggml_type, const void *w0, const void *w1, const void *w2, const void *x, void *y0, void *y1, void *y2, int32_t M,
                                      int32_t n0, int32_t n1, int32_t n2, int32_t K, int32_t dtype, void *stream) {
  return gguf_multi(ggml_type, w0, w1, w2, x, y0, y1, y2, M, n0, n1, n2, K, dtype, 0, stream);
}
extern "C" int32_t mrs_mmq_gguf_multi_chained(int32_t ggml_type, const void *w0, const void *w1, const void *w2, const void *x, void *y0, void *y1, void *y2,
                                              int32_t M, int32_t n0, int32_t n1, int32_t n2, int32_t K, int32_t dtype, void *stream) {
  return gguf_multi(ggml_type, w0, w1, w2, x, y0, y1, y2, M, n0, n1, n2, K, dtype, 1, stream);
}
