// w4a16.cu — W4A16 (GPTQ / AWQ int4) linears and dense f16/bf16 ones at small batches, on the 5th-gen tensor cores.
//
// Replaces the reference's Marlin path behind its own symbols
//   marlin_{gptq,awq}_4bit_{f16,bf16}, {gptq,awq}_marlin_repack     REF mistralrs-quant/src/gptq/marlin_ffi.rs:6-81,
//   kernels/marlin/marlin_kernel.cuh (one kernel for every m), marlin_repack.cu:255,473
// and the dense small-batch lm_head of GPTQ checkpoints (REF kernels/gemv/gemv.cu, candle matmul).
//
// int4: the dequantising GEMM of mmq_ts.cuh (weight rows as the MMA's M, dequantised into tensor memory) over the tiles below; one launch
// for any number of tokens.
// Dense: "swap-AB" as well — per CTA one 128-row weight tile x one K split, 320 threads: warp 0 TMA, warp 1 MMA issuer, all of warps
// 2 .. 9 epilogue.  Split-K CTAs of one tile form a thread-block cluster (<= 4): partial accumulators go to the leader's shared memory
// through DSMEM and are summed in a fixed order — deterministic, no global scratch.
//
// Repacked weight layout ("mrs int4 tiles", same byte count as the checkpoint tensor so the
// reference's result buffer [K/16, N*16/8] i32 fits): [K/64][N][32 B]; the 32 bytes of (k-step, row)
// hold 64 nibbles, word w = k 8w..8w+7 with nibble j < 4 <-> k = 2j and nibble 4+j <-> k = 2j+1 (so
// that `q & 0x000f000f` yields the f16x2 pair (k, k+1)).
#include "mmq_ts.cuh"

#include <stdio.h>

namespace mrs {

constexpr int WA_BM = 128;      // weight rows per CTA (UMMA M)
constexpr int WA_BK = 64;       // K per stage
constexpr int WA_STAGES = 4;
constexpr int WA_DQ_WARPS = 8;
constexpr int WA_THREADS = 64 + WA_DQ_WARPS * 32;
constexpr int WA_A_BYTES = WA_BM * WA_BK * 2;   // 16 KB

struct WaParams {
  void *y;                 // [M, N]
  int M, N, K, dtype;
  int m0;                  // first token of this pass
  int ksteps_per_split;    // K-steps (of 64) per split CTA
  int pdl;                 // link of a programmatic-dependent-launch chain: x comes from the upstream grid
};

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive_release() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait_acquire() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t map_to_rank(uint32_t local_smem_addr, uint32_t rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local_smem_addr), "r"(rank));
  return remote;
}
__device__ __forceinline__ void st_cluster_f32_at(uint32_t remote_addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote_addr), "f"(v) : "memory");
}
// arrive on another CTA's mbarrier; release at cluster scope orders this thread's earlier remote stores before it
__device__ __forceinline__ void mbar_arrive_remote(uint32_t remote_bar_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote_bar_addr) : "memory");
}
__device__ __forceinline__ void mbar_wait_cluster(uint64_t *bar, uint32_t parity) {
  asm volatile(
      "{\n\t.reg .pred P1;\n\tWAITC_LOOP:\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P1, [%0], %1;\n\t"
      "@P1 bra WAITC_DONE;\n\tbra WAITC_LOOP;\n\tWAITC_DONE:\n\t}" ::"r"(smem_u32(bar)),
      "r"(parity)
      : "memory");
}

// ---- shared epilogue: TMEM -> registers -> [cluster split-K reduction] -> y ----------------------
// Called by ALL threads of the CTA; `epi` marks the 8 epilogue warps (warp ids 2..9), two per TMEM lane
// quarter.  Split-K: the non-leader CTAs push their partial tile straight into a DEDICATED region of the
// leader's shared memory (red[rank-1][token][row], never aliased with the operand rings, so no "rings drained"
// rendezvous is needed) and then arrive, thread by thread with release.cluster, on the leader's `red_bar`;
// the leader adds the partials in rank order (deterministic).  The only cluster barrier is the start-up one
// (arrive right after the mbarrier init in the kernel prologue, wait here, long since complete), which
// guarantees the leader's barrier exists before anybody arrives on it.
template <int NT>
__device__ __forceinline__ void wa_epilogue(const WaParams &p, float *red, uint64_t *red_bar, uint64_t *acc_full, uint32_t tmem_base,
                                            int nk, int ksplit, uint32_t rank, int n0, int rows_valid) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int CPW = NT / 2;              // columns (tokens) per epilogue warp: two warps share a lane quarter
  const bool epi = warp >= 2 && warp < 2 + WA_DQ_WARPS;
  const int q = warp & 3, half = (warp - 2) >> 2;
  const int row = q * 32 + lane;           // TMEM lane = weight row inside the tile
  auto ld16 = [&](int col, float *dstv) {
    uint32_t v[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)col));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) dstv[i] = __uint_as_float(v[i]);
  };
  __syncwarp();
  // PDL: y (and everything written two kernels ago) may only be overwritten once the upstream grid has completed;
  // this late in the kernel the wait returns at once — and every CTA must pass it so that completion stays transitive
  if (p.pdl) pdl_wait();
  if constexpr (NT <= 64) {
    float acc[CPW];
    if (epi) {
      if (nk > 0) {
        mbar_wait(acc_full, 0);
        tc_fence_after();
#pragma unroll
        for (int c0 = 0; c0 < CPW; c0 += 16) ld16(half * CPW + c0, acc + c0);
      } else {
#pragma unroll
        for (int i = 0; i < CPW; i++) acc[i] = 0.f;
      }
    }
    if (ksplit > 1) {
      cluster_wait_acquire();              // start-up barrier (every thread of every CTA arrived in the prologue)
      if (epi && rank != 0) {
        const uint32_t rbase = map_to_rank(smem_u32(red + ((size_t)(rank - 1) * NT + half * CPW) * WA_BM + row), 0u);
#pragma unroll
        for (int i = 0; i < CPW; i++) st_cluster_f32_at(rbase + (uint32_t)i * (WA_BM * 4), acc[i]);
        mbar_arrive_remote(map_to_rank(smem_u32(red_bar), 0u));
      }
      if (epi && rank == 0) {
        mbar_wait_cluster(red_bar, 0);
        for (int s = 1; s < ksplit; s++)
#pragma unroll
          for (int i = 0; i < CPW; i++) acc[i] += red[((size_t)(s - 1) * NT + half * CPW + i) * WA_BM + row];
      }
    }
    if (epi && rank == 0 && row < rows_valid) {
      const int nrow = n0 + row;
#pragma unroll
      for (int i = 0; i < CPW; i++) {
        const int tok = p.m0 + half * CPW + i;
        if (tok < p.M) store_act(p.y, (int64_t)tok * p.N + nrow, acc[i], p.dtype);
      }
    }
  } else {
    // large token tiles (no split-K): stream the accumulators out 16 columns at a time
    if (epi && nk > 0) {
      mbar_wait(acc_full, 0);
      tc_fence_after();
#pragma unroll 1
      for (int c0 = 0; c0 < CPW; c0 += 16) {
        float v[16];
        ld16(half * CPW + c0, v);
        if (row < rows_valid) {
#pragma unroll
          for (int i = 0; i < 16; i++) {
            const int tok = p.m0 + half * CPW + c0 + i;
            if (tok < p.M) store_act(p.y, (int64_t)tok * p.N + n0 + row, v[i], p.dtype);
          }
        }
      }
    }
  }
}

// ---- dense 16-bit weights: A tiles straight from TMA, one ring -------------------------------------
template <int NT>
__global__ void __launch_bounds__(WA_THREADS, NT <= 64 ? 2 : 1)
w16_dense_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const WaParams p) {
  constexpr int X_BYTES = NT * 128;
  constexpr int STAGE = WA_A_BYTES + X_BYTES;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t *bars = (uint64_t *)(smem + WA_STAGES * STAGE);
  uint64_t *in_full = bars, *empty = bars + WA_STAGES, *acc_full = bars + 2 * WA_STAGES, *red_bar = acc_full + 1;
  uint32_t *tmem_slot = (uint32_t *)(red_bar + 1);
  float *red = (float *)((uint8_t *)bars + 256);   // split-K partials (present only when ksplit > 1)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = blockIdx.x * WA_BM;
  const int ksplit = gridDim.y;
  const uint32_t rank = (ksplit > 1) ? cluster_ctarank() : 0u;
  const int nk_total = p.K / WA_BK;
  const int kb0 = (int)rank * p.ksteps_per_split;
  const int nk = max(0, min(p.ksteps_per_split, nk_total - kb0));
  const int rows_valid = min(WA_BM, p.N - n0);
  if (p.pdl && tid == 0) pdl_launch_dependents();
  if (tid == 0) {
    for (int s = 0; s < WA_STAGES; s++) { mbar_init(&in_full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(acc_full, 1);
    mbar_init(red_bar, (uint32_t)(ksplit - 1) * WA_DQ_WARPS * 32u);
    fence_mbar_init();
  }
  constexpr uint32_t TCOLS = NT < 32 ? 32 : NT;
  if (warp == 1) tmem_alloc(tmem_slot, TCOLS);
  tc_fence_before();
  __syncthreads();
  if (ksplit > 1) cluster_arrive_release();   // start-up cluster barrier; waited on in the epilogue
  tc_fence_after();
  // REDUX result lives in a uniform register: the MMA issue loop gets uniform operands (no per-MMA waterfall)
  const uint32_t tmem_base = __reduce_max_sync(0xffffffffu, *tmem_slot);
  if (warp == 0) {
    if (lane == 0) {
      if (p.pdl) pdl_wait();   // (weights and activations share one stage here: the whole stream waits for the upstream grid)
      int stage = 0, phase = 0;
      for (int i = 0; i < nk; i++) {
        const int kb = kb0 + i;
        mbar_wait(&empty[stage], phase ^ 1);
        uint8_t *st = smem + (size_t)stage * STAGE;
        mbar_arrive_expect_tx(&in_full[stage], X_BYTES + WA_A_BYTES);
        tma_load_2d(st, &tmap_w, kb * WA_BK, n0, &in_full[stage]);
        tma_load_2d(st + WA_A_BYTES, &tmap_x, kb * WA_BK, p.m0, &in_full[stage]);
        if (++stage == WA_STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    const uint32_t fmt = (p.dtype == MRS_BF16) ? 1u : 0u;
    const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(WA_BM >> 4) << 24);
    int stage = 0, phase = 0;
    for (int i = 0; i < nk; i++) {
      mbar_wait(&in_full[stage], phase);
      tc_fence_after();
      if (lane == 0) {
        const uint8_t *as = smem + (size_t)stage * STAGE, *xs = as + WA_A_BYTES;
#pragma unroll
        for (int k = 0; k < WA_BK / 16; k++)
          umma_f16(tmem_base, umma_desc_sw128(as) + (uint64_t)(2 * k), umma_desc_sw128(xs) + (uint64_t)(2 * k), idesc, (i | k) ? 1u : 0u);
        umma_commit(&empty[stage]);
        if (i == nk - 1) umma_commit(acc_full);
      }
      __syncwarp();
      if (++stage == WA_STAGES) { stage = 0; phase ^= 1; }
    }
  }
  wa_epilogue<NT>(p, red, red_bar, acc_full, tmem_base, nk, ksplit, rank, n0, rows_valid);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TCOLS);
}

// ---------------------------------------------------------------- repack kernels
// GPTQ checkpoint [K/8, N] i32 (nibble j of word (k8, n) = k 8*k8 + j) -> mrs int4 tiles; `perm`
// (argsort of g_idx, REF gptq_cuda.rs:573-583) gathers source rows exactly like
// gptq_marlin_repack does: packed row k' takes checkpoint row perm[k'].
__global__ void repack_gptq_kernel(const uint32_t *__restrict__ qw, const int32_t *__restrict__ perm, uint32_t *__restrict__ out,
                                   int K, int N) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;   // one output word: (ks, n, w)
  const int64_t total = (int64_t)(K / 64) * N * 8;
  if (idx >= total) return;
  const int w = (int)(idx & 7);
  const int n = (int)((idx >> 3) % N);
  const int ks = (int)((idx >> 3) / N);
  uint32_t o = 0;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const int kdst = ks * 64 + w * 8 + j;
    const int ksrc = perm ? perm[kdst] : kdst;
    const uint32_t nib = (qw[(size_t)(ksrc >> 3) * N + n] >> (4 * (ksrc & 7))) & 0xFu;
    const int pos = (j & 1) ? 4 + (j >> 1) : (j >> 1);
    o |= nib << (4 * pos);
  }
  out[idx] = o;
}
// AWQ checkpoint [K, N/8] i32 (nibble i of word (k, c) = column 8c + {0,2,4,6,1,3,5,7}[i]) -> mrs int4 tiles
__global__ void repack_awq_kernel(const uint32_t *__restrict__ qw, uint32_t *__restrict__ out, int K, int N) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t total = (int64_t)(K / 64) * N * 8;
  if (idx >= total) return;
  const int w = (int)(idx & 7);
  const int n = (int)((idx >> 3) % N);
  const int ks = (int)((idx >> 3) / N);
  const int c7 = n & 7;
  const int ipos = (c7 & 1) ? 4 + (c7 >> 1) : (c7 >> 1);   // inverse of {0,2,4,6,1,3,5,7}
  uint32_t o = 0;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const int k = ks * 64 + w * 8 + j;
    const uint32_t nib = (qw[(size_t)k * (N >> 3) + (n >> 3)] >> (4 * ipos)) & 0xFu;
    const int pos = (j & 1) ? 4 + (j >> 1) : (j >> 1);
    o |= nib << (4 * pos);
  }
  out[idx] = o;
}

// ---------------------------------------------------------------- host
template <int NT>
static cudaError_t launch_dense(const CUtensorMap &tx, const CUtensorMap &tw, WaParams p, int ksplit, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((p.N + WA_BM - 1) / WA_BM, ksplit);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (ksplit > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 1; attr[na].val.clusterDim.y = ksplit; attr[na].val.clusterDim.z = 1;
    na++;
  }
  if (p.pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    na++;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  auto kern = w16_dense_kernel<NT>;
  const size_t smem = 1024 + (size_t)WA_STAGES * (WA_A_BYTES + NT * 128) + 256 + (size_t)(ksplit - 1) * NT * WA_BM * 4;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cfg.blockDim = dim3(WA_THREADS);
  cfg.dynamicSmemBytes = smem;
  return cudaLaunchKernelEx(&cfg, kern, tx, tw, p);
}

// split K over a cluster when the row tiles alone leave SMs idle (two CTAs per SM are resident)
static int pick_ksplit(int N, int K, int NT) {
  if (NT > 64) return 1;   // large token tiles stream their epilogue; compute-bound anyway
  int sms = 148;
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int tiles = (N + WA_BM - 1) / WA_BM, nk = K / WA_BK;
  const int slots = 2 * sms;
  int ks = 1;
  for (int c = 2; c <= 4; c *= 2) {
    const int per = ((nk + c - 1) / c + 1) & ~1;
    const bool fits = 1024 + (size_t)WA_STAGES * (WA_A_BYTES + NT * 128) + 256 + (size_t)(c - 1) * NT * WA_BM * 4 <= 227 * 1024;
    if (tiles * c <= slots && per >= 4 && per * (c - 1) < nk && fits) ks = c;
  }
  return ks;
}

static bool wa_refused(const void *x, const void *w, int K, int dtype, cudaError_t &e) {
  e = K % WA_BK != 0 || (dtype != MRS_F16 && dtype != MRS_BF16) ? cudaErrorInvalidValue
      : ((uintptr_t)x & 15) || ((uintptr_t)w & 15) ? cudaErrorMisalignedAddress : cudaSuccess;
  return e != cudaSuccess;
}

static cudaError_t run_dense(const void *x, const void *w, void *y, int M, int K, int N, int dtype, cudaStream_t st, int pdl = 0) {
  if (M <= 0 || N <= 0) return cudaSuccess;
  cudaError_t e;
  if (wa_refused(x, w, K, dtype, e)) return e;
  CUtensorMap tx, tw;
  for (int m0 = 0; m0 < M; m0 += 256) {
    const int mt = M - m0 < 256 ? M - m0 : 256;
    const int NT = mt <= 32 ? 32 : mt <= 64 ? 64 : mt <= 128 ? 128 : 256;
    if (!tc_make_map_2d(&tx, x, (uint64_t)M, (uint64_t)K, WA_BK, (uint32_t)NT, dtype)) return cudaErrorInvalidValue;
    if (!tc_make_map_2d(&tw, w, (uint64_t)N, (uint64_t)K, WA_BK, WA_BM, dtype)) return cudaErrorInvalidValue;
    WaParams p = {};
    p.y = y; p.M = M; p.N = N; p.K = K; p.dtype = dtype; p.m0 = m0;
    p.pdl = (pdl && M <= 256) ? 1 : 0;   // (one pass only: a second token pass would race the first one's output)
    const int ks = pick_ksplit(N, K, NT);
    p.ksteps_per_split = ks > 1 ? (((K / WA_BK + ks - 1) / ks + 1) & ~1) : K / WA_BK;
    e = NT == 32 ? launch_dense<32>(tx, tw, p, ks, st) : NT == 64 ? launch_dense<64>(tx, tw, p, ks, st)
        : NT == 128 ? launch_dense<128>(tx, tw, p, ks, st) : launch_dense<256>(tx, tw, p, ks, st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

static cudaError_t run_int4(const void *x, const void *w, const void *scales, const int32_t *qzeros, void *y, int M, int K, int N, int group, int dtype,
                            int scale_perm, cudaStream_t st, int pdl = 0, bool scales_other = false) {
  if (M <= 0 || N <= 0) return cudaSuccess;
  cudaError_t e;
  if (K % WA_BK != 0 || (dtype != MRS_F16 && dtype != MRS_BF16)) return cudaErrorInvalidValue;
  if (group <= 0) group = K;
  if (group % 32 != 0 || K % group != 0 || N % 8 != 0) return cudaErrorInvalidValue;
  if (qzeros != nullptr && N % 32 != 0) return cudaErrorInvalidValue;   // zero-point rows travel as 16-byte bulk copies
  if (wa_refused(x, w, K, dtype, e)) return e;
  // scale and zero-point rows travel as bulk copies, which start on 16-byte boundaries (N makes their rows multiples of 16 bytes)
  if (((uintptr_t)scales & 15) || ((uintptr_t)qzeros & 15)) return cudaErrorMisalignedAddress;
  const TsDevice &d = ts_device();
  if ((e = ts_refused(d)) != cudaSuccess) return e;
  // (a span of a row: 128 B of nibbles and its scales; 800: the dequantisers' weight in the plan's estimate, two operations a weight)
  const TsPlan plan = ts_plan(M, N, K, 128 + 2 * ((TS_SPAN_K + group - 1) / group), 800, 0, d);
  const TsCall c = {w, x, y, M, N, K, 0, dtype, plan.nt, plan.tiles_m, plan.ksplit, d.sms, d.timeouts, st, scales, qzeros, group, scale_perm, pdl ? 1 : 0};
  return scales_other ? ts_launch<TS_INT4_OTHER>(c) : ts_launch<TS_INT4>(c);
}

template cudaError_t ts_launch<TS_INT4>(const TsCall &);
template cudaError_t ts_launch<TS_INT4_OTHER>(const TsCall &);

}  // namespace mrs

using namespace mrs;

// ---- B200-native entries ---------------------------------------------------------------------
// Y[M,N] = X[M,K] . W^T, W = repacked int4 (mrs tiles, see gptq_marlin_repack below); scales
// [K/group, N] in dtype (0 f16 / 1 bf16), group <= 0: one group; qzeros: AWQ raw zero points or NULL
// (symmetric, zero point 8); scale_perm: 0 plain, 1/2 Marlin-permuted scale columns.
extern "C" int32_t mrs_w4a16_gemm(const void *x, const void *w_tiles, const void *scales, const int32_t *qzeros, void *y,
                                  int32_t M, int32_t K, int32_t N, int32_t group, int32_t dtype, int32_t scale_perm,
                                  void *stream) {
  return (int32_t)run_int4(x, w_tiles, scales, qzeros, y, M, K, N, group, dtype, scale_perm, (cudaStream_t)stream);
}
// Y[M,N] = X[M,K] . W[N,K]^T with dense 16-bit W (the lm_head of GPTQ/AWQ checkpoints at decode batch)
extern "C" int32_t mrs_dense_linear(const void *x, const void *w, void *y, int32_t M, int32_t K, int32_t N, int32_t dtype,
                                    void *stream) {
  return (int32_t)run_dense(x, w, y, M, K, N, dtype, (cudaStream_t)stream);
}
// the same two as links of a programmatic-dependent-launch chain (decode layer stack): the weight stream starts while
// the upstream kernel is still running; x is read, and y written, only after it has completed
extern "C" int32_t mrs_w4a16_gemm_pdl(const void *x, const void *w_tiles, const void *scales, const int32_t *qzeros, void *y,
                                      int32_t M, int32_t K, int32_t N, int32_t group, int32_t dtype, int32_t scale_perm,
                                      int32_t pdl, void *stream) {
  return (int32_t)run_int4(x, w_tiles, scales, qzeros, y, M, K, N, group, dtype, scale_perm, (cudaStream_t)stream, pdl);
}
extern "C" int32_t mrs_dense_linear_pdl(const void *x, const void *w, void *y, int32_t M, int32_t K, int32_t N, int32_t dtype,
                                        int32_t pdl, void *stream) {
  return (int32_t)run_dense(x, w, y, M, K, N, dtype, (cudaStream_t)stream, pdl);
}

// ---- the reference's Marlin symbols (REF mistralrs-quant/src/gptq/marlin_ffi.rs:6-81) ----------
// `weight` of the matmuls is what our own *_marlin_repack wrote (the Rust side treats it as opaque);
// `scales` arrive column-permuted by marlin_permute_scales (REF gptq_cuda.rs:542-565): the 64-wide
// permutation when group < K/8 (the reference passes in_dim / pack_factor as size_k), else the
// 32-wide one; `workspace` (Marlin's lock array) is not needed.
static int marlin_common(const void *inputs, const int32_t *weight, const void *scales, const void *zeros, void *out, int m,
                         int k, int n, int groupsize, int dtype, int is_awq, int64_t stream, bool scales_other = false) {
  cudaError_t status = cudaGetLastError();
  if (status != cudaSuccess) return (int)status;
  const int group = groupsize <= 0 ? k : groupsize;
  const int perm_kind = (groupsize > 0 && groupsize < k / 8) ? 1 : 2;
  const cudaError_t e = run_int4(inputs, weight, scales, is_awq ? (const int32_t *)zeros : nullptr, out, m, k, n, group,
                               dtype, perm_kind, (cudaStream_t)stream, 0, scales_other);
  return e == cudaSuccess ? (int)cudaGetLastError() : (int)e;
}
extern "C" int marlin_gptq_4bit_f16(const void *inputs, const int32_t *weight, const void *scales, const void *zeros,
                                    const void *out, int m, int k, int n, const void *workspace, int groupsize, int64_t stream) {
  (void)workspace;
  return marlin_common(inputs, weight, scales, zeros, (void *)out, m, k, n, groupsize, MRS_F16, 0, stream);
}
extern "C" int marlin_gptq_4bit_bf16(const void *inputs, const int32_t *weight, const void *scales, const void *zeros,
                                     const void *out, int m, int k, int n, const void *workspace, int groupsize, int64_t stream) {
  (void)workspace;
  return marlin_common(inputs, weight, scales, zeros, (void *)out, m, k, n, groupsize, MRS_BF16, 0, stream);
}
extern "C" int marlin_awq_4bit_f16(const void *inputs, const int32_t *weight, const void *scales, const void *zeros,
                                   const void *out, int m, int k, int n, const void *workspace, int groupsize, int64_t stream) {
  (void)workspace;
  return marlin_common(inputs, weight, scales, zeros, (void *)out, m, k, n, groupsize, MRS_F16, 1, stream);
}
extern "C" int marlin_awq_4bit_bf16(const void *inputs, const int32_t *weight, const void *scales, const void *zeros,
                                    const void *out, int m, int k, int n, const void *workspace, int groupsize, int64_t stream) {
  (void)workspace;
  return marlin_common(inputs, weight, scales, zeros, (void *)out, m, k, n, groupsize, MRS_BF16, 1, stream);
}

// The same with scales in their own 16-bit format (scale_dtype, 0 f16 / 1 bf16): a checkpoint's f16 scales under bf16 rows are rounded as the
// kernel reads them, not by a pass of 3.7 us before each call.
extern "C" int mrs_marlin_4bit(const void *inputs, const int32_t *weight, const void *scales, const void *zeros, void *out, int m, int k, int n,
                               int groupsize, int dtype, int scale_dtype, int is_awq, int64_t stream) {
  if (scale_dtype != MRS_F16 && scale_dtype != MRS_BF16) return (int)cudaErrorInvalidValue;
  return marlin_common(inputs, weight, scales, zeros, out, m, k, n, groupsize, dtype, is_awq, stream, scale_dtype != dtype);
}

// weight [k/8, n] i32, perm [k] i32 (argsort of g_idx; the reference always passes one), result: k*n/2 bytes
extern "C" void gptq_marlin_repack(const void *weight, const void *perm, const void *result, int k, int n, int bits,
                                   int64_t stream) {
  if (bits != 4 || k % 64 != 0 || n % 8 != 0) {
    fprintf(stderr, "mrs_b200: gptq_marlin_repack supports 4-bit weights with k %% 64 == 0 (got bits %d, k %d, n %d)\n", bits, k, n);
    return;
  }
  const int64_t total = (int64_t)(k / 64) * n * 8;
  repack_gptq_kernel<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>((const uint32_t *)weight, (const int32_t *)perm,
                                                                                    (uint32_t *)result, k, n);
}
// in [k, n] i32 with n = out_dim / 8 (REF marlin_repack.cu:473-483), perm unused
extern "C" void awq_marlin_repack(const void *in, const void *perm, const void *out, int k, int n, int bits, int64_t stream) {
  (void)perm;
  const int size_n = n * 8;
  if (bits != 4 || k % 64 != 0) {
    fprintf(stderr, "mrs_b200: awq_marlin_repack supports 4-bit weights with k %% 64 == 0 (got bits %d, k %d)\n", bits, k);
    return;
  }
  const int64_t total = (int64_t)(k / 64) * size_n * 8;
  repack_awq_kernel<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>((const uint32_t *)in, (uint32_t *)out, k, size_n);
}
