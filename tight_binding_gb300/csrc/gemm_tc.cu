// gemm_tc.cu — the Kubo moment matrix mu_mn on the 5th-generation tensor cores.
//
// mu_mn = sum_k conj(L_m[k]) R_n[k] over stored Chebyshev blocks in split precision
// (3 x FP16): the stores hold s x = hi + lo per real number, hi = half(s x) and lo =
// half(s x - hi) (|lo| <= 2^-11 |s x|, 22 significant bits), with a power of two s per
// block row that keeps the values inside FP16's range (split_store.cuh).  An FP16 and a
// TF32 number have the same 11 significant bits, and kind::f16 runs at twice the rate of
// kind::tf32.  With the real and imaginary parts in rows of their own,
//   Re mu = Lr Rr + Li Ri,  Im mu = Lr Ri - Li Rr,
//   A B ~ A_hi B_hi + A_hi B_lo + A_lo B_hi           (FP32 accumulation).
//
// One CTA: a 128 (m) x 128 (n) complex output tile over a K range (split-K).  A stage
// is one K tile of the stores (32 values of k: 128-byte rows of hi and lo halves, re and
// im, for A and for B, 64 KB), loaded by TMA with the 128-byte swizzle straight into the
// UMMA K-major SWIZZLE_128B layout, three stages deep; nothing converts.  Per 16 k and
// product the issuing thread runs D[Re|Im] += A_re x [B_re|B_im] (N = 256, the parts lie one
// after the other), D[Re] += A_im x B_im and D[Im] += (-A_im) x B_re (N = 128, A negated by the
// instruction).  Two CTAs of a cluster share an m tile (adjacent n tiles): each loads
// half of the A boxes and multicasts them to both, and a stage is reused only when both
// CTAs' MMAs have released it (their commits arrive on both CTAs' barriers).
// Roles:
//   warp 17    TMA producer: one thread issues the boxes of each stage;
//   warp 16    TMEM allocation and, lane 0, MMA issue + tcgen05.commit;
//   warps 0-15 epilogue (64 columns each): every kChunk tiles read the accumulator with
//              tcgen05.ld (double-buffered in TMEM, all 512 columns) and add it into FP32
//              registers, every kFlush chunks add those into the CTA's FP64 partial tile
//              in global memory (column after column, so that a warp's 32 rows are one
//              256-byte access; L2 holds it): long FP32 sums lose the accuracy the Kubo weights
//              need, and 128 x 128 complex float-float pairs would fill the register file.
// What bounds it: shared memory, and the power cap on long runs.  The MMAs of 16 k read 3
// x (12 + 16) KB and the TMA writes 32 KB in the 768 clocks of the 12 products at full
// rate, 151 bytes a clock against 128.  FCC 128^3, M = 1024, R = 8: 268 ms, 1,578 TFLOP/s of
// issued products, 81% of cuBLAS' bf16 burst rate and 92% of its sustained rate (638 ms
// with complex64 stores split into TF32 pairs by converter warps, 70% of the TF32 rate;
// 410 ms with a row-major partial tile, whose flush held the accumulators up); square
// 256^2, M = 512, R = 16: 10.2 -> 4.2 ms.
// Error against 64 bits, relative to the largest |L_m||R_n|: K = 2^21 and 2^22, M = 2: 1.5e-6 for
// equal blocks (2.2e-6 with the TF32 pairs, whose chunk sums went into float-float pairs: FP16
// products take 16 k at a time, so a chunk of 128 k is half as many FP32 accumulations),
// 1.6e-6 where the amplitude grows by e^12 along k (2.4e-6), 5.6e-7 for positive ones
// (1.4e-6); 1.6e-6, 1.7e-6 and 6e-7 at M = 1024, K = 2^16 (2.3e-6, 2.4e-6, 1.5e-6).  The FP32 register
// sum is some twentieth of that: with kFlush = 16, 8, 4 the errors are within 6% of these,
// and the GEMM takes 8, 29, 80% longer (square 256^2: 10, 31, 75%).
// Every mbarrier wait is bounded; on timeout the CTA records an error, waits
// (bounded) for its copies and MMAs in flight and frees its tensor memory.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "split_store.cuh"
#include "tbk_internal.h"

namespace tbk {
namespace {

constexpr int kTM = 128;            // MMA M (output rows m per CTA)
constexpr int kTN = 128;            // complex output columns n per CTA
constexpr int kKS = kSplitTile;     // k per stage: one K tile of the stores (2 MMA k-steps of 16)
constexpr int kChunk = 4;           // stages per FP32 accumulation in tensor memory (128 k)
constexpr int kFlush = 32;          // chunks per FP32 register sum
constexpr int kStages = 3;
constexpr int kEpiWarps = 16;
constexpr int kMmaWarp = kEpiWarps;
constexpr int kTmaWarp = kMmaWarp + 1;
constexpr int kThreads = 32 * (kTmaWarp + 1);
constexpr uint32_t kAccCols = 2 * kTN;          // one accumulator: Re | Im
constexpr uint32_t kTmemCols = 2 * kAccCols;    // double-buffered: all of tensor memory
static_assert(kTmemCols == 512, "tensor memory");
constexpr uint32_t kWait = 1u << 24;

// stage layout: A re | A im | B re | B im; 128 rows of 128 bytes (32 hi, 32 lo) each
constexpr int kPart = kTM * kKS * 4;            // 16 KB
constexpr int kOffB = 2 * kPart;
constexpr int kStageBytes = 4 * kPart;          // 64 KB
constexpr int kSmemBytes = kStages * kStageBytes + 1024;   // + alignment slack
constexpr uint32_t kTxBytes = kStageBytes;
constexpr uint32_t kSBO = 1024;                 // 8 rows x 128 B swizzle atom
constexpr uint32_t kLo = kKS * 2;               // bytes from a row's hi halves to its lo halves

enum : int { kErrFull = 1, kErrEmpty = 2, kErrAcc = 4, kErrAccEmpty = 8, kErrDrain = 16, kErrRaw = 32 };

__device__ __forceinline__ uint32_t s_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint64_t* b, uint32_t c) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s_u32(b)), "r"(c) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s_u32(b)) : "memory");
}
__device__ __forceinline__ void bar_arrive_tx(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t parity) {
  for (uint32_t it = 0; it < kWait; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(s_u32(b)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int32_t x, int32_t y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          s_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(s_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tma_load_2d_mc(void* dst, const CUtensorMap* map, int32_t x, int32_t y, uint64_t* bar,
                                               uint16_t mask) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.multicast::cluster"
      " [%0], [%1, {%2, %3}], [%4], %5;" ::"r"(s_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(s_u32(bar)), "h"(mask)
      : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void tc_commit_mc(uint64_t* b, uint16_t mask) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          s_u32(b)),
      "h"(mask)
      : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* b) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s_u32(b))
               : "memory");
}
// Shared-memory matrix descriptor: K-major, 128-byte swizzle, version 1; the
// leading offset is unused for swizzled K-major operands, the stride offset is
// one 8-row swizzle atom.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)((kSBO >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// Instruction descriptors, kind::f16: D F32, A/B FP16, both K-major, N, M; A negated.
constexpr uint32_t idesc(int n, bool neg_a) {
  return (1u << 4) | (neg_a ? 1u << 13 : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTM >> 4) << 24);
}
// D (tmem) += A . B (shared-memory descriptors)
template <int N, bool NEG>
__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc(N, NEG)), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
// L, Rb: split stores of M blocks (split_store.cuh), seen by the tensor maps as rows of
// 64 halves: row (k tile * 2 + part) * M + m.  The CTA covers rows m0.., n0.. and K
// tiles [t0, t1).  Writes FP64 partial tiles (of s_m s_n mu).
__global__ void __launch_bounds__(kThreads, 1) mu_tc_kernel(const __grid_constant__ CUtensorMap map_l,
                                                            const __grid_constant__ CUtensorMap map_r, int32_t M,
                                                            int32_t n_tiles_k, int32_t tiles_split,
                                                            double* __restrict__ part, int* __restrict__ err) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full_bar[kStages], empty_bar[kStages], acc_full[2], acc_empty[2], drain_bar;
  __shared__ uint32_t tmem_base_s;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // blockIdx.x = m_tile * n_tiles_p + n_tile (n_tiles_p even): cluster pairs
  // share the m tile
  const int n_tiles_p = ((M + kTN - 1) / kTN + 1) & ~1;
  const int32_t m0 = (int32_t)(blockIdx.x / n_tiles_p) * kTM;
  const int32_t n0 = (int32_t)(blockIdx.x % n_tiles_p) * kTN;
  const uint32_t crank = cluster_rank();
  const int32_t t0 = (int32_t)blockIdx.y * tiles_split;
  const int32_t n_slabs = max(0, min(n_tiles_k - t0, tiles_split));
  const int32_t n_chunks = (n_slabs + kChunk - 1) / kChunk;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { bar_init(&full_bar[s], 1); bar_init(&empty_bar[s], 2); }
    for (int b = 0; b < 2; ++b) { bar_init(&acc_full[b], 1); bar_init(&acc_empty[b], kEpiWarps); }
    bar_init(&drain_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(&tmem_base_s)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();        // the peer's barriers exist before any multicast reaches them
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;

  if (warp == kTmaWarp) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_l) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_r) : "memory");
      int32_t issued = 0;
      for (int32_t s = 0; s < n_slabs; ++s) {
        const int st = s % kStages;
        const uint32_t ph = (uint32_t)(s / kStages) & 1u;
        if (!bar_wait(&empty_bar[st], ph ^ 1u)) { atomicOr(err, kErrEmpty); break; }
        unsigned char* sb = smem + (size_t)st * kStageBytes;
        bar_arrive_tx(&full_bar[st], kTxBytes);
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const int32_t row = ((t0 + s) * 2 + p) * M;
          // this CTA's half of the A box, to both CTAs of the pair
          tma_load_2d_mc(sb + p * kPart + crank * (kPart / 2), &map_l, 0, row + m0 + (int32_t)crank * (kTM / 2),
                         &full_bar[st], (uint16_t)0x3);
          tma_load_2d(sb + kOffB + p * kPart, &map_r, 0, row + n0, &full_bar[st]);
        }
        issued = s + 1;
      }
      // copies in flight complete before the CTA may leave (bounded)
      for (int32_t s = max(0, issued - kStages); s < issued; ++s)
        if (!bar_wait(&full_bar[s % kStages], (uint32_t)(s / kStages) & 1u)) { atomicOr(err, kErrRaw); break; }
    }
    __syncwarp();
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------ MMA issue
    if (lane == 0) {
      bool ok = true;
      int32_t s = 0;
      for (int32_t c = 0; c < n_chunks && ok; ++c) {
        const int b = c & 1;
        const uint32_t acc = tmem + (uint32_t)b * kAccCols;
        if (c >= 2) {
          if (!bar_wait(&acc_empty[b], (uint32_t)((c - 2) >> 1) & 1u)) { atomicOr(err, kErrAccEmpty); ok = false; break; }
          tc_fence_after();
        }
        const int32_t s_end = min(n_slabs, (c + 1) * kChunk);
        uint32_t accumulate = 0;
        for (; s < s_end; ++s) {
          const int st = s % kStages;
          if (!bar_wait(&full_bar[st], (uint32_t)(s / kStages) & 1u)) { atomicOr(err, kErrFull); ok = false; break; }
          tc_fence_after();
          const uint32_t sb = s_u32(smem + (size_t)st * kStageBytes);
#pragma unroll
          for (int j = 0; j < kKS / 16; ++j) {
            // part 0 re, 1 im; 16 halves = 32 B along the swizzled row
            auto A = [&](int p, uint32_t lo) { return smem_desc_sw128(sb + (uint32_t)(p * kPart + j * 32) + lo); };
            auto B = [&](int p, uint32_t lo) { return smem_desc_sw128(sb + (uint32_t)(kOffB + p * kPart + j * 32) + lo); };
#pragma unroll
            for (int q = 0; q < 3; ++q) {
              const uint32_t la = q == 2 ? kLo : 0, lb = q == 1 ? kLo : 0;     // hi hi, hi lo, lo hi
              mma_f16<2 * kTN, false>(acc, A(0, la), B(0, lb), accumulate);
              accumulate = 1;
              mma_f16<kTN, false>(acc, A(1, la), B(1, lb), 1u);
              mma_f16<kTN, true>(acc + kTN, A(1, la), B(0, lb), 1u);
            }
          }
          tc_commit_mc(&empty_bar[st], (uint16_t)0x3);   // frees the stage (in both CTAs) when these MMAs finish
        }
        if (ok) tc_commit(&acc_full[b]);   // accumulator chunk ready for the epilogue
      }
      // all MMAs this thread issued have completed before tensor memory is freed
      tc_commit(&drain_bar);
      if (!bar_wait(&drain_bar, 0)) atomicOr(err, kErrDrain);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ epilogue
    const int grp = warp & 3;           // TMEM lanes 32*grp .. 32*grp+31
    const int colq = warp >> 2;         // columns 64*colq ..: 0, 1 Re; 2, 3 Im
    float acc[64];
#pragma unroll
    for (int j = 0; j < 64; ++j) acc[j] = 0.f;
    double* dst = part + (((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * kAccCols + colq * 64) * kTM + 32 * grp + lane;
    bool fresh = true;                  // the partial tile has not been written yet
    for (int32_t c = 0; c < n_chunks; ++c) {
      const int b = c & 1;
      if (!bar_wait(&acc_full[b], (uint32_t)(c >> 1) & 1u)) { atomicOr(err, kErrAcc); break; }
      tc_fence_after();
      const uint32_t taddr = tmem + ((uint32_t)(32 * grp) << 16) + (uint32_t)b * kAccCols + (uint32_t)(colq * 64);
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        float v[16];
        tmem_ld16(taddr + 16u * h, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[16 * h + j] += v[j];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) bar_arrive(&acc_empty[b]);
      if ((c + 1) % kFlush == 0 || c + 1 == n_chunks) {
#pragma unroll
        for (int h = 0; h < 8; ++h) {                    // 8 values in flight: the sums fill the registers
          double o[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] = fresh ? 0.0 : __ldcg(dst + (8 * h + j) * kTM);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            __stcg(dst + (8 * h + j) * kTM, o[j] + (double)acc[8 * h + j]);
            acc[8 * h + j] = 0.f;
          }
          asm volatile("" ::: "memory");
        }
        fresh = false;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
  cluster_sync();        // no multicast or remote arrive targets a CTA that has left
}

// acc += (split-K partials summed in order) / (s_m s_n), one CTA row of tile rows per
// output column; nothing where the stores are marked unusable (the caller then forms the
// chunk from complex64 stores).  The mark goes to *bad_out beside the kernel's error, for one
// read-back.
__global__ void __launch_bounds__(kTM) mu_tc_reduce_kernel(const double* __restrict__ part, int32_t M, int32_t n_tiles_p,
                                                           int32_t tiles, int32_t nsplit, const float* __restrict__ sl,
                                                           int32_t sl_stride, const float* __restrict__ sr,
                                                           int32_t sr_stride, const int* __restrict__ bad,
                                                           int* __restrict__ bad_out, double2* __restrict__ acc) {
  const int32_t n = blockIdx.x, mt = blockIdx.y, m = mt * kTM + threadIdx.x;
  if (n == 0 && m == 0) *bad_out = *bad;
  if (m >= M || *bad) return;
  const int64_t tile = (int64_t)mt * n_tiles_p + n / kTN, step = (int64_t)tiles * kAccCols * kTM;
  const double* p = part + (tile * kAccCols + n % kTN) * kTM + threadIdx.x;
  double r = 0.0, i = 0.0;
#pragma unroll 4
  for (int32_t s = 0; s < nsplit; ++s) { r += p[s * step]; i += p[s * step + kTN * kTM]; }
  const double f = 1.0 / ((double)sl[m * sl_stride] * (double)sr[n * sr_stride]);   // a power of two
  acc[(int64_t)m * M + n].x += f * r;
  acc[(int64_t)m * M + n].y += f * i;
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// Tensor map over a split store: rows of 64 halves (128 B), `rows` rows, boxes of
// 64 halves x box_rows rows, 128-byte swizzle, zero fill past the end.
int block_map(CUtensorMap* map, const void* base, int64_t rows, uint32_t box_rows) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return fail(TBK_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  const cuuint64_t dims[2] = {64, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {128};
  const cuuint32_t box[2] = {64, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(TBK_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return TBK_OK;
}

}  // namespace

int mu_gemm_tc(const SplitStore& L, const SplitStore& Rb, int32_t M, int64_t K, double* mu_acc, bool* usable,
               cudaStream_t st) {
  if (M < 1 || K < 1) return fail(TBK_ERR_INVALID, "mu_gemm_tc: empty problem");
  if (((uintptr_t)L.data | (uintptr_t)Rb.data) & 15) return fail(TBK_ERR_INVALID, "mu_gemm_tc: blocks must be 16-byte aligned");
  static std::once_flag once;
  static cudaError_t configured = cudaSuccess;
  std::call_once(once, [] {
    configured = cudaFuncSetAttribute(mu_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
  });
  TBK_CUDA(configured);
  const int64_t tiles_k = (K + kKS - 1) / kKS;           // K tiles of the store (zero padded)
  if (tiles_k * 2 * (int64_t)M > INT32_MAX) return fail(TBK_ERR_UNSUPPORTED, "mu_gemm_tc: store too large for TMA rows");
  CUtensorMap map_l, map_r;
  TBK_TRY(block_map(&map_l, L.data, tiles_k * 2 * M, kTM / 2));
  TBK_TRY(block_map(&map_r, Rb.data, tiles_k * 2 * M, kTN));
  const int m_tiles = (M + kTM - 1) / kTM, n_tiles = ((M + kTN - 1) / kTN + 1) & ~1;   // pairs
  const int tiles = m_tiles * n_tiles;
  // split K (whole accumulation chunks per split) so that the CTAs fill whole
  // waves of one CTA per SM: the fewest splits whose last wave is >= 95% full
  const int sms = sm_count();
  const int64_t chunks = (tiles_k + kChunk - 1) / kChunk;
  int nsplit = 1;
  double best = 0.0;
  for (int ns = 1; ns <= 256 && ns <= chunks; ++ns) {
    const int64_t units = (int64_t)tiles * ns;
    const int64_t waves = (units + sms - 1) / sms;
    const double eff = (double)units / (double)(waves * sms);
    if (eff > best + 1e-9) { best = eff; nsplit = ns; }
    if (eff >= 0.95 && units >= sms) { nsplit = ns; break; }
  }
  const int64_t tiles_split = (chunks + nsplit - 1) / nsplit * kChunk;
  nsplit = (int)((tiles_k + tiles_split - 1) / tiles_split);
  DevBuf part, errb;
  TBK_TRY(part.alloc(sizeof(double) * (size_t)nsplit * tiles * kAccCols * kTM));
  TBK_TRY(errb.alloc(2 * sizeof(int)));
  TBK_CUDA(cudaMemsetAsync(errb.p, 0, 2 * sizeof(int), st));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles, nsplit);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  TBK_CUDA(cudaLaunchKernelEx(&cfg, mu_tc_kernel, map_l, map_r, M, (int32_t)tiles_k, (int32_t)tiles_split,
                              part.as<double>(), errb.as<int>()));
  mu_tc_reduce_kernel<<<dim3(M, m_tiles), kTM, 0, st>>>(part.as<double>(), M, n_tiles, tiles, nsplit, L.scale,
                                                        L.scale_stride, Rb.scale, Rb.scale_stride, L.bad,
                                                        errb.as<int>() + 1, reinterpret_cast<double2*>(mu_acc));
  TBK_CHECK_LAUNCH();
  int h[2] = {0, 0};
  TBK_CUDA(cudaMemcpyAsync(h, errb.p, sizeof(h), cudaMemcpyDeviceToHost, st));
  TBK_CUDA(cudaStreamSynchronize(st));
  if (h[0]) return fail(TBK_ERR_TIMEOUT, "tensor-core mu_nm kernel gave up waiting (code %d)", h[0]);
  *usable = h[1] == 0;
  return TBK_OK;
}

}  // namespace tbk
