// kubo.cu — Kubo conductivities from double-Chebyshev moments.
//
//   aL_m = g_m AL T_m(H~) BL |r>,   aR_n = g_n AR T_n(H~) BR |r>
//   mu_mn = sum_{sites, r} conj(aL_m) aR_n                        (a GEMM L^H R)
// Bastin sigma_xy: AL = BL = 1, AR = v_x, BR = v_y        (TB/snippets.h:306-456)
// Greenwood sigma_xx: AL = BL = v_x, AR = BR = 1           (TB/snippets.h:225-304)
// generate_V_moments: as Greenwood with the Dirichlet kernel (TB/snippets.h:491-518)
//
// The stored blocks (Cheb_first_kind_seq_on_bases, TB/numerical.h:333-344) are
// complex64 in HBM in a K-tiled layout: element k of block m lives at
// ((k / 16) * M + m) * 16 + k % 16, so the 16-element K slab of any run of
// consecutive blocks is contiguous (one coalesced 128-byte row per block) for
// the mu GEMM.  For the tensor-core GEMM they are FP16 (hi, lo) pairs of the same
// size (split_store.cuh).  They are produced by the fused recursion
// step of kpm.cu, in place on two blocks (T_m over T_{m-2}); the outer operator AL/AR
// is applied inside the step or after it, and each stored value rounded once.
// Random vectors are processed in chunks so that both sides fit the block
// budget; mu accumulates over chunks in FP64 on the device.  The Gamma
// contractions (FP64) and the Bastin integration follow TB/snippets.h:343-449.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cmath>
#include <cstdlib>
#include <mutex>
#include <type_traits>
#include <vector>

#include "kpm_device.cuh"
#include "split_store.cuh"
#include "tbk_internal.h"

namespace tbk {

namespace {

// ------------------------------------------------------------------ CUDA-core GEMM
// C[m][n] += sum_k conj(L[m][k]) R[n][k] for a K range per CTA (split-K), blocks in the
// K-tiled layout; FP32 products, FP32 sums over 32 values of k added into float-float pairs by
// TwoSum (48 bits, on the FP32 pipe: FP64 sums of the chunks took twice the time of the
// products), FP64 partial tiles.  64 x 32 complex outputs per CTA, 4 x 2 per thread.  What
// bounds it: the FP32 pipe and the issue slots in front of it (86% busy with scalar code, whose
// re += a b + c d is a product, an FMA and an addition).  So two neighbouring k share packed
// FMAs, one in each half (32 of them for 12 shared-memory reads), and the real and imaginary
// parts lie apart in shared memory, where a read then is a packed operand; rows are 34 words
// apart (no bank conflicts); the K tiles arrive by cp.async, three deep.  The halves are added
// before the TwoSum: 17 roundings of half a chunk's sum, where the scalar form made 32 of all
// of it.  M = 200, K = 56,064: 2.20 ms with 2 x 2 outputs per thread and FP64 sums, 0.81 ms
// scalar with 4 x 2, 0.68 ms so (53% of the issue slots, the FP32 pipe in front; 16-byte
// shared-memory reads: 0.70).
constexpr int kGT = 32;      // output tile (complex) per CTA side of the FP64 form, and n here
constexpr int kGM = 64;      // m
constexpr int kGStages = 3;
constexpr int kGPitch = 34;  // a K tile's 16 real parts, its 16 imaginary parts and two of padding

__device__ __forceinline__ void cp_async4(void* dst, const void* src, bool real) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(real ? 4 : 0)
               : "memory");
}
// hi + lo += v in both halves: TwoSum (Knuth)
__device__ __forceinline__ void ff_add2(uint64_t& hi, uint64_t& lo, uint64_t v) {
  const uint64_t s = f2_add(hi, v), b = f2_sub(s, hi);
  lo = f2_add(lo, f2_add(f2_sub(hi, f2_sub(s, b)), f2_sub(v, b)));
  hi = s;
}

// K tiles [t0, t1) of blockIdx.z; M blocks per K tile in both stores
__global__ void __launch_bounds__(256) mu_gemm_cc_kernel(const float2* __restrict__ L, const float2* __restrict__ Rb,
                                                         int32_t M, int64_t tiles, int64_t tiles_split,
                                                         double2* __restrict__ part) {
  __shared__ __align__(16) float sm[kGStages][kGM + kGT][kGPitch];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int32_t m0 = blockIdx.y * kGM, n0 = blockIdx.x * kGT;
  const int64_t t0 = (int64_t)blockIdx.z * tiles_split, t1 = min(tiles, t0 + tiles_split);
  // 6 values of a stage per thread: value tx of rows ty, ty + 16, ...; rows past M read as zero
  auto load = [&](int64_t t) {
    if (t < t1) {
      float(*st)[kGPitch] = sm[(t - t0) % kGStages];
#pragma unroll
      for (int q = 0; q < (kGM + kGT) / 16; ++q) {
        const int row = ty + 16 * q;
        const bool left = row < kGM;
        const int32_t b = left ? m0 + row : n0 + row - kGM;
        const float2* src = (left ? L : Rb) + (t * M + min(b, M - 1)) * 16 + tx;
        cp_async4(&st[row][tx], &src->x, b < M);
        cp_async4(&st[row][16 + tx], &src->y, b < M);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // sums over even | odd k; float-float sums of re | im
  uint64_t ar[4][2] = {}, ai[4][2] = {}, hi[4][2] = {}, lo[4][2] = {};
  load(t0);
  load(t0 + 1);
  for (int64_t t = t0; t < t1; ++t) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const float(*st)[kGPitch] = sm[(t - t0) % kGStages];
    auto pair = [&](int row, int at) { return *reinterpret_cast<const uint64_t*>(&st[row][at]); };
#pragma unroll
    for (int kk = 0; kk < 16; kk += 2) {
      uint64_t ax[4], ay[4], bx[2], by[2];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        ax[i] = pair(ty + 16 * i, kk);
        ay[i] = pair(ty + 16 * i, 16 + kk);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        bx[j] = pair(kGM + tx + 16 * j, kk);
        by[j] = pair(kGM + tx + 16 * j, 16 + kk);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint64_t nx = bx[j] ^ 0x8000000080000000ull;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          // conj(a) * b
          ar[i][j] = f2_fma(ax[i], bx[j], ar[i][j]);
          ai[i][j] = f2_fma(ax[i], by[j], ai[i][j]);
          ar[i][j] = f2_fma(ay[i], by[j], ar[i][j]);
          ai[i][j] = f2_fma(ay[i], nx, ai[i][j]);
        }
      }
    }
    load(t + 2);                 // over the stage that every thread left before this barrier
    // FP32 sums cover two K tiles (32 values of k) only: long FP32 accumulations lose accuracy
    // where the sum is much smaller than its terms (mu_nm at large m, n)
    if (((t - t0) & 1) || t + 1 == t1) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float r0, r1, i0, i1;
          f2_unpack(ar[i][j], r0, r1);
          f2_unpack(ai[i][j], i0, i1);
          ff_add2(hi[i][j], lo[i][j], f2_pack(__fadd_rn(r0, r1), __fadd_rn(i0, i1)));
          ar[i][j] = ai[i][j] = 0;
        }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int32_t m = m0 + ty + 16 * i, n = n0 + tx + 16 * j;
      float hr, hm, lr, lm;
      f2_unpack(hi[i][j], hr, hm);
      f2_unpack(lo[i][j], lr, lm);
      // an infinite sum's second part is NaN: the first alone then
      if (m < M && n < M)
        part[((int64_t)blockIdx.z * M + m) * M + n] =
            make_double2(isfinite(hr) ? (double)hr + (double)lr : (double)hr, isfinite(hm) ? (double)hm + (double)lm : (double)hm);
    }
}

__global__ void mu_split_reduce_kernel(const double2* __restrict__ part, int32_t M, int32_t nsplit,
                                       double2* __restrict__ acc) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= (int64_t)M * M) return;
  double r = 0.0, i = 0.0;
  for (int32_t s = 0; s < nsplit; ++s) { const double2 v = part[(int64_t)s * M * M + q]; r += v.x; i += v.y; }
  acc[q].x += r;
  acc[q].y += i;
}

// acc += L^H R of complex64 K-tiled stores.  K is split into at most 64 partial M x M
// blocks of 512 values of k or more, and at least into those of 16,384 or K / 64: within
// that, the fewest splits whose CTAs (two per SM) leave at most a twentieth of their last
// wave empty, or the split that leaves least (M = 32, K = 30,000: 105 -> 56 us; M = 128, K =
// 65,536: 253 -> 245).
int mu_gemm_cc(const float2* L, const float2* Rb, int32_t M, int64_t K, DevBuf* part, double2* acc, cudaStream_t st) {
  const int64_t tiles = (K + 15) / 16;
  const dim3 out((M + kGT - 1) / kGT, (M + kGM - 1) / kGM);
  const int64_t wave = 2LL * sm_count(), longest = std::max<int64_t>(1024, (tiles + 63) / 64);
  int64_t split = longest;
  double best = 0.0;
  for (int64_t ns = (tiles + longest - 1) / longest; ns <= 64 && (ns == 1 || tiles / ns >= 32); ++ns) {
    const int64_t units = (int64_t)out.x * out.y * ns, waves = (units + wave - 1) / wave;
    const double eff = (double)units / (double)(waves * wave);
    if (eff <= best + 1e-9) continue;
    best = eff;
    split = (tiles + ns - 1) / ns;
    if (eff >= 0.95) break;
  }
  const int32_t nsplit = (int32_t)((tiles + split - 1) / split);
  const size_t need = sizeof(double2) * (size_t)nsplit * M * M;
  if (part->bytes < need) TBK_TRY(part->alloc(need));
  mu_gemm_cc_kernel<<<dim3(out.x, out.y, nsplit), 256, 0, st>>>(L, Rb, M, tiles, split, part->as<double2>());
  TBK_CHECK_LAUNCH();
  mu_split_reduce_kernel<<<(unsigned)(((int64_t)M * M + 255) / 256), 256, 0, st>>>(part->as<double2>(), M, nsplit, acc);
  TBK_CHECK_LAUNCH();
  return TBK_OK;
}

// FP64 reference GEMM on complex128 K-tiled blocks: C[m][n] += sum_k
// conj(L[m][k]) R[n][k] with every product and sum in FP64 (split-K partials,
// reduced in a fixed order by mu_split_reduce_kernel).
constexpr int kGK64 = 16;
__global__ void __launch_bounds__(256) mu_gemm_f64_kernel(const double2* __restrict__ L,
                                                          const double2* __restrict__ Rb, int32_t M, int64_t K,
                                                          int64_t ksplit, double2* __restrict__ part) {
  __shared__ double2 Ls[kGT][kGK64 + 1], Rs[kGT][kGK64 + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int32_t m0 = blockIdx.y * kGT, n0 = blockIdx.x * kGT;
  const int64_t k0 = (int64_t)blockIdx.z * ksplit;
  const int64_t k1 = min(K, k0 + ksplit);
  double dr[2][2] = {{0, 0}, {0, 0}}, di[2][2] = {{0, 0}, {0, 0}};
  for (int64_t kb = k0; kb < k1; kb += kGK64) {
    for (int q = threadIdx.x; q < kGT * kGK64; q += 256) {
      const int row = q / kGK64, kk = q % kGK64;
      const int64_t k = kb + kk;
      const double2 z = make_double2(0.0, 0.0);
      Ls[row][kk] = (m0 + row < M && k < k1) ? L[((k >> 4) * M + (m0 + row)) * 16 + (k & 15)] : z;
      Rs[row][kk] = (n0 + row < M && k < k1) ? Rb[((k >> 4) * M + (n0 + row)) * 16 + (k & 15)] : z;
    }
    __syncthreads();
#pragma unroll 4
    for (int kk = 0; kk < kGK64; ++kk) {
      const double2 a[2] = {Ls[ty * 2][kk], Ls[ty * 2 + 1][kk]};
      const double2 b[2] = {Rs[tx * 2][kk], Rs[tx * 2 + 1][kk]};
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          dr[i][j] = fma(a[i].x, b[j].x, fma(a[i].y, b[j].y, dr[i][j]));
          di[i][j] = fma(a[i].x, b[j].y, fma(-a[i].y, b[j].x, di[i][j]));
        }
    }
    __syncthreads();
  }
  for (int i = 0; i < 2; ++i)
    for (int j = 0; j < 2; ++j) {
      const int32_t m = m0 + ty * 2 + i, n = n0 + tx * 2 + j;
      if (m < M && n < M) part[((int64_t)blockIdx.z * M + m) * M + n] = make_double2(dr[i][j], di[i][j]);
    }
}

// work block -> block m of a complex128 K-tiled store (the FP64 reference form)
__device__ __forceinline__ double2 to_c128(double2 v) { return v; }
__device__ __forceinline__ double2 to_c128(float2 v) { return make_double2(v.x, v.y); }
__device__ __forceinline__ double2 to_c128(dd2 v) {
  return make_double2((double)v.x.hi + (double)v.x.lo, (double)v.y.hi + (double)v.y.lo);
}
template <typename CT>
__global__ void store_block64_kernel(const CT* __restrict__ src, double2* __restrict__ store, int32_t m, int32_t M,
                                     int64_t n) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
    store[((q >> 4) * M + m) * 16 + (q & 15)] = to_c128(src[q]);
}

// work block -> block m of the complex64 K-tiled store (complex128 work blocks
// are rounded once per element); 16 consecutive k form one contiguous 128-byte
// row of the tile
__device__ __forceinline__ float2 to_c64(double2 v) { return make_float2(__double2float_rn(v.x), __double2float_rn(v.y)); }
__device__ __forceinline__ float2 to_c64(float2 v) { return v; }
__device__ __forceinline__ float2 to_c64(dd2 v) { return make_float2(__fadd_rn(v.x.hi, v.x.lo), __fadd_rn(v.y.hi, v.y.lo)); }
// (blockIdx.y: several blocks of n values in a row)
template <typename CT>
__global__ void round_block_kernel(const CT* __restrict__ src, float2* __restrict__ store, int32_t m, int32_t M,
                                   int64_t n) {
  src += blockIdx.y * n;
  m += blockIdx.y;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
    store[((q >> 4) * M + m) * 16 + (q & 15)] = to_c64(src[q]);
}

// columns [c0, c0 + Rc) of a 2 Rc-wide site-major block <- an Rc-wide block
template <typename CT>
__global__ void pack_cols_kernel(int64_t n_pad, int32_t Rc, int32_t c0, const CT* __restrict__ src,
                                 CT* __restrict__ dst) {
  const int64_t tot = n_pad * Rc;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < tot; q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = q / Rc;
    dst[row * 2 * Rc + c0 + (q - row * Rc)] = src[q];
  }
}
// block m of a K-tiled store (k = row * Rc + column) <- columns [c0, c0 + Rc)
// of a 2 Rc-wide block, rounded to complex64
template <typename CT>
__global__ void round_cols_kernel(int64_t n_pad, int32_t Rc, int32_t c0, const CT* __restrict__ src,
                                  float2* __restrict__ store, int32_t m, int32_t M) {
  const int64_t tot = n_pad * Rc;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < tot; q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = q / Rc;
    store[((q >> 4) * M + m) * 16 + (q & 15)] = to_c64(src[row * 2 * Rc + c0 + (q - row * Rc)]);
  }
}

// The largest row sum of |a_ij| (|re| + |im| of complex entries) of an operator: |A x| is at
// most that many times |x|, in the maximum and, for a Hermitian or antihermitian A, in the
// root mean square.  *gain is the FP32 bits of the largest so far (NaN above infinity).
__global__ void __launch_bounds__(256) operator_gain_kernel(int32_t n, const int32_t* __restrict__ soff,
                                                            const float* __restrict__ val,
                                                            const float* __restrict__ diag, int vw,
                                                            unsigned int* __restrict__ gain) {
  const int32_t r = blockIdx.x * 256 + threadIdx.x;
  float sum = 0.f;
  if (r < n) {
    const int64_t base = soff[r >> 5] + (r & 31);
    const int32_t w = (soff[(r >> 5) + 1] - soff[r >> 5]) >> 5;
    for (int q = 0; q < vw; ++q) {
      sum += fabsf(diag[(int64_t)vw * r + q]);
      for (int32_t k = 0; k < w; ++k) sum += fabsf(val[vw * (base + (int64_t)k * 32) + q]);
    }
  }
  const unsigned int m = __reduce_max_sync(0xffffffffu, __float_as_uint(sum));
  if ((threadIdx.x & 31) == 0 && m != 0u) atomicMax(gain, m);
}

// The scale of an FP16-pair store (split_store.cuh) of blocks gain x, from the n values of the
// first x: a power of two that takes gain times their root mean square to 2^6, or gain times
// their maximum to 2^13 where that is less.  Not from the first block itself: an operator that
// (nearly) vanishes on the start vectors does not vanish on T_m of them.  gain null: 1.  The
// last CTA to finish sums the others' partials in a fixed order.  (blockIdx.y: several blocks of n
// values in a row, each with a scale, partials and a counter of its own.)
constexpr int kStatThreads = 256;
template <typename CT>
__global__ void __launch_bounds__(kStatThreads) split_scale_kernel(const CT* __restrict__ src, int64_t n,
                                                                   double* __restrict__ part,
                                                                   unsigned int* __restrict__ count,
                                                                   const float* __restrict__ gain,
                                                                   float* __restrict__ scale, int* __restrict__ bad) {
  src += blockIdx.y * n;
  part += 2 * (int64_t)blockIdx.y * gridDim.x;
  count += blockIdx.y;
  scale += blockIdx.y;
  float big = 0.f;
  double sum = 0.0;
  for (int64_t q = (int64_t)blockIdx.x * kStatThreads + threadIdx.x; q < n; q += (int64_t)gridDim.x * kStatThreads) {
    const float2 v = to_c64(src[q]);
    const float m = fmaxf(fabsf(v.x), fabsf(v.y));
    big = (v.x != v.x || v.y != v.y) ? INFINITY : fmaxf(big, m);
    sum += (double)v.x * v.x + (double)v.y * v.y;
  }
  __shared__ double s_sum[kStatThreads / 32];
  __shared__ float s_big[kStatThreads / 32];
  __shared__ bool last;
  auto block_reduce = [&](double& v, float& m) {          // valid in warp 0
    __syncthreads();
    for (int pass = 0; pass < 2; ++pass) {
      for (int o = 16; o > 0; o >>= 1) {
        v += __shfl_xor_sync(0xffffffffu, v, o);
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      }
      if (pass == 1) break;
      if ((threadIdx.x & 31) == 0) { s_sum[threadIdx.x >> 5] = v; s_big[threadIdx.x >> 5] = m; }
      __syncthreads();
      if (threadIdx.x >= 32) break;
      const bool in = threadIdx.x < kStatThreads / 32;
      v = in ? s_sum[threadIdx.x] : 0.0;
      m = in ? s_big[threadIdx.x] : 0.f;
    }
  };
  block_reduce(sum, big);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = sum;
    part[2 * blockIdx.x + 1] = big;
    __threadfence();
    last = atomicAdd(count, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  sum = 0.0;
  big = 0.f;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += kStatThreads) {
    sum += __ldcg(part + 2 * b);
    big = fmaxf(big, (float)__ldcg(part + 2 * b + 1));
  }
  block_reduce(sum, big);
  if (threadIdx.x == 0) {
    const double f = gain ? (double)*gain : 1.0, mx = f * big, rms = f * sqrt(sum / (2.0 * (double)n));
    float s = 1.f;                                       // zero blocks
    if (!(mx < (double)INFINITY)) *bad = 1;
    else if (mx > 0.0) s = ldexpf(1.f, max(-120, min(120, min(12 - ilogb(mx), 6 - ilogb(rms)))));
    *scale = s;
    *count = 0;
  }
}

// work block -> block m of an FP16-pair store (blockIdx.y as above)
template <typename CT>
__global__ void split_block_kernel(const CT* __restrict__ src, __half* __restrict__ store, int32_t m, int32_t M,
                                   int64_t n, const float* __restrict__ scale, int* __restrict__ bad) {
  src += blockIdx.y * n;
  m += blockIdx.y;
  const float s = __ldg(scale + blockIdx.y);
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const float2 v = to_c64(src[q]);
    split_put(store, M, m, q, v.x, v.y, s, bad);
  }
}
// the same from columns [c0, c0 + Rc) of a 2 Rc-wide block
template <typename CT>
__global__ void split_cols_kernel(int64_t n_pad, int32_t Rc, int32_t c0, const CT* __restrict__ src,
                                  __half* __restrict__ store, int32_t m, int32_t M, const float* __restrict__ scale,
                                  int* __restrict__ bad) {
  const float s = __ldg(scale);
  const int64_t tot = n_pad * Rc;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < tot; q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = q / Rc;
    const float2 v = to_c64(src[row * 2 * Rc + c0 + (q - row * Rc)]);
    split_put(store, M, m, q, v.x, v.y, s, bad);
  }
}

__global__ void mu_kernel_scale_kernel(double2* __restrict__ mu, const double* __restrict__ g, int32_t M) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= (int64_t)M * M) return;
  const double s = g[q / M] * g[q % M];
  mu[q].x *= s;
  mu[q].y *= s;
}

// ------------------------------------------------------------------ Gamma contractions (FP64)
// Both spectra are double trigonometric sums over (m, n).  The product rule
//   cos(m th) e^{i n th} = (e^{i (n+m) th} + e^{i (n-m) th}) / 2
// collects them into one series over q = n + m and q = |n - m|: the M^2 moments
// are summed once along their antidiagonals and diagonals, and each energy then
// costs a series of 2M - 1 terms instead of M^2.  With w_mn = a_m a_n mu_mn / 2,
//   U_q = sum_{n+m=q} w,  D_q = sum_{n+m=q} (n - m) w,  V_d = sum_{n-m=d} w,
//   P_q = V_q + V_-q (V_0 at q = 0),  I_q = V_q - V_-q,  A = U + P,  B = D + q I:
//   zeta  (1-e^2)^2 vol = sum_q cos(q th) (2 e A_q - i s B_q) + sin(q th) (s q A_q + 2 i e I_q)
//   sigma (1-e^2) R     = - sum_q cos(q th) Re A_q
// where e = cos th and s = sin th.  As M x M sums per energy the two were bound by
// the FP64 pipe (6 FMAs per moment and energy): M = 512, 1,024 energies took 4.00 +
// 0.94 ms in their kernels, 5.62 ms for both calls with the host copies; as series
// both calls take 0.25 ms, nearly all of it copies and launches.
constexpr int kDiagThreads = 128;
constexpr int kDiagRows = 16;       // rows of mu per CTA: M = 512 gives 256 CTAs
constexpr int kSeriesThreads = 128; // evaluation: one warp per energy

// Partial sums over kDiagRows rows: thread t takes the antidiagonal n + m = t and
// the diagonal n - m = t - (M - 1), both read along rows (coalesced).
// part: per row chunk, planes U, V and (BASTIN) D of 2M - 1 values.
template <bool BASTIN>
__global__ void __launch_bounds__(kDiagThreads) diag_sums_kernel(const double2* __restrict__ mu, int32_t M,
                                                                 double2* __restrict__ part) {
  const int32_t L = 2 * M - 1;
  const int32_t t = blockIdx.x * kDiagThreads + threadIdx.x;
  if (t >= L) return;
  const int32_t m0 = blockIdx.y * kDiagRows;
  double2 u = make_double2(0.0, 0.0), v = u, d = u;
#pragma unroll 8
  for (int32_t k = 0; k < kDiagRows; ++k) {
    const int32_t m = m0 + k;
    if (m >= M) break;
    const double am = m == 0 ? 0.5 : 1.0;                  // a_m a_n / 2 = 2 with a_0 = 1, a_k = 2
    const int32_t n = t - m, n2 = t - (M - 1) + m;
    if (n >= 0 && n < M) {
      const double2 x = mu[(int64_t)m * M + n];
      const double f = am * (n == 0 ? 1.0 : 2.0);
      u.x += f * x.x;
      if constexpr (BASTIN) {
        const double g = f * (double)(n - m);
        u.y += f * x.y;
        d.x += g * x.x;
        d.y += g * x.y;
      }
    }
    if (n2 >= 0 && n2 < M) {
      const double2 x = mu[(int64_t)m * M + n2];
      const double f = am * (n2 == 0 ? 1.0 : 2.0);
      v.x += f * x.x;
      if constexpr (BASTIN) v.y += f * x.y;
    }
  }
  double2* p = part + (int64_t)blockIdx.y * (BASTIN ? 3 : 2) * L;
  p[t] = u;
  p[L + t] = v;
  if constexpr (BASTIN) p[2 * L + t] = d;
}

// The row chunks summed, then the series coefficients A, (BASTIN) B and I: 32 q per CTA,
// its 8 warps taking every 8th chunk (one thread per q waits for 5 loads a chunk, 20 us at
// 32 chunks).
constexpr int kCoefWarps = 8;
template <bool BASTIN>
__global__ void __launch_bounds__(32 * kCoefWarps) series_coef_kernel(const double2* __restrict__ part, int32_t M,
                                                                      int32_t chunks, double2* __restrict__ coef) {
  const int32_t L = 2 * M - 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int32_t q = blockIdx.x * 32 + lane;
  double2 v[4] = {};                                       // U, D, V_q, V_-q
  auto add = [](double2& s, double2 x) { s.x += x.x; s.y += x.y; };
  if (q < L)
    for (int32_t c = warp; c < chunks; c += kCoefWarps) {
      const double2* p = part + (int64_t)c * (BASTIN ? 3 : 2) * L;
      add(v[0], p[q]);
      if constexpr (BASTIN) add(v[1], p[2 * L + q]);
      if (q < M) {
        add(v[2], p[L + (M - 1) + q]);
        add(v[3], p[L + (M - 1) - q]);
      }
    }
  __shared__ double2 sh[kCoefWarps][4][32];
#pragma unroll
  for (int k = 0; k < 4; ++k) sh[warp][k][lane] = v[k];
  __syncthreads();
  if (warp != 0 || q >= L) return;
  for (int w = 1; w < kCoefWarps; ++w)
#pragma unroll
    for (int k = 0; k < 4; ++k) add(v[k], sh[w][k][lane]);
  const double2 u = v[0], d = v[1], vp = v[2];
  const double2 vm = q == 0 ? make_double2(0.0, 0.0) : v[3];        // the main diagonal counts once
  const double2 i = q == 0 ? vm : make_double2(vp.x - vm.x, vp.y - vm.y);
  coef[q] = make_double2(u.x + vp.x + vm.x, u.y + vp.y + vm.y);
  if constexpr (BASTIN) {
    coef[L + q] = make_double2(d.x + q * i.x, d.y + q * i.y);
    coef[2 * L + q] = i;
  }
}

// One warp per energy: lane l takes q = l, l + 32, ..., with (cos, sin)(q th)
// advanced by the rotation through 32 th.
template <bool BASTIN>
__global__ void __launch_bounds__(kSeriesThreads) series_eval_kernel(const double2* __restrict__ coef, int32_t M,
                                                                     int32_t n_eps, const double* __restrict__ eps,
                                                                     double norm, double* __restrict__ out) {
  const int32_t k = blockIdx.x * (kSeriesThreads / 32) + (threadIdx.x >> 5);
  if (k >= n_eps) return;
  const int32_t lane = threadIdx.x & 31, L = 2 * M - 1;
  const double e = eps[k], th = acos(e);
  double c, s, cr, sr;
  sincos(lane * th, &s, &c);
  sincos(32 * th, &sr, &cr);
  double2 s1 = make_double2(0.0, 0.0), s2 = s1, s3 = s1, s4 = s1;   // A cos, B cos, q A sin, I sin
  for (int32_t q = lane; q < L; q += 32) {
    const double2 a = coef[q];
    s1.x += a.x * c;
    if constexpr (BASTIN) {
      const double2 b = coef[L + q], i = coef[2 * L + q];
      const double qs = q * s;
      s1.y += a.y * c;
      s2.x += b.x * c;
      s2.y += b.y * c;
      s3.x += a.x * qs;
      s3.y += a.y * qs;
      s4.x += i.x * s;
      s4.y += i.y * s;
    }
    const double cn = c * cr - s * sr;
    s = s * cr + c * sr;
    c = cn;
  }
  // e^2 rounded, as in the formulas themselves (TB/snippets.h:343-349): near e = 1 the weight 1/(1 - e^2)^2
  // shows its last bits, 3.4e-11 at the first of 1,024 nodes
  const double q = __dsub_rn(1.0, __dmul_rn(e, e)), sn = sqrt(q);
  double zr, zi = 0.0;
  if constexpr (BASTIN) {
    zr = 2.0 * e * s1.x + sn * s2.y + sn * s3.x - 2.0 * e * s4.y;
    zi = 2.0 * e * s1.y - sn * s2.x + sn * s3.y + 2.0 * e * s4.x;
  } else {
    zr = s1.x;
  }
  for (int o = 16; o > 0; o >>= 1) {
    zr += __shfl_xor_sync(0xffffffffu, zr, o);
    if constexpr (BASTIN) zi += __shfl_xor_sync(0xffffffffu, zi, o);
  }
  if (lane == 0) {
    if constexpr (BASTIN) {
      const double den = q * q * norm;
      out[2 * k] = zr / den;
      out[2 * k + 1] = zi / den;
    } else {
      out[k] = -zr / q / norm;
    }
  }
}

template <bool BASTIN>
int moment_series(int32_t M, const double* mu, int32_t n_eps, const double* eps, double norm, double* out,
                  cudaStream_t st) {
  ScratchScope scope(st);
  const int32_t L = 2 * M - 1, chunks = (M + kDiagRows - 1) / kDiagRows, planes = BASTIN ? 3 : 2;
  const size_t mb = sizeof(double2) * (size_t)M * M, cb = sizeof(double2) * (size_t)planes * L;
  const size_t ob = sizeof(double) * (BASTIN ? 2 : 1) * (size_t)n_eps;
  DevBuf ws;                                             // one workspace: mu, partials, coefficients, results, energies
  TBK_TRY(ws.alloc(mb + cb * (chunks + 1) + ob + sizeof(double) * n_eps));
  double2* dm = ws.as<double2>();
  double2* part = dm + (size_t)M * M;
  double2* coef = part + (size_t)chunks * planes * L;
  double* dz = reinterpret_cast<double*>(coef + (size_t)planes * L);
  double* de = dz + (BASTIN ? 2 : 1) * (size_t)n_eps;
  TBK_CUDA(cudaMemcpyAsync(dm, mu, mb, cudaMemcpyHostToDevice, st));
  TBK_CUDA(cudaMemcpyAsync(de, eps, sizeof(double) * n_eps, cudaMemcpyHostToDevice, st));
  const int32_t qb = (L + kDiagThreads - 1) / kDiagThreads;
  diag_sums_kernel<BASTIN><<<dim3(qb, chunks), kDiagThreads, 0, st>>>(dm, M, part);
  TBK_CHECK_LAUNCH();
  series_coef_kernel<BASTIN><<<(L + 31) / 32, 32 * kCoefWarps, 0, st>>>(part, M, chunks, coef);
  TBK_CHECK_LAUNCH();
  constexpr int kPer = kSeriesThreads / 32;
  series_eval_kernel<BASTIN><<<(n_eps + kPer - 1) / kPer, kSeriesThreads, 0, st>>>(coef, M, n_eps, de, norm, dz);
  TBK_CHECK_LAUNCH();
  TBK_CUDA(cudaMemcpyAsync(out, dz, ob, cudaMemcpyDeviceToHost, st));
  TBK_CUDA(cudaStreamSynchronize(st));
  return TBK_OK;
}

// timing of the last tbk_kubo_mu call (CUDA events on the caller's stream)
struct KuboTiming { double ms_blocks = 0, ms_gemm = 0, gemm_flops = 0, block_bytes = 0; int chunks = 0; };
KuboTiming g_kubo_timing;        // the last solve's timing (calls may come from several threads)
std::mutex g_kubo_timing_mu;

// TBK_TRACE=1: tbk_kubo_mu prints the host time of its phases to stderr
// (synchronising at each phase boundary, which it otherwise does not)
struct PhaseTrace {
  bool on;
  cudaStream_t st;
  std::chrono::steady_clock::time_point t0;
  std::vector<std::pair<const char*, double>> marks;
  explicit PhaseTrace(cudaStream_t s) : st(s), t0(std::chrono::steady_clock::now()) {
    const char* e = getenv("TBK_TRACE");
    on = e && atoi(e) != 0;
  }
  void mark(const char* name) {
    if (!on) return;
    cudaStreamSynchronize(st);
    marks.emplace_back(name, std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count());
  }
  ~PhaseTrace() {
    if (!on) return;
    double prev = 0.0;
    fprintf(stderr, "tbk_kubo_mu phases (ms):");
    for (auto& m : marks) {
      fprintf(stderr, " %s %.2f", m.first, m.second - prev);
      prev = m.second;
    }
    fprintf(stderr, "\n");
  }
};

// The stored blocks and work blocks of a call made outside a server come
// from a stream-ordered pool that keeps up to kKuboPoolKeep bytes between
// calls: stores of that size are then reused instead of mapped and unmapped
// every call (the 256 x 256, M = 512, R = 16 Bastin case: 8.6 GB, whose
// cudaFree took 5.7 ms of a 36 ms call).
// Larger stores keep plain allocations (a 137 GB store from the pool, then
// trimmed, measured 0.2 s slower than cudaMalloc and cudaFree); each call
// trims the pool back to kKuboPoolKeep before it returns.
constexpr uint64_t kKuboPoolKeep = 16ull << 30;
cudaMemPool_t kubo_pool() {
  static std::mutex mu;
  static cudaMemPool_t pools[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return nullptr; }
  std::lock_guard<std::mutex> lk(mu);
  if (!pools[dev]) {
    cudaMemPoolProps pp = {};
    pp.allocType = cudaMemAllocationTypePinned;
    pp.location.type = cudaMemLocationTypeDevice;
    pp.location.id = dev;
    if (cudaMemPoolCreate(&pools[dev], &pp) != cudaSuccess) {
      cudaGetLastError();
      pools[dev] = nullptr;
      return nullptr;
    }
    uint64_t keep = kKuboPoolKeep;
    cudaMemPoolSetAttribute(pools[dev], cudaMemPoolAttrReleaseThreshold, &keep);
  }
  return pools[dev];
}

// f(block as its element type) for a work block in a recursion precision
template <typename Fn>
int with_block(int prec, const void* p, Fn&& f) {
  if (prec == TBK_PREC_FP64) f(static_cast<const double2*>(p));
  else if (prec == TBK_PREC_DD) f(static_cast<const dd2*>(p));
  else f(static_cast<const float2*>(p));
  TBK_CHECK_LAUNCH();
  return TBK_OK;
}

// Scratch of split_scale_kernel, the two sides' scales and the flag of values that do
// not fit.
struct SplitScales {
  DevBuf buf;                  // 7 words: scale of the left, of the right side; bad; count, gain of each side; the partials
  int alloc(cudaStream_t st) {
    TBK_TRY(buf.alloc(sizeof(double) * (4 + 8 * sm_count())));
    TBK_CUDA(cudaMemsetAsync(buf.p, 0, 4 * sizeof(double), st));
    return TBK_OK;
  }
  float* scale(int h) const { return buf.as<float>() + h; }
  int* bad() const { return buf.as<int>() + 2; }
  // the output operator of side h
  int set_operator(int h, const EllDev& E, cudaStream_t st) const {
    operator_gain_kernel<<<(E.n_rows + 255) / 256, 256, 0, st>>>(E.n_rows, E.slice_off.as<int32_t>(), E.val32.as<float>(),
                                                                 E.diag32.as<float>(), E.cplx ? 2 : 1,
                                                                 buf.as<unsigned int>() + 5 + h);
    TBK_CHECK_LAUNCH();
    return TBK_OK;
  }
  // h: the side, each with scratch of its own; gain: the stored blocks are its operator's products
  template <typename CT>
  void find(const CT* src, int64_t n, float* out, int h, bool gain, cudaStream_t st) const {
    const int g = (int)std::max<int64_t>(1, std::min<int64_t>((n + kStatThreads - 1) / kStatThreads, 2 * sm_count()));
    split_scale_kernel<CT><<<g, kStatThreads, 0, st>>>(src, n, buf.as<double>() + 4 + 4 * h * sm_count(),
                                                       buf.as<unsigned int>() + 3 + h,
                                                       gain ? buf.as<float>() + 5 + h : nullptr, out, bad());
  }
};

// Blocks of up to this size leave much of the GPU idle in one recursion: both sides of
// square 256x256 with a flux, M = 512, 16 vectors (8 MB a block), took 9.8 ms one after the
// other, the operator's products in a pass of their own, and take 7.9 ms on two streams;
// honeycomb 91x77, M = 200, 3 vectors, 1.25 and 0.75 ms.  The stream costs some 20 us a call: whole
// calls of 1 and 2 streams, square 80x80, 8 vectors, M = 4: 261, 262 us; 12: 333, 309; 24: 427, 367.
constexpr double kDualBlock = 16e6;
constexpr int64_t kDualSteps = 8;     // steps a side

// A stream beside the caller's, of its priority, for the length of a call
struct SecondStream {
  cudaStream_t st = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  int create(cudaStream_t beside) {
    int prio = 0;
    TBK_CUDA(cudaStreamGetPriority(beside, &prio));
    TBK_CUDA(cudaStreamCreateWithPriority(&st, cudaStreamNonBlocking, prio));
    TBK_CUDA(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
    TBK_CUDA(cudaEventCreateWithFlags(&join, cudaEventDisableTiming));
    return TBK_OK;
  }
  ~SecondStream() {
    if (st) {
      cudaStreamSynchronize(st);
      cudaStreamDestroy(st);
    }
    if (fork) cudaEventDestroy(fork);
    if (join) cudaEventDestroy(join);
  }
};

// Vectors per chunk of the block recursions (n_pad rows, M blocks a side, sel bytes a stored
// value; both stored sides within the budget; 1 when no width fits).  A chunk costs the two
// sides' steps, each a launch (4.5 us), the matrix (5 bytes a row) and 32 bytes a row and
// vector, twice as fast where the two vectors stay in L2 beside the stores that pass through
// it (FCC 64^3: 8.5 us a step at width 4, 20.7 at 8), then the GEMM's products; stores that
// the pool does not keep cost their mapping every call (137 GB: 57 ms to free, 5 to
// allocate).  So large problems take narrow chunks: FCC 128^3, M = 1024, R = 8: 648 ms at
// width 4, 625 at 2, 721 at 1 (complex64 lanes carry two vectors: 1 is not taken while 2
// fits); FCC 64^3: 96.7 at 8, 79.1 at 4, 76.1 at 2; honeycomb 1024^2, M = 512: 243 at 8, 216
// at 4 and 2; square 512^2 with a flux, R = 12: 48.3 at 6, 42.2 at 4.  Double-float and FP64
// recursions, both alike so that their GEMMs sum in the same order, take powers of two only (the
// kernels of other widths cost them more than they save: honeycomb 305x310, M = 301, R = 16,
// double-float, 42.5 ms at 6).  The FP64 GEMM of the reference form wants long K: wide chunks (Lieb
// 276x274, M = 60, R = 16: 143 ms at 4, 122 at 16).  both: a power of two (the widths of the one
// recursion that carries both sides).
int pick_chunk(int R, bool both, int prec, bool f64b, int32_t M, int64_t n_pad, double sel, double budget) {
  const double per_vector = 2.0 * M * n_pad * sel;
  if (both) {
    int c = 1;
    while (c < R && c < 32) c <<= 1;
    while (c > 1 && per_vector * c > budget) c >>= 1;
    return c;
  }
  constexpr double kStepMs = 4.5e-3, kRowMs = 0.8e-9, kL2Ms = 4e-9, kHbmMs = 8e-9, kGemmMs = 8e-12, kMapMs = 0.45e-9;
  int best = 1;
  double least = 0.0;
  for (int cap = 32; cap > 1; cap -= 2) {
    const int w = step_width(TBK_PREC_MIXED, R, cap), chunks = (R + w - 1) / w;
    const double bytes = per_vector * w, pooled = bytes + 8.0 * 16.0 * n_pad * w;
    if (bytes > budget || (prec != TBK_PREC_MIXED && (w & (w - 1)))) continue;
    const double value = (!f64b && 16.0 * n_pad * w <= 20e6 ? kL2Ms : kHbmMs) + M * kGemmMs;
    const double ms = chunks * 2.0 * M * (kStepMs + n_pad * (kRowMs + w * value)) +
                      (pooled > (double)kKuboPoolKeep ? kMapMs * bytes : 0.0);
    if (best > 1 && ms >= least) continue;
    best = w;
    least = ms;
  }
  return best;
}

}  // namespace
}  // namespace tbk

using namespace tbk;

extern "C" {

int tbk_kubo_mu(tbk_sparse Ht, tbk_sparse AL, tbk_sparse BL, tbk_sparse AR, tbk_sparse BR, int32_t M, int32_t R,
                uint64_t seed, const double* kets, int32_t kernel_kind, double kp0, double kp1, int32_t flags,
                double block_budget_gb, double* mu_out, void* stream) {
  if (!Ht || !mu_out) return fail(TBK_ERR_INVALID, "tbk_kubo_mu: null argument");
  if (M < 1 || R < 1) return fail(TBK_ERR_INVALID, "tbk_kubo_mu: M and R must be >= 1");
  if (Ht->rows != Ht->cols) return fail(TBK_ERR_INVALID, "tbk_kubo_mu: H must be square");
  tbk_sparse ops[4] = {AL, BL, AR, BR};
  for (auto* o : ops)
    if (o && (o->rows != Ht->rows || o->cols != Ht->cols)) return fail(TBK_ERR_INVALID, "tbk_kubo_mu: operator size mismatch");
  cudaStream_t st = as_stream(stream);
  ScratchScope scope(st);
  PhaseTrace trace(st);
  // outside a server (which sets its own pool): stores and work blocks that
  // the pool keeps come from kubo_pool (decided below, once their size is known)
  AsyncAllocCtx kctx{};
  const int32_t n = Ht->rows;
  TBK_TRY(ensure_ell(Ht, st));
  for (auto* o : ops) if (o) TBK_TRY(ensure_ell(o, st));
  trace.mark("ell");
  const int64_t n_pad = (int64_t)Ht->ell.n_slices * 32;
  // default budget: 60% of the free device memory
  double budget = block_budget_gb * 1e9;
  if (block_budget_gb <= 0) {
    size_t fr = 0, tot = 0;
    TBK_CUDA(cudaMemGetInfo(&fr, &tot));
    budget = 0.6 * (double)fr;
  }
  const bool f64b = (flags & TBK_MU_FP64_BLOCKS) != 0;   // FP64 reference form: complex128 blocks, FP64 GEMM
  const double sel = f64b ? 16.0 : 8.0;                   // bytes per stored element
  const int prec = (flags & TBK_MU_MIXED_RECURSION) ? TBK_PREC_MIXED
                   : (flags & TBK_MU_DD_RECURSION)  ? TBK_PREC_DD
                                                    : TBK_PREC_FP64;
  // chunk of random vectors: both stored sides within the budget
  const int Rc = pick_chunk(R, (flags & TBK_MU_BOTH_SIDES) != 0, prec, f64b, M, n_pad, sel, budget);
  if (2.0 * M * n_pad * Rc * sel > budget)
    return fail(TBK_ERR_BUDGET, "stored Chebyshev blocks need %.1f GB > budget %.1f GB", 2.0 * M * n_pad * sel / 1e9,
                budget / 1e9);
  const int64_t blk = n_pad * Rc;                       // complex entries per block
  // stored blocks: complex64 or FP16 pairs.  Recursion and operator applications:
  // complex128 work blocks by default (the Chebyshev recursion accumulates rounding
  // error near the band edges, where the Kubo weights 1/(1-e^2)^2 are largest; each
  // stored value is rounded to complex64 exactly once); TBK_MU_MIXED_RECURSION
  // runs them in complex64 with FP32 H~ (HBM-bound instead of FP64-pipe-bound).
  const size_t csz = prec == TBK_PREC_MIXED ? sizeof(float2) : sizeof(double2);
  DevBuf Ls, Rs, work, partd, part, macc, gdev, kstage;
  bool use_tc = !f64b && (flags & TBK_MU_TENSOR) != 0;   // FP16-pair stores and the tensor-core GEMM
  const int64_t blk16 = (blk + 31) / 32 * 32;           // K padded to whole tiles of either store (zeros)
  if ((!tl_async_alloc || tl_async_alloc->scratch) && 2.0 * sel * blk16 * M + 8.0 * csz * blk <= (double)kKuboPoolKeep) {
    kctx.pool = kubo_pool();
    kctx.stream = st;
  }
  {
    const AsyncAllocCtx* outer = tl_async_alloc;
    if (kctx.pool) tl_async_alloc = &kctx;
    const int a = Ls.alloc((size_t)sel * blk16 * M), b = a == TBK_OK ? Rs.alloc((size_t)sel * blk16 * M) : a;
    tl_async_alloc = outer;
    TBK_TRY(b);
  }
  // both sides as one recursion of width 2 Rc (TBK_MU_BOTH_SIDES) when every
  // output operator can be fused into the step (the gathers move twice the
  // bytes per row; the stored values are the same bits)
  bool both = !f64b && (flags & TBK_MU_BOTH_SIDES) && (flags & TBK_MU_FUSED_OPS) &&
              2 * Rc <= (prec == TBK_PREC_MIXED ? 64 : 32) && (prec != TBK_PREC_MIXED || Rc >= 2);
  for (tbk_sparse_s* o : {AL, AR}) {
    if (!both || !o) continue;
    bool same = false;
    TBK_TRY(same_ell_structure(Ht, o, &same, st));
    both = same;
  }
  // small blocks: the two sides' recursions run side by side on two streams
  const int64_t steps = (int64_t)M * ((R + Rc - 1) / Rc);   // of one side
  const bool dual = !both && !f64b && (double)csz * blk <= kDualBlock && steps >= kDualSteps;
  {
    const AsyncAllocCtx* outer = tl_async_alloc;
    if (kctx.pool) tl_async_alloc = &kctx;
    const int a = work.alloc(csz * blk * (both ? 8 : dual ? 7 : 4));
    tl_async_alloc = outer;
    TBK_TRY(a);
  }
  // the stores write every k < n Rc of every block; the entries of padded
  // rows (n <= row < n_pad) and of the K tail up to whole tiles must read as
  // zero.  In the K-tiled layouts (16 k a tile; FP16 pairs: 32) they all lie
  // in the K tiles from floor(n Rc / tile) on: one contiguous region (the
  // stores overwrite its written part afterwards)
  auto zero_tail = [&]() -> int {
    const int64_t kt = use_tc ? kSplitTile : 16, kt0 = (int64_t)n * Rc / kt, kt1 = (blk + kt - 1) / kt;
    const size_t tile = (size_t)sel * kt * M;           // bytes of one K tile of all M blocks
    if (kt1 > kt0) {
      TBK_CUDA(cudaMemsetAsync(Ls.as<char>() + kt0 * tile, 0, (size_t)(kt1 - kt0) * tile, st));
      TBK_CUDA(cudaMemsetAsync(Rs.as<char>() + kt0 * tile, 0, (size_t)(kt1 - kt0) * tile, st));
    }
    return TBK_OK;
  };
  TBK_TRY(zero_tail());
  SplitScales sc;
  if (use_tc) TBK_TRY(sc.alloc(st));
  for (int h = 0; h < 2 && use_tc; ++h)
    if (h ? AR : AL) TBK_TRY(sc.set_operator(h, (h ? AR : AL)->ell, st));
  TBK_CUDA(cudaMemsetAsync(work.p, 0, work.bytes, st));
  TBK_TRY(macc.alloc(sizeof(double2) * (size_t)M * M));
  TBK_CUDA(cudaMemsetAsync(macc.p, 0, macc.bytes, st));
  if (kets) {
    TBK_TRY(kstage.alloc(sizeof(double2) * (size_t)n * R));
    TBK_CUDA(cudaMemcpyAsync(kstage.p, kets, sizeof(double2) * (size_t)n * R, cudaMemcpyHostToDevice, st));
  }
  int grid = 1, grid_op = 1;                             // of the steps; with an operator product in the ELL form
  TBK_TRY(step_config(Ht, Rc, prec, &grid, st));
  TBK_TRY(step_config(Ht, Rc, prec, &grid_op, st, false));
  int gmax = std::max(grid, grid_op);
  for (auto* o : ops)
    if (o) { int g2; TBK_TRY(step_config(o, Rc, prec, &g2, st)); gmax = std::max(gmax, g2); }
  int grid2 = 1;
  if (both) {
    TBK_TRY(step_config(Ht, 2 * Rc, prec, &grid2, st, false));
    gmax = std::max(gmax, grid2);
    if (prec == TBK_PREC_DD)
      for (tbk_sparse_s* o : {AL, AR}) if (o) TBK_TRY(ensure_ell_dd(o, st));
  }
  TBK_TRY(partd.alloc(sizeof(double) * 2 * gmax));
  trace.mark("alloc+classes");
  char* wb = work.as<char>();
  auto wblk = [&](int i) { return static_cast<void*>(wb + (size_t)i * blk * csz); };
  void* v0 = wblk(3);
  // algorithmic DRAM bytes of the block phase: vector blocks read / written,
  // matrix (ELL columns + values + diagonal) per pass, complex64 stores
  double rec_bytes = 0.0;
  const double vecb = (double)blk * csz, stb = (double)blk * 8.0;
  const int vsz = prec == TBK_PREC_MIXED ? 4 : 8;
  // class form (row classes): the row's class byte and diagonal; the table is in shared memory
  auto ell_bytes = [&](tbk_sparse_s* A, bool cols) {
    const double hv = (double)vsz * (A->ell.cplx ? 2 : 1);
    if (cols && (A->ell.cls_state == 1 || (prec == TBK_PREC_MIXED && A->ell.cls32_state == 1))) return (double)A->rows * (1.0 + hv);
    return (double)A->ell.n_entries * ((cols ? 4.0 : 0.0) + hv) + (double)A->rows * hv;
  };
  // Complex64 recursions take the operator's products inside the step wherever H~ and the
  // operator have joint row classes: one pass over the vectors' neighbours per block
  // instead of two (FCC 128^3, 4 vectors: 77.9 us against 56.5 + 83.7); and where H~ runs in
  // the ELL form anyway, whose columns they then load once (a flux).  Comparing the matrices and
  // finding the classes costs some 60 us an operator, a product of its own 3 us a step or more:
  // whole calls with and without, honeycomb 31x29, 3 vectors, M = 4: 365, 255 us; 24: 496, 455; 32:
  // 539, 535; 48: 636, 684; 100: 964, 1205.
  constexpr int64_t kFuseSteps = 32;
  struct Fused {
    bool on = false;
    ClassSet32 pair;
    int grid = 1;
  } fused[2];
  for (int h = 0; h < 2 && !both && !f64b; ++h) {
    tbk_sparse_s* Aout = h ? AR : AL;
    Fused& F = fused[h];
    F.grid = grid;
    const bool mixed = prec == TBK_PREC_MIXED;
    if (!Aout || !((flags & TBK_MU_FUSED_OPS) || (mixed && steps >= kFuseSteps))) continue;
    bool v_real = false;
    TBK_TRY(same_ell_structure(Ht, Aout, &F.on, st, mixed ? &v_real : nullptr));
    if (F.on && prec == TBK_PREC_DD) TBK_TRY(ensure_ell_dd(Aout, st));
    // (joint classes are at least H~'s: none where it has none)
    if (F.on && mixed && !v_real && steps >= kFuseSteps && has_row_classes(Ht, prec))
      TBK_TRY(pair_classes32(Ht, Aout, &F.pair, st));
    if (F.pair.n_cls > 0) {
      TBK_TRY(pair_config(Ht, Rc, F.pair, &F.grid));
    } else {
      F.on = F.on && ((flags & TBK_MU_FUSED_OPS) || !has_row_classes(Ht, prec));
      if (F.on) F.grid = grid_op;
    }
  }
  cudaStream_t q = st;                                   // the stream the side being issued runs on
  auto apply = [&](tbk_sparse_s* A, const void* x, void* y) -> int {   // y = A x
    rec_bytes += 2 * vecb + ell_bytes(A, true);
    int g;
    TBK_TRY(step_config(A, Rc, prec, &g, st));
    return step_any(A, Rc, prec, x, y, nullptr, true, partd.as<double>(), g, q, nullptr, true, nullptr, false);
  };
  const unsigned gblk = (unsigned)std::min<int64_t>((blk + 255) / 256, 65535);
  auto round_to = [&](const void* src, const KStore& ks, int32_t m) -> int {
    rec_bytes += vecb + stb;
    return with_block(prec, src, [&](auto p) {
      if (ks.split)
        split_block_kernel<<<gblk, 256, 0, q>>>(p, reinterpret_cast<__half*>(ks.store[0]), m, M, blk, ks.scale[0], ks.bad);
      else
        round_block_kernel<<<gblk, 256, 0, q>>>(p, ks.store[0], m, M, blk);
    });
  };
  auto find_scale = [&](const void* src, int h) -> int {   // of a side whose recursion starts from src
    return with_block(prec, src, [&](auto p) { sc.find(p, blk, sc.scale(h), h, (h ? AR : AL) != nullptr, q); });
  };
  // FP64 reference form: block m of the complex128 store from a work block
  auto store64 = [&](const void* src, void* store, int32_t m) -> int {
    rec_bytes += vecb + 2 * stb;
    const unsigned g = (unsigned)std::min<int64_t>((blk + 255) / 256, 65535);
    double2* d = static_cast<double2*>(store);
    if (prec == TBK_PREC_FP64) store_block64_kernel<double2><<<g, 256, 0, q>>>(static_cast<const double2*>(src), d, m, M, blk);
    else if (prec == TBK_PREC_DD) store_block64_kernel<dd2><<<g, 256, 0, q>>>(static_cast<const dd2*>(src), d, m, M, blk);
    else store_block64_kernel<float2><<<g, 256, 0, q>>>(static_cast<const float2*>(src), d, m, M, blk);
    TBK_CHECK_LAUNCH();
    return TBK_OK;
  };
  // vectors past L2: every pass starts where the one before it ended (FCC 128^3, 2 vectors:
  // 38.5 -> 37.5 us a step; honeycomb 1024^2, 4 vectors: 32.4 -> 30.6; inside L2 1% slower)
  const bool zigzag = 2.0 * csz * blk > 32e6;
  // block m of `store` = A x, written by the product itself (no work block)
  auto apply_to_store = [&](tbk_sparse_s* A, const void* x, void* scratch, KStore ks, int32_t m) -> int {
    rec_bytes += vecb + ell_bytes(A, true) + stb;
    int g;
    TBK_TRY(step_config(A, Rc, prec, &g, st));
    ks.km[0] = m;
    return step_any(A, Rc, prec, x, scratch, nullptr, true, partd.as<double>(), g, q, &ks, false, nullptr, true, nullptr,
                    zigzag && (m & 1) == 0);
  };
  // one side: store[m] = Aout T_m(H~) (Bin v0), m < M; each step writes its
  // complex64 block (Aout absent) or feeds the product that does
  // TBK_MU_FUSED_OPS: with an output operator that shares H~'s ELL structure
  // (a commutator [X, H~] does), step m also forms Aout T_{m-1} from the x it
  // gathers and writes block m-1: one pass over the matrix and the vectors per
  // block instead of two.  The stored values are the same bits either way.
  // steps m_begin <= m < m_end of side h on stream q; the side ends with step M
  auto side = [&](int h, int32_t m_begin, int32_t m_end) -> int {
    tbk_sparse_s* Aout = h ? AR : AL;
    tbk_sparse_s* Bin = h ? BR : BL;
    const int w0 = dual && h ? 4 : 0;                     // this side's work blocks
    void* r[2] = {wblk(w0), wblk(w0 + 1)};                // T_m over T_{m-2}: one block less in L2
    void* tmpA = wblk(w0 + 2);
    const Fused& F = fused[h];
    const bool fuse = F.on;
    KStore ks;
    ks.store[0] = (h ? Rs : Ls).as<float2>();
    ks.kM = M;
    ks.split = use_tc;
    ks.scale[0] = sc.scale(h);
    ks.bad = sc.bad();
    for (int32_t m = m_begin; m < m_end; ++m) {
      if (m == 0) {
        if (Bin) TBK_TRY(apply(Bin, v0, r[0]));
        else TBK_CUDA(cudaMemcpyAsync(r[0], v0, csz * blk, cudaMemcpyDeviceToDevice, q));
      }
      void* y = r[m & 1];
      const void* x = m >= 1 ? r[(m - 1) & 1] : nullptr;
      const void* pv = m >= 2 ? y : nullptr;
      if (f64b) {                                         // recursion, operator, complex128 store
        if (m == M) break;
        if (m >= 1) {
          rec_bytes += (m >= 2 ? 3 : 2) * vecb + ell_bytes(Ht, true);
          TBK_TRY(step_any(Ht, Rc, prec, x, y, pv, m == 1, partd.as<double>(), grid, q, nullptr, true, nullptr,
                           false));
        }
        if (Aout) TBK_TRY(apply(Aout, y, tmpA));
        TBK_TRY(store64(Aout ? tmpA : y, ks.store[0], m));
      } else if (m == 0) {
        if (use_tc) TBK_TRY(find_scale(y, h));
        if (!Aout) TBK_TRY(round_to(y, ks, 0));
        else if (!fuse) TBK_TRY(apply_to_store(Aout, y, tmpA, ks, 0));
      } else if (m < M) {
        rec_bytes += (m >= 2 ? 3 : 2) * vecb + ell_bytes(Ht, true) + ((fuse || !Aout) ? stb : 0.0) +
                     (fuse ? ell_bytes(Aout, false) : 0.0);
        ks.km[0] = fuse ? m - 1 : m;
        TBK_TRY(step_any(Ht, Rc, prec, x, y, pv, m == 1, partd.as<double>(), F.grid, q,
                         fuse || !Aout ? &ks : nullptr, true, fuse ? Aout : nullptr, false,
                         F.pair.n_cls > 0 ? &F.pair : nullptr, zigzag && (m & 1)));
        if (Aout && !fuse) TBK_TRY(apply_to_store(Aout, y, tmpA, ks, m));
      } else if (fuse) {
        TBK_TRY(apply_to_store(Aout, x, tmpA, ks, M - 1));
      }
    }
    return TBK_OK;
  };
  // both sides at once: columns [0, Rc) carry the left side (BL v0), [Rc, 2 Rc)
  // the right side (BR v0); step m stores T_m of a side without an output
  // operator as block m and A T_{m-1} of a side with one as block m-1
  auto both_sides = [&]() -> int {
    const size_t b2 = csz * blk * 2;
    char* base = wb + csz * blk * 4;                     // two 2 Rc-wide blocks after the four Rc-wide ones
    void* r[2] = {base, base + b2};
    void* half[2] = {wblk(0), wblk(1)};
    tbk_sparse_s* Bin[2] = {BL, BR};
    tbk_sparse_s* Aout[2] = {AL, AR};
    float2* stores[2] = {Ls.as<float2>(), Rs.as<float2>()};
    KStore ks;
    ks.halves = 2;
    ks.kM = M;
    ks.split = use_tc;
    ks.bad = sc.bad();
    for (int h = 0; h < 2; ++h) {
      ks.store[h] = stores[h];
      ks.usev[h] = Aout[h] ? 1 : 0;
      ks.vval[h] = Aout[h] ? ell_vals(Aout[h]->ell, prec) : nullptr;
      ks.vdiag[h] = Aout[h] ? ell_diag(Aout[h]->ell, prec) : nullptr;
      ks.scale[h] = sc.scale(h);
    }
    for (int h = 0; h < 2; ++h) {
      if (Bin[h]) TBK_TRY(apply(Bin[h], v0, half[h]));
      else TBK_CUDA(cudaMemcpyAsync(half[h], v0, csz * blk, cudaMemcpyDeviceToDevice, st));
      if (use_tc) TBK_TRY(find_scale(half[h], h));
      TBK_TRY(with_block(prec, half[h], [&](auto p) {
        using CT = std::remove_const_t<std::remove_pointer_t<decltype(p)>>;
        pack_cols_kernel<CT><<<gblk, 256, 0, st>>>(n_pad, Rc, h * Rc, p, static_cast<CT*>(r[0]));
      }));
      if (!Aout[h])
        TBK_TRY(with_block(prec, r[0], [&](auto p) {
          if (use_tc)
            split_cols_kernel<<<gblk, 256, 0, st>>>(n_pad, Rc, h * Rc, p, reinterpret_cast<__half*>(stores[h]), 0, M,
                                                    ks.scale[h], ks.bad);
          else
            round_cols_kernel<<<gblk, 256, 0, st>>>(n_pad, Rc, h * Rc, p, stores[h], 0, M);
        }));
    }
    rec_bytes += 2 * (vecb + 2 * vecb);                  // start halves packed into the wide block
    for (int h = 0; h < 2; ++h) rec_bytes += Aout[h] ? 0.0 : 2 * vecb + stb;
    for (int32_t m = 1; m < M; ++m) {
      rec_bytes += 2 * (m >= 2 ? 3 : 2) * vecb + ell_bytes(Ht, true) + 2 * stb;
      for (int h = 0; h < 2; ++h) rec_bytes += Aout[h] ? ell_bytes(Aout[h], false) : 0.0;
      for (int h = 0; h < 2; ++h) ks.km[h] = Aout[h] ? m - 1 : m;
      TBK_TRY(step_ks(Ht, 2 * Rc, prec, r[(m - 1) & 1], r[m & 1], m >= 2 ? r[m & 1] : nullptr, m == 1,
                      partd.as<double>(), grid2, st, ks));
    }
    if (AL || AR) {                                      // A T_{M-1} -> block M-1 (the new vector is not kept)
      for (int h = 0; h < 2; ++h) ks.km[h] = Aout[h] ? M - 1 : -1;
      TBK_TRY(step_ks(Ht, 2 * Rc, prec, r[(M - 1) & 1], r[M & 1], M >= 2 ? r[M & 1] : nullptr, M == 1,
                      partd.as<double>(), grid2, st, ks));
    }
    return TBK_OK;
  };
  // split-K of the FP64 form: at least 16,384 K values per CTA, at most 64 partial M x M blocks
  const int64_t ksplit = std::max<int64_t>(16384, (blk + 63) / 64);
  const int32_t nsplit = (int32_t)((blk + ksplit - 1) / ksplit);
  if (f64b) TBK_TRY(part.alloc(sizeof(double2) * (size_t)nsplit * M * M));
  SecondStream second;
  if (dual) TBK_TRY(second.create(st));
  cudaEvent_t ev[3];
  for (auto& e : ev) TBK_CUDA(cudaEventCreate(&e));
  KuboTiming tm;
  for (int32_t r0 = 0; r0 < R; r0 += Rc) {
    TBK_CUDA(cudaEventRecord(ev[0], st));
    if (kets) TBK_TRY(load_block_any(prec, n, R, r0, Rc, kstage.as<double2>(), v0, st));
    else TBK_TRY(random_block_any(prec, n, R, r0, Rc, seed, v0, st));
    auto blocks = [&]() -> int {
      if (both) return both_sides();
      if (!dual) {
        TBK_TRY(side(0, 0, M + 1));
        return side(1, 0, M + 1);
      }
      TBK_CUDA(cudaEventRecord(second.fork, st));
      TBK_CUDA(cudaStreamWaitEvent(second.st, second.fork, 0));
      for (int32_t m = 0; m <= M; ++m) {                 // issued in turn, so that neither side waits for the host
        q = second.st;
        const int s1 = side(1, m, m + 1);
        q = st;
        TBK_TRY(s1);
        TBK_TRY(side(0, m, m + 1));
      }
      TBK_CUDA(cudaEventRecord(second.join, second.st));
      TBK_CUDA(cudaStreamWaitEvent(st, second.join, 0));
      return TBK_OK;
    };
    TBK_TRY(blocks());
    TBK_CUDA(cudaEventRecord(ev[1], st));
    trace.mark("blocks");
    if (f64b) {
      dim3 g((M + kGT - 1) / kGT, (M + kGT - 1) / kGT, nsplit);
      mu_gemm_f64_kernel<<<g, 256, 0, st>>>(Ls.as<double2>(), Rs.as<double2>(), M, blk, ksplit, part.as<double2>());
      TBK_CHECK_LAUNCH();
      mu_split_reduce_kernel<<<(unsigned)(((int64_t)M * M + 255) / 256), 256, 0, st>>>(part.as<double2>(), M, nsplit,
                                                                                       macc.as<double2>());
      TBK_CHECK_LAUNCH();
    }
    if (use_tc) {
      const SplitStore L{Ls.as<__half>(), sc.scale(0), 0, sc.bad()}, R_{Rs.as<__half>(), sc.scale(1), 0, sc.bad()};
      bool usable = false;
      TBK_TRY(mu_gemm_tc(L, R_, M, blk, macc.as<double>(), &usable, st));
      if (!usable) {                                     // values past FP16's range: complex64 stores from here on
        use_tc = false;
        float ms = 0.f;                                  // the blocks count twice, the GEMM so far not
        TBK_CUDA(cudaEventElapsedTime(&ms, ev[0], ev[1]));
        tm.ms_blocks += ms;
        TBK_CUDA(cudaEventRecord(ev[0], st));
        TBK_TRY(zero_tail());
        TBK_TRY(blocks());
        TBK_CUDA(cudaEventRecord(ev[1], st));
      }
    }
    if (!use_tc && !f64b)
      TBK_TRY(mu_gemm_cc(Ls.as<float2>(), Rs.as<float2>(), M, blk, &part, macc.as<double2>(), st));
    TBK_CUDA(cudaEventRecord(ev[2], st));
    TBK_CUDA(cudaEventSynchronize(ev[2]));
    trace.mark("gemm");
    float a = 0.f, b = 0.f;
    TBK_CUDA(cudaEventElapsedTime(&a, ev[0], ev[1]));
    TBK_CUDA(cudaEventElapsedTime(&b, ev[1], ev[2]));
    tm.ms_blocks += a;
    tm.ms_gemm += b;
    tm.gemm_flops += 8.0 * M * (double)M * (double)blk * (use_tc ? 3.0 : 1.0);   // real flops of the products issued
    tm.block_bytes += rec_bytes;
    rec_bytes = 0.0;
    tm.chunks += 1;
  }
  for (auto& e : ev) cudaEventDestroy(e);
  {
    std::lock_guard<std::mutex> lk(g_kubo_timing_mu);
    g_kubo_timing = tm;
  }
  // kernel factors g_m g_n (FP64)
  std::vector<double> g(M);
  TBK_TRY(tbk_kernel_seq(kernel_kind, M, kp0, kp1, g.data()));
  TBK_TRY(gdev.alloc(sizeof(double) * M));
  TBK_CUDA(cudaMemcpyAsync(gdev.p, g.data(), sizeof(double) * M, cudaMemcpyHostToDevice, st));
  mu_kernel_scale_kernel<<<(unsigned)(((int64_t)M * M + 255) / 256), 256, 0, st>>>(macc.as<double2>(), gdev.as<double>(), M);
  TBK_CHECK_LAUNCH();
  TBK_CUDA(cudaMemcpyAsync(mu_out, macc.p, sizeof(double2) * (size_t)M * M, cudaMemcpyDeviceToHost, st));
  TBK_CUDA(cudaStreamSynchronize(st));
  trace.mark("scale+readback");
  Ls.release();
  Rs.release();
  work.release();
  if (kctx.pool) {
    TBK_CUDA(cudaStreamSynchronize(st));
    TBK_CUDA(cudaMemPoolTrimTo(kctx.pool, kKuboPoolKeep));   // keep at most kKuboPoolKeep bytes
  }
  trace.mark("free");
  return TBK_OK;
}

int tbk_mu_from_blocks(int32_t M, int64_t K, const double* L, const double* Rb, int32_t flags, double* mu_out,
                       void* stream) {
  if (M < 1 || K < 1 || !L || !Rb || !mu_out) return fail(TBK_ERR_INVALID, "tbk_mu_from_blocks: bad argument");
  cudaStream_t st = as_stream(stream);
  ScratchScope scope(st);
  const bool tensor = (flags & TBK_MU_TENSOR) != 0;
  const int64_t K16 = (K + 31) / 32 * 32;                // whole tiles of either store
  // blocks go up several at a time: a copy and three launches for each of them took 29 us a
  // block (392 blocks of 7 values: 12.7 ms -> 0.3 ms)
  constexpr int64_t kStageBytes = 32 << 20;
  const int32_t per = (int32_t)std::max<int64_t>(1, std::min<int64_t>({M, kStageBytes / (16 * K), 65535}));
  // CTAs of a block: enough together to fill the GPU, partials for all
  const int gs = (int)std::max<int64_t>(1, std::min<int64_t>((K + kStatThreads - 1) / kStatThreads,
                                                             (2 * sm_count() + per - 1) / per));
  // zeroed: both stores, the sums, the scale search's mark and counters; not zeroed: its partials, the
  // scales, the stage
  const size_t store = sizeof(float2) * M * K16, sums = sizeof(double2) * (size_t)M * M;
  const size_t stat = sizeof(double) * 2 * gs * (size_t)per, scal = (sizeof(float) * 2 * M + 15) / 16 * 16;
  DevBuf zero, work, part;
  TBK_TRY(zero.alloc(2 * store + sums + sizeof(int) * ((size_t)per + 1)));
  TBK_TRY(work.alloc(stat + scal + sizeof(double2) * K * per));
  TBK_CUDA(cudaMemsetAsync(zero.p, 0, zero.bytes, st));
  void* Ld = zero.p;
  void* Rd = zero.as<char>() + store;
  double2* acc = reinterpret_cast<double2*>(zero.as<char>() + 2 * store);
  int* bad = reinterpret_cast<int*>(acc + (size_t)M * M);
  unsigned int* count = reinterpret_cast<unsigned int*>(bad + 1);
  float* scales = reinterpret_cast<float*>(work.as<char>() + stat);   // one for every block
  double2* stage = reinterpret_cast<double2*>(work.as<char>() + stat + scal);
  const unsigned gk = (unsigned)std::min<int64_t>((K + 255) / 256, std::max<int64_t>(1, 4096 / per));
  auto upload = [&](bool split) -> int {
    for (int side = 0; side < 2; ++side) {
      void* dst = side ? Rd : Ld;
      const double* src = side ? Rb : L;
      for (int32_t m = 0; m < M; m += per) {
        const int32_t nb = std::min(per, M - m);
        const double2* from = stage;
        TBK_CUDA(cudaMemcpyAsync(stage, src + 2 * (int64_t)m * K, sizeof(double2) * K * nb, cudaMemcpyHostToDevice, st));
        if (split) {
          float* s = scales + side * M + m;
          split_scale_kernel<<<dim3(gs, nb), kStatThreads, 0, st>>>(from, K, work.as<double>(), count, nullptr, s, bad);
          TBK_CHECK_LAUNCH();
          split_block_kernel<<<dim3(gk, nb), 256, 0, st>>>(from, static_cast<__half*>(dst), m, M, K, s, bad);
        } else {
          round_block_kernel<<<dim3(gk, nb), 256, 0, st>>>(from, static_cast<float2*>(dst), m, M, K);
        }
        TBK_CHECK_LAUNCH();
      }
    }
    return TBK_OK;
  };
  TBK_TRY(upload(tensor));
  cudaEvent_t ev[2];
  for (auto& e : ev) TBK_CUDA(cudaEventCreate(&e));
  TBK_CUDA(cudaEventRecord(ev[0], st));
  bool formed = false;
  if (tensor) {
    const SplitStore ls{static_cast<__half*>(Ld), scales, 1, bad};
    const SplitStore rs{static_cast<__half*>(Rd), scales + M, 1, bad};
    TBK_TRY(mu_gemm_tc(ls, rs, M, K, reinterpret_cast<double*>(acc), &formed, st));
    if (!formed) {                                       // infinities or NaN: complex64 blocks
      TBK_CUDA(cudaMemsetAsync(Ld, 0, 2 * store, st));
      TBK_TRY(upload(false));
      TBK_CUDA(cudaEventRecord(ev[0], st));
    }
  }
  if (!formed) TBK_TRY(mu_gemm_cc(static_cast<float2*>(Ld), static_cast<float2*>(Rd), M, K, &part, acc, st));
  TBK_CUDA(cudaEventRecord(ev[1], st));
  TBK_CUDA(cudaMemcpyAsync(mu_out, acc, sizeof(double2) * (size_t)M * M, cudaMemcpyDeviceToHost, st));
  TBK_CUDA(cudaStreamSynchronize(st));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, ev[0], ev[1]);
  for (auto& e : ev) cudaEventDestroy(e);
  KuboTiming tm;
  tm.ms_gemm = ms;
  tm.gemm_flops = 8.0 * M * (double)M * (double)K * (formed ? 3.0 : 1.0);
  tm.block_bytes = 2.0 * M * (double)K * 8.0;
  tm.chunks = 1;
  {
    std::lock_guard<std::mutex> lk(g_kubo_timing_mu);
    g_kubo_timing = tm;
  }
  return TBK_OK;
}

int tbk_kubo_release(void) {
  scratch_trim();
  cudaMemPool_t pl = kubo_pool();
  if (!pl) return TBK_OK;
  TBK_CUDA(cudaDeviceSynchronize());
  TBK_CUDA(cudaMemPoolTrimTo(pl, 0));
  return TBK_OK;
}

int tbk_kubo_last_timing(double* ms_blocks, double* ms_gemm, double* gemm_flops, double* block_bytes, int32_t* chunks) {
  KuboTiming t;
  {
    std::lock_guard<std::mutex> lk(g_kubo_timing_mu);
    t = g_kubo_timing;
  }
  if (ms_blocks) *ms_blocks = t.ms_blocks;
  if (ms_gemm) *ms_gemm = t.ms_gemm;
  if (gemm_flops) *gemm_flops = t.gemm_flops;
  if (block_bytes) *block_bytes = t.block_bytes;
  if (chunks) *chunks = t.chunks;
  return TBK_OK;
}

int tbk_kubo_bastin_zeta(int32_t M, const double* mu, int32_t n_eps, const double* eps, double vol, double* zeta_out,
                         void* stream) {
  if (M < 1 || !mu || n_eps < 0 || (n_eps && (!eps || !zeta_out))) return fail(TBK_ERR_INVALID, "tbk_kubo_bastin_zeta: bad argument");
  if (n_eps == 0) return TBK_OK;
  return moment_series<true>(M, mu, n_eps, eps, vol, zeta_out, as_stream(stream));
}

int tbk_kubo_greenwood_sigma(int32_t M, const double* mu, int32_t n_eps, const double* eps, double R,
                             double* sigma_out, void* stream) {
  if (M < 1 || !mu || n_eps < 0 || (n_eps && (!eps || !sigma_out)) || !(R > 0))
    return fail(TBK_ERR_INVALID, "tbk_kubo_greenwood_sigma: bad argument");
  if (n_eps == 0) return TBK_OK;
  return moment_series<false>(M, mu, n_eps, eps, R, sigma_out, as_stream(stream));
}

// Bastin: drop N/24 nodes at each end, ascending order, cumulative trapezoid from
// E = 0 outward with the half-cell weights of TB/snippets.h:421-449 (host, O(N)).
int tbk_kubo_bastin_integrate(int32_t N, const double* eps, const double* zeta, double* E_out, double* re_out,
                              double* im_out, int32_t* n_out) {
  if (N < 4 || !eps || !zeta || !E_out || !re_out || !im_out || !n_out)
    return fail(TBK_ERR_INVALID, "tbk_kubo_bastin_integrate: bad argument");
  const int32_t cut = N / 24;
  const int32_t n = N - 2 * cut;
  std::vector<double> E(n), zr(n), zi(n);
  for (int32_t k = 0; k < n; ++k) {     // drop(cut) | take(N - 2 cut) | reverse
    const int32_t src = cut + (n - 1 - k);
    E[k] = eps[src];
    zr[k] = zeta[2 * src];
    zi[k] = zeta[2 * src + 1];
  }
  const int32_t e0 = (int32_t)(std::upper_bound(E.begin(), E.end(), 0.0) - E.begin());
  if (e0 < 1 || e0 >= n) return fail(TBK_ERR_INVALID, "bastin integration: E = 0 not inside the node range");
  std::vector<double> ri(n, 0.0), ii(n, 0.0);
  ri[e0] = (zr[e0] * 3 / 4 + zr[e0 - 1] / 4) * (E[e0] - E[e0 - 1]) / 2;
  ri[e0 - 1] = -(zr[e0] / 4 + zr[e0 - 1] * 3 / 4) * (E[e0] - E[e0 - 1]) / 2;
  for (int32_t i = e0 + 1; i < n; ++i) {
    ri[i] = ri[i - 1] + (zr[i] + zr[i - 1]) / 2 * (E[i] - E[i - 1]);
    ii[i] = ii[i - 1] + (zi[i] + zi[i - 1]) / 2 * (E[i] - E[i - 1]);
  }
  for (int32_t i = e0 - 2; i >= 0; --i) {
    ri[i] = ri[i + 1] - (zr[i] + zr[i + 1]) / 2 * (E[i + 1] - E[i]);
    ii[i] = ii[i + 1] - (zi[i] + zi[i + 1]) / 2 * (E[i + 1] - E[i]);
  }
  for (int32_t k = 0; k < n; ++k) { E_out[k] = E[k]; re_out[k] = ri[k]; im_out[k] = ii[k]; }
  *n_out = n;
  return TBK_OK;
}

}  // extern "C"
