// split_store.cuh — Chebyshev blocks stored as FP16 pairs for the tensor-core GEMM.
//
// A stored complex64 value x of block m becomes s x = hi + lo with hi = half(s x) and
// lo = half(s x - hi): 22 significant bits, as the pair of TF32 numbers that kind::tf32
// products take.  Per K tile of 32 values and block, one 128-byte row holds the real
// parts (32 hi, 32 lo) and one the imaginary parts: value k of block m sits at halves
// k % 32 (hi) and 32 + k % 32 (lo) of row (k / 32 * 2 + part) * M + m.  8 bytes per value,
// as a complex64 store; a warp of the recursion writes whole 128-byte lines, and 128
// consecutive blocks of a part are a contiguous box for TMA.
// s is a power of two (exact).  FP16 spans 2^-24 .. 65504.  T_m of a matrix with spectrum
// in [-1, 1] does not grow in the root mean square, so s follows from the start vector x of
// the recursion and a bound g on what the output operator multiplies by: g times x's root mean
// square lies near 2^6 and g times its maximum at 2^13 at most.  Later values may grow by 2^10
// over the former (2^3 over the latter, where x is one spike), and values down to 2^-9 of it
// keep all 22 bits.  Values that do not fit (a recursion outside [-1, 1], infinities,
// NaN) set a flag, and the caller forms the chunk from complex64 stores instead.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace tbk {

constexpr int kSplitTile = 32;      // k per K tile

// One side's store.  scale[m * scale_stride]: s of block m.  bad: set when a value did
// not fit (shared by both sides).
struct SplitStore {
  __half* data = nullptr;
  const float* scale = nullptr;
  int32_t scale_stride = 0;
  int* bad = nullptr;
};

// (re, im) of value k into block m of M
__device__ __forceinline__ void split_put(__half* data, int32_t M, int32_t m, int64_t k, float re, float im, float s,
                                          int* bad) {
  const float a = re * s, b = im * s;
  if (!(fmaxf(fabsf(a), fabsf(b)) < 65504.f) || a != a || b != b) *bad = 1;
  const __half ah = __float2half_rn(a), bh = __float2half_rn(b);
  __half* p = data + (((k >> 5) * 2) * M + m) * 64 + (k & 31);
  const int64_t ip = (int64_t)M * 64;
  p[0] = ah;
  p[32] = __float2half_rn(a - __half2float(ah));
  p[ip] = bh;
  p[ip + 32] = __float2half_rn(b - __half2float(bh));
}
// values k, k + 1 (k even), 4-byte accesses
__device__ __forceinline__ void split_put2(__half* data, int32_t M, int32_t m, int64_t k, float re0, float im0,
                                           float re1, float im1, float s, int* bad) {
  const float a0 = re0 * s, b0 = im0 * s, a1 = re1 * s, b1 = im1 * s;
  const float big = fmaxf(fmaxf(fabsf(a0), fabsf(b0)), fmaxf(fabsf(a1), fabsf(b1)));
  const float sum = (a0 + b0) + (a1 + b1);               // NaN where any value is one
  if (!(big < 65504.f) || sum != sum) *bad = 1;
  const __half2 ah = __floats2half2_rn(a0, a1), bh = __floats2half2_rn(b0, b1);
  const float2 af = __half22float2(ah), bf = __half22float2(bh);
  __half2* p = reinterpret_cast<__half2*>(data + (((k >> 5) * 2) * M + m) * 64 + (k & 31));
  const int64_t im = (int64_t)M * 32;
  p[0] = ah;
  p[16] = __floats2half2_rn(a0 - af.x, a1 - af.y);
  p[im] = bh;
  p[im + 16] = __floats2half2_rn(b0 - bf.x, b1 - bf.y);
}

int mu_gemm_tc(const SplitStore& L, const SplitStore& Rb, int32_t M, int64_t K, double* mu_acc, bool* usable,
               cudaStream_t st);   // gemm_tc.cu: mu_acc += L^H R, *usable false (and nothing added) where bad is set

}  // namespace tbk
