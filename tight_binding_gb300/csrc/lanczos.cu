// lanczos.cu — spectral range of a Hermitian sparse matrix on the device.
//
// The reference estimates (E_min, E_max) for GreenFunction(N, HE, ref_HE,
// epsilon) with a Spectra Lanczos eigensolver on the CPU and refuses matrices
// above 5,000 rows (TB/numerical.h:24-46, TB/lattice.h:560-566).  Here: k steps
// of the Hermitian Lanczos three-term recursion on the device (complex128, one
// vector, scalars kept on the device and read back once), then the extreme
// eigenvalues of the k x k tridiagonal matrix by Sturm-sequence bisection on the
// host.  The residual norm beta_{k+1} |s_k| of each extreme
// Ritz pair is returned with it: an eigenvalue of the matrix lies within that
// distance of the Ritz value.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "host_model.h"
#include "kpm_device.cuh"
#include "kpm_step.cuh"
#include "tbk_internal.h"

namespace tbk {
namespace {

// The iteration keeps the vectors unnormalised, v_j = u_j / b_j with b_j = |u_j|,
// and every scalar on the device, so an iteration is two launches and no host
// round trip:
//   w       = H u_j                          partial sums of <u_j|w>
//   u_(j+1) = w / b_j - (alpha_j / b_j) u_j - (b_j / b_(j-1)) u_(j-1),
//             alpha_j = <u_j|w> / b_j^2      partial sums of |u_(j+1)|^2
// b_j has the size of H's entries, <u_j|w> that of their cube: entries far from 1 are brought
// near it by a power of two in the update's coefficients (lz_scale), which costs nothing per row.
// Each CTA of the update sums both sets of partials itself (fixed order, the same
// value in every CTA).  GB300 starts one FP64 warp instruction every 64 clocks on
// each quarter of an SM, so the kernels count FP64 instructions: 10 and 6 FMAs per
// row of a real H with 3 neighbours, two CTAs per SM so that the block sums stay
// few against the rows, and the scalars formed by one thread.
// 1,025,280-site honeycomb, 200 iterations: 21.9 ms with a 38 us product (the step
// kernel, with a norm it did not need), an 18 us update, a 6 us scaling and two host
// round trips (48 us) per iteration; 10.0 ms now (22 + 21 us).
constexpr int kLzThreads = 512;
constexpr int kLzWarps = kLzThreads / 32;

// Power of two for H from the upper word of its largest |entry|: 1 within 2^-200 .. 2^200
__host__ __device__ inline int lz_scale_exponent(uint32_t top) {
  const int e = (int)(top >> 20) - 1023;
  if (top == 0u || e == 1024 || (e >= -200 && e <= 200)) return 0;    // zero matrix; infinities, NaN
  return e < 0 ? (e < -1000 ? 1000 : -e) : -e < -1000 ? -1000 : -e;
}
__global__ void __launch_bounds__(kLzThreads) lanczos_max_kernel(const double* __restrict__ v, int64_t n,
                                                                 uint32_t* __restrict__ top) {
  __shared__ uint32_t sh;
  if (threadIdx.x == 0) sh = 0;
  __syncthreads();
  uint32_t m = 0;
  for (int64_t i = (int64_t)blockIdx.x * kLzThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kLzThreads)
    m = max(m, (uint32_t)__double2hiint(v[i]) & 0x7fffffffu);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(&sh, m);
  __syncthreads();
  if (threadIdx.x == 0) atomicMax(top, sh);
}

__device__ __forceinline__ double lz_warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// sum over the CTA, valid in thread 0
__device__ __forceinline__ double lz_block_sum(double v, double* sh) {
  v = lz_warp_sum(v);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x >= 32) return 0.0;
  return lz_warp_sum(threadIdx.x < kLzWarps ? sh[threadIdx.x] : 0.0);
}
// fixed-order sum of k partials by one warp
__device__ __forceinline__ double lz_partials(const double* __restrict__ p, int32_t k) {
  double a = 0.0, b = 0.0;
  for (int32_t q = threadIdx.x & 31; q < k; q += 64) {
    a += p[q];
    if (q + 32 < k) b += p[q + 32];
  }
  return lz_warp_sum(a + b);
}

// w = H u, part[block] = partial of Re <u|w>; one row per thread.  CLS: neighbours and
// values from the class table (in shared memory), else from the sliced ELL.
template <bool CPLX_H, bool CLS>
__global__ void __launch_bounds__(kLzThreads) lanczos_product_kernel(
    int32_t n, const int32_t* __restrict__ soff, const int32_t* __restrict__ ecol, const double* __restrict__ eval,
    const double* __restrict__ diag, const ClassTab ct, const double2* __restrict__ u, double2* __restrict__ w,
    double* __restrict__ part) {
  using HV = HVal<double, CPLX_H>;
  extern __shared__ __align__(16) unsigned char lz_smem[];
  __shared__ double sh[kLzWarps];
  const double* s_val = reinterpret_cast<const double*>(lz_smem);
  const int32_t* s_off = nullptr;
  const int32_t* s_cnt = nullptr;
  if constexpr (CLS) {
    const int32_t ne = ct.n_cls * ct.w, vw = ne * (CPLX_H ? 4 : 2);
    uint32_t* sw = reinterpret_cast<uint32_t*>(lz_smem);
    const uint32_t* gv = static_cast<const uint32_t*>(ct.val);
    for (int32_t q = threadIdx.x; q < vw; q += kLzThreads) sw[q] = gv[q];
    for (int32_t q = threadIdx.x; q < ne; q += kLzThreads) sw[vw + q] = (uint32_t)ct.off[q];
    for (int32_t q = threadIdx.x; q < ct.n_cls; q += kLzThreads) sw[vw + ne + q] = (uint32_t)ct.cnt[q];
    s_off = reinterpret_cast<const int32_t*>(sw + vw);
    s_cnt = reinterpret_cast<const int32_t*>(sw + vw + ne);
    __syncthreads();
  }
  double dot = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * kLzThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kLzThreads) {
    const int32_t r = (int32_t)i;
    const LaneV<double, 1> xs = ld_ro<double, 1>(u + r);
    LaneV<double, 1> acc;
    acc.re[0] = 0;
    acc.im[0] = 0;
    HV::load(diag, r).template fma<1>(xs, acc);
    if constexpr (CLS) {
      const int32_t c = __ldg(ct.cls + r), cnt = s_cnt[c], tb = c * ct.w;
      int32_t k = 0;
      for (; k + 4 <= cnt; k += 4) {
        LaneV<double, 1> xv[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) xv[q] = ld_ro<double, 1>(u + min(max(r + s_off[tb + k + q], 0), n - 1));
#pragma unroll
        for (int q = 0; q < 4; ++q) HV::load_smem(s_val, tb + k + q).template fma<1>(xv[q], acc);
      }
#pragma unroll 1
      for (; k < cnt; ++k)
        HV::load_smem(s_val, tb + k).template fma<1>(ld_ro<double, 1>(u + min(max(r + s_off[tb + k], 0), n - 1)), acc);
    } else {
      const int32_t s = r >> 5, o = soff[s], wd = (soff[s + 1] - o) >> 5;
      const int64_t b = (int64_t)o + (r & 31);
      int32_t k = 0;
      for (; k + 4 <= wd; k += 4) {
        LaneV<double, 1> xv[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) xv[q] = ld_ro<double, 1>(u + __ldg(ecol + b + (int64_t)(k + q) * 32));
#pragma unroll
        for (int q = 0; q < 4; ++q) HV::load(eval, b + (int64_t)(k + q) * 32).template fma<1>(xv[q], acc);
      }
#pragma unroll 1
      for (; k < wd; ++k)
        HV::load(eval, b + (int64_t)k * 32).template fma<1>(ld_ro<double, 1>(u + __ldg(ecol + b + (int64_t)k * 32)), acc);
    }
    dot = fma(xs.re[0], acc.re[0], dot);
    dot = fma(xs.im[0], acc.im[0], dot);
    st_v<double, 1>(w + r, acc);
  }
  const double a = lz_block_sum(dot, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = a;
}

// u_(j+1) over w; scal[2 j] = alpha_j, scal[2 j + 1] = b_j, of H times its power of two (top).
// pnorm: |u_j|^2 partials of the update before (j > 0).
__global__ void __launch_bounds__(kLzThreads) lanczos_update_kernel(
    int32_t n, int32_t j, double2* __restrict__ w, const double2* __restrict__ u, const double2* __restrict__ up,
    const double* __restrict__ pdot, const double* __restrict__ pnorm, double* __restrict__ onorm,
    double* __restrict__ scal, const uint32_t* __restrict__ top) {
  __shared__ double sh[kLzWarps], sdot, snorm, coef[3];
  const int warp = threadIdx.x >> 5;
  if (warp == 0) {
    const double a = lz_partials(pdot, (int32_t)gridDim.x);
    if (threadIdx.x == 0) sdot = a;
  } else if (warp == 1) {
    const double q = j > 0 ? lz_partials(pnorm, (int32_t)gridDim.x) : 1.0;   // |u_0| = 1
    if ((threadIdx.x & 31) == 0) snorm = q;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const double f = __hiloint2double((1023 + lz_scale_exponent(*top)) << 20, 0);
    const double b = sqrt(snorm), inv = 1.0 / b, alpha = sdot * f * inv * inv;
    coef[0] = inv * f;
    coef[1] = -alpha * inv;
    coef[2] = j > 0 ? -b / scal[2 * j - 1] : 0.0;
    if (blockIdx.x == 0) {
      scal[2 * j] = alpha;
      scal[2 * j + 1] = b;
    }
  }
  __syncthreads();
  const double cw = coef[0], cu = coef[1], cp = coef[2];
  double s = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * kLzThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kLzThreads) {
    const double2 x = w[i], v = u[i], p = up[i];
    double2 o;
    o.x = fma(cp, p.x, fma(cu, v.x, cw * x.x));
    o.y = fma(cp, p.y, fma(cu, v.y, cw * x.y));
    w[i] = o;
    s = fma(o.x, o.x, s);
    s = fma(o.y, o.y, s);
  }
  s = lz_block_sum(s, sh);
  if (threadIdx.x == 0) onorm[blockIdx.x] = s;
}

// b_k after the last update
__global__ void lanczos_norm_kernel(const double* __restrict__ pnorm, int32_t nb, double* __restrict__ out) {
  const double q = lz_partials(pnorm, nb);
  if (threadIdx.x == 0) *out = sqrt(q);
}

template <bool CPLX_H, bool CLS>
int lanczos_product(const EllDev& E, const ClassTab& ct, const double2* u, double2* w, double* part, int grid,
                    cudaStream_t st) {
  const size_t smem = CLS ? class_smem(E, TBK_PREC_FP64) : 0;
  lanczos_product_kernel<CPLX_H, CLS><<<grid, kLzThreads, smem, st>>>(
      E.n_rows, E.slice_off.as<int32_t>(), E.col.as<int32_t>(), E.val64.as<double>(), E.diag64.as<double>(), ct, u, w,
      part);
  TBK_CHECK_LAUNCH();
  return TBK_OK;
}

// number of eigenvalues of the tridiagonal (a, b) below x (Sturm sequence)
int sturm_count(const std::vector<double>& a, const std::vector<double>& b, double x) {
  int c = 0;
  double q = 1.0;
  for (size_t i = 0; i < a.size(); ++i) {
    const double bb = i ? b[i - 1] * b[i - 1] : 0.0;
    q = a[i] - x - (i ? bb / q : 0.0);
    if (q == 0.0) q = 1e-300;
    if (q < 0) ++c;
  }
  return c;
}
// the k-th smallest eigenvalue (0-based) by bisection inside [lo, hi]
double tridiag_eig(const std::vector<double>& a, const std::vector<double>& b, int k, double lo, double hi) {
  for (int it = 0; it < 200 && hi - lo > 1e-15 * std::max(1.0, std::fabs(lo) + std::fabs(hi)); ++it) {
    const double mid = 0.5 * (lo + hi);
    if (sturm_count(a, b, mid) > k) hi = mid;
    else lo = mid;
  }
  return 0.5 * (lo + hi);
}
// last component of the unit eigenvector of the tridiagonal for eigenvalue th
// (forward recurrence of the characteristic polynomials, then normalised)
double last_component(const std::vector<double>& a, const std::vector<double>& b, double th) {
  const size_t k = a.size();
  std::vector<double> x(k);
  x[0] = 1.0;
  if (k > 1) x[1] = (th - a[0]) / b[0];
  for (size_t i = 2; i < k; ++i) {
    x[i] = ((th - a[i - 1]) * x[i - 1] - b[i - 2] * x[i - 2]) / b[i - 1];
    if (std::fabs(x[i]) > 1e150)              // keep the recurrence finite
      for (size_t q = 0; q <= i; ++q) x[q] *= 1e-150;
  }
  double nrm = 0.0, mx = 0.0;
  for (double v : x) mx = std::max(mx, std::fabs(v));
  if (!(mx > 0.0) || !std::isfinite(mx)) return 1.0;
  for (double v : x) nrm += (v / mx) * (v / mx);
  return std::fabs(x[k - 1] / mx) / std::sqrt(nrm);
}

}  // namespace
}  // namespace tbk

using namespace tbk;

extern "C" {

int tbk_spectral_range(tbk_sparse A, int32_t iters, uint64_t seed, double* e_min, double* e_max, double* res_min,
                       double* res_max, void* stream) {
  if (!A || !e_min || !e_max) return fail(TBK_ERR_INVALID, "tbk_spectral_range: null argument");
  if (A->rows != A->cols) return fail(TBK_ERR_INVALID, "tbk_spectral_range: matrix must be square");
  if (iters < 2) return fail(TBK_ERR_INVALID, "tbk_spectral_range: iters must be >= 2");
  cudaStream_t st = as_stream(stream);
  ScratchScope scope(st);
  const int32_t n = A->rows;
  TBK_TRY(ensure_classes(A, st));
  const EllDev& E = A->ell;
  const ClassTab ct = class_tab(E, TBK_PREC_FP64);
  const bool cls = ct.n_cls > 0, cplx = E.cplx != 0;
  const int64_t n_pad = (int64_t)E.n_slices * 32;
  const int32_t k_max = std::min<int64_t>(iters, (int64_t)2 * n);
  DevBuf vb[3], part, upart, scal;
  for (auto& b : vb) {
    TBK_TRY(b.alloc(sizeof(double2) * n_pad));
    TBK_CUDA(cudaMemsetAsync(b.p, 0, b.bytes, st));
  }
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((n + kLzThreads - 1) / kLzThreads, 2 * sm_count()));
  TBK_TRY(part.alloc(sizeof(double) * grid));
  TBK_TRY(upart.alloc(sizeof(double) * 2 * grid));
  TBK_TRY(scal.alloc(sizeof(double) * (2 * (size_t)k_max + 2)));   // the largest entry, b_k, then the scalars
  uint32_t* top = scal.as<uint32_t>();
  double* ab = scal.as<double>() + 2;
  TBK_CUDA(cudaMemsetAsync(top, 0, sizeof(double), st));
  const int64_t words = A->nnz * (A->is_complex ? 2 : 1);
  lanczos_max_kernel<<<(int)std::max<int64_t>(1, std::min<int64_t>((words + kLzThreads - 1) / kLzThreads, 2 * sm_count())),
                       kLzThreads, 0, st>>>(A->values.as<double>(), words, top);
  TBK_CHECK_LAUNCH();
  double2* v = vb[0].as<double2>();      // u_j
  double2* vp = vb[1].as<double2>();     // u_(j-1)
  double2* w = vb[2].as<double2>();
  // u_0: the seeded random phases (unit norm)
  TBK_TRY(random_block_any(TBK_PREC_FP64, n, 1, 0, 1, seed, v, st));
  // the scalars of k iterations, without H's power of two
  std::vector<double> hs;
  auto read = [&](int32_t k) -> int {
    hs.resize(2 * (size_t)k + 2);
    TBK_CUDA(cudaMemcpyAsync(hs.data(), scal.p, sizeof(double) * hs.size(), cudaMemcpyDeviceToHost, st));
    TBK_CUDA(cudaStreamSynchronize(st));
    uint32_t h;
    std::memcpy(&h, hs.data(), sizeof(h));
    if (const int e = lz_scale_exponent(h))
      for (double& x : hs) x = std::ldexp(x, -e);
    return TBK_OK;
  };
  // A vanishing norm after iteration j: an invariant subspace, the scalars after it are not used
  auto ends = [&](int32_t j) { return !(hs[2 * j + 5] > 1e-13 * std::max(1.0, std::fabs(hs[2 * j + 2]))); };
  // Looked for after 4, 16, 64 ... iterations (a read-back of some 15 us each), so that a matrix
  // of few distinct eigenvalues does not run all of them
  int32_t k_run = 0;
  for (int32_t look = 4; k_run < k_max; ++k_run) {
    const int32_t j = k_run;
    if (j == look) {
      TBK_TRY(read(j));
      bool done = false;
      for (int32_t i = 0; i + 1 < j && !done; ++i) done = ends(i);
      if (done) break;
      look = look > INT32_MAX / 4 ? INT32_MAX : 4 * look;
    }
    TBK_TRY(cplx ? (cls ? lanczos_product<true, true>(E, ct, v, w, part.as<double>(), grid, st)
                        : lanczos_product<true, false>(E, ct, v, w, part.as<double>(), grid, st))
                 : (cls ? lanczos_product<false, true>(E, ct, v, w, part.as<double>(), grid, st)
                        : lanczos_product<false, false>(E, ct, v, w, part.as<double>(), grid, st)));
    double* in = upart.as<double>() + (j & 1) * grid;
    double* out = upart.as<double>() + ((j + 1) & 1) * grid;
    lanczos_update_kernel<<<grid, kLzThreads, 0, st>>>(n, j, w, v, vp, part.as<double>(), in, out, ab, top);
    TBK_CHECK_LAUNCH();
    double2* t = vp;
    vp = v;
    v = w;
    w = t;
  }
  lanczos_norm_kernel<<<1, 32, 0, st>>>(upart.as<double>() + (k_run & 1) * grid, grid, scal.as<double>() + 1);
  TBK_CHECK_LAUNCH();
  TBK_TRY(read(k_run));
  // T = tridiag(beta, alpha, beta)
  std::vector<double> alpha, beta;
  double bprev = 0.0;
  for (int32_t j = 0; j < k_run; ++j) {
    alpha.push_back(hs[2 * j + 2]);
    bprev = j + 1 < k_run ? hs[2 * j + 5] : hs[1];
    if (j + 1 == k_run || ends(j)) break;
    beta.push_back(bprev);
  }
  // extreme Ritz values of T_k (Gershgorin interval for the bisection)
  double lo = 1e300, hi = -1e300;
  for (size_t i = 0; i < alpha.size(); ++i) {
    const double r = (i ? std::fabs(beta[i - 1]) : 0.0) + (i < beta.size() ? std::fabs(beta[i]) : 0.0);
    lo = std::min(lo, alpha[i] - r);
    hi = std::max(hi, alpha[i] + r);
  }
  const int k = (int)alpha.size();
  std::vector<double> bb(beta.begin(), beta.begin() + std::max(0, k - 1));
  const double tmin = tridiag_eig(alpha, bb, 0, lo, hi);
  const double tmax = tridiag_eig(alpha, bb, k - 1, lo, hi);
  *e_min = tmin;
  *e_max = tmax;
  if (res_min) *res_min = bprev * last_component(alpha, bb, tmin);
  if (res_max) *res_max = bprev * last_component(alpha, bb, tmax);
  return TBK_OK;
}

}  // extern "C"
