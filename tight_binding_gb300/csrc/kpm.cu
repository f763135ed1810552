// kpm.cu — Chebyshev (KPM) moments on sm_103a.
//
// Replaces cuda::Cheb_first_kind_seq_braket (TB/numerics_cuda.cu:190-323): the
// reference runs one cuSPARSE SpMM (two for real H) plus one blocking cuBLAS dot
// per moment.  Here one fused kernel per recursion step
//     v_{n+1} = 2 H~ v_n - v_{n-1}      (v_1 = H~ v_0 on the first step)
// streams the block of R vectors once, gathers the neighbours' 128-bit vector
// slices through L1/L2, writes v_{n+1} over v_{n-1} in place, and folds the
// moment dot products into the same pass with warp-shuffle reductions.  Per-CTA
// FP64 partial sums go to a small buffer; one reduction at the end sums them in
// a fixed order (deterministic, no atomics).
//
// Vector blocks are site-major: the R vectors of one site are contiguous (256 B
// for R = 32 complex64), so every gathered neighbour is one coalesced row.
//
// Two precisions:
//   TBK_PREC_FP64 : complex128 vectors, FP64 H~ (the plain drop-in)
//   TBK_PREC_DD   : double-float vectors and H~ (hi + lo FP32 pairs, ~48 bits),
//                   FP32-pipe arithmetic, per-thread double-float sums
//   TBK_PREC_MIXED: complex64 vectors, FP32 H~, FP32 per-thread sums promoted
//                   to FP64 for every reduction above the thread.
// With bras == kets (DoS) the Chebyshev product rule gives two moments per step:
//   mu_2n = 2 <v_n|v_n> - mu_0,   mu_2n+1 = 2 <v_n+1|v_n> - mu_1.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cmath>
#include <mutex>
#include <vector>

#include "host_model.h"
#include "kpm_device.cuh"
#include "kpm_step.cuh"
#include "tbk_internal.h"

namespace tbk {

}  // namespace tbk
#include "kpm_tma.cuh"
#include "kpm_fused.cuh"
#include "kpm_small.cuh"
#include "kpm_persist.cuh"
namespace tbk {

// Column-major complex128 (Eigen) -> site-major work block of width Rp.
template <typename F>
__global__ void load_block_kernel(int32_t n, int32_t R, int32_t r0, int32_t rc, int32_t Rp,
                                  const double2* __restrict__ src, typename C2<F>::T* __restrict__ dst) {
  __shared__ double2 tile[32][33];
  const int32_t i0 = blockIdx.x * 32;
  const int32_t c0 = blockIdx.y * 32;
  // read: consecutive threads walk consecutive sites of one vector
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    int32_t c = c0 + k, i = i0 + threadIdx.x;
    double2 v = make_double2(0.0, 0.0);
    if (c < rc && i < n && r0 + c < R) v = src[(int64_t)(r0 + c) * n + i];
    tile[k][threadIdx.x] = v;
  }
  __syncthreads();
  // write: consecutive threads walk consecutive vectors of one site
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    int32_t i = i0 + k, c = c0 + threadIdx.x;
    if (i < n && c < Rp) {
      double2 v = tile[threadIdx.x][k];
      typename C2<F>::T o;
      o.x = (F)v.x; o.y = (F)v.y;
      dst[(int64_t)i * Rp + c] = o;
    }
  }
}

// Device random-phase kets exp(2 pi i u)/sqrt(N), u = u01(seed, r, i), site-major.  Bound
// by the FP64 pipe (the sincos): 1/sqrt(N) comes from the host, and indices of blocks
// below 2^32 values divide in 32 bits.  152,306 x 4: 51 -> 36 us.
template <typename F, typename I>
__global__ void random_block_kernel(int32_t n, int32_t R, int32_t r0, int32_t Rp, uint64_t seed, double inv,
                                    typename C2<F>::T* __restrict__ dst) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= (int64_t)n * Rp) return;
  const int32_t i = (int32_t)((I)g / (I)Rp), c = (int32_t)((I)g % (I)Rp);
  typename C2<F>::T o;
  if (r0 + c < R) {
    double th = 6.283185307179586476925286766559 * u01(seed, (uint64_t)(r0 + c), (uint64_t)i);
    double s, cs;
    sincos(th, &s, &cs);
    o.x = (F)(cs * inv); o.y = (F)(s * inv);
  } else {
    o.x = 0; o.y = 0;
  }
  dst[g] = o;
}
template <typename F>
static void random_block(int32_t n, int32_t R, int32_t r0, int32_t Rp, uint64_t seed, void* dst, cudaStream_t st) {
  const int64_t tot = (int64_t)n * Rp;
  const unsigned g = (unsigned)((tot + 255) / 256);
  const double inv = 1.0 / std::sqrt((double)n);
  auto d = static_cast<typename C2<F>::T*>(dst);
  if (tot < (1ll << 32)) random_block_kernel<F, uint32_t><<<g, 256, 0, st>>>(n, R, r0, Rp, seed, inv, d);
  else random_block_kernel<F, int64_t><<<g, 256, 0, st>>>(n, R, r0, Rp, seed, inv, d);
}

// Fixed-order sum of the per-CTA partials of every (chunk, step, slot).  mirror: CTA b ran tile b in odd
// steps too, where a step kernel's CTA b runs the last tile but b.
__global__ void reduce_partials_kernel(const double* __restrict__ part, int32_t n_chunks, int32_t n_steps,
                                       int32_t nblk, int mirror, double* __restrict__ sums) {
  const int32_t step = blockIdx.x, slot = blockIdx.y;
  double acc = 0.0;
  __shared__ double sh[256];
  for (int32_t ch = 0; ch < n_chunks; ++ch) {
    const double* p = part + (((int64_t)ch * n_steps + step) * 2 + slot) * nblk;
    double a = 0.0;
    for (int32_t b = threadIdx.x; b < nblk; b += blockDim.x) a += p[mirror && (step & 1) ? nblk - 1 - b : b];
    sh[threadIdx.x] = a;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
      if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
      __syncthreads();
    }
    if (threadIdx.x == 0) acc += sh[0];
    __syncthreads();
  }
  if (threadIdx.x == 0) sums[step * 2 + slot] = acc;
}

// Assemble mu_k (FP64) from the step sums.
__global__ void assemble_moments_kernel(const double* __restrict__ sums, int32_t n_mom, int32_t doubling,
                                        double* __restrict__ mu) {
  int32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n_mom) return;
  if (doubling) {
    // step s holds <v_s|v_s> (slot 0) and <v_s|v_{s-1}> (slot 1); step 0 holds mu_0, mu_1
    const double mu0 = sums[0], mu1 = sums[1];
    if (k == 0) mu[k] = mu0;
    else if (k == 1) mu[k] = mu1;
    else if (k & 1) mu[k] = 2.0 * sums[2 * ((k + 1) >> 1) + 1] - mu1;   // mu_2s-1, s = (k+1)/2
    else mu[k] = 2.0 * sums[2 * (k >> 1)] - mu0;                         // mu_2s,   s = k/2
  } else {
    // step 0 holds <b|v1> in slot 0 and <b|v0> in slot 1; step s>0 holds <b|v_{s+1}>
    if (k == 0) mu[k] = sums[1];
    else mu[k] = sums[2 * (k - 1)];
  }
}


constexpr int kTmaStages = 4;
// polls of the staged kernel's ring waits and the cooperative recursion's meetings before they
// give up (tbk_set_wait_limit)
std::atomic<uint32_t> g_wait_limit{kWaitLimit};

template <typename F, int R, bool CPLX_H, bool BRAKET>
static int tma_kernel_setup(int smem, int* occ) {
  auto kern = kpm_tma_step_kernel<F, R, CPLX_H, BRAKET, kTmaStages>;
  TBK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  int nb = 0;
  TBK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, kTmaThreads, smem));
  *occ = nb;
  return TBK_OK;
}

template <typename F, int R, bool CPLX_H>
static int launch_tma_r(const StepArgs& a, const TmaLayout& L, bool first, bool braket, int grid, cudaStream_t st) {
  using CT = typename C2<F>::T;
  const int smem = L.stage_bytes * kTmaStages;
  auto x = static_cast<const CT*>(a.x);
  auto y = static_cast<CT*>(a.y);
  auto b = static_cast<const CT*>(a.bras);
  auto ev = static_cast<const F*>(a.eval);
  auto dg = static_cast<const F*>(a.diag);
  const uint32_t lim = g_wait_limit.load(std::memory_order_relaxed);
  if (braket)
    kpm_tma_step_kernel<F, R, CPLX_H, true, kTmaStages><<<grid, kTmaThreads, smem, st>>>(
        a.n, a.n_slices, a.n_tiles, L, a.soff, a.ecol, ev, dg, x, y, b, a.part, a.store, a.reverse, a.gather,
        first ? 1 : 0, a.err, lim);
  else
    kpm_tma_step_kernel<F, R, CPLX_H, false, kTmaStages><<<grid, kTmaThreads, smem, st>>>(
        a.n, a.n_slices, a.n_tiles, L, a.soff, a.ecol, ev, dg, x, y, b, a.part, a.store, a.reverse, a.gather,
        first ? 1 : 0, a.err, lim);
  TBK_CHECK_LAUNCH();
  return TBK_OK;
}

#define TBK_R_SWITCH(R, CALL64, CALL)                                   \
  switch (R) {                                                          \
    case 1: CALL(1); case 2: CALL(2); case 4: CALL(4); case 8: CALL(8);   \
    case 16: CALL(16); case 32: CALL(32); case 64: CALL64(64);          \
  }

template <typename F, bool CPLX_H>
static int launch_tma(int R, const StepArgs& a, const TmaLayout& L, bool first, bool braket, int grid,
                      cudaStream_t st) {
#define TBK_CALL(RR) return launch_tma_r<F, RR, CPLX_H>(a, L, first, braket, grid, st)
#define TBK_CALL64(RR) if constexpr (sizeof(F) == 4) { TBK_CALL(RR); } break
  TBK_R_SWITCH(R, TBK_CALL64, TBK_CALL)
#undef TBK_CALL
#undef TBK_CALL64
  return fail(TBK_ERR_UNSUPPORTED, "chunk width %d not instantiated", R);
}

template <typename F, bool CPLX_H>
static int tma_setup(int R, bool braket, int smem, int* occ) {
#define TBK_CALL(RR) return braket ? tma_kernel_setup<F, RR, CPLX_H, true>(smem, occ) : tma_kernel_setup<F, RR, CPLX_H, false>(smem, occ)
#define TBK_CALL64(RR) if constexpr (sizeof(F) == 4) { TBK_CALL(RR); } break
  TBK_R_SWITCH(R, TBK_CALL64, TBK_CALL)
#undef TBK_CALL
#undef TBK_CALL64
  return fail(TBK_ERR_UNSUPPORTED, "chunk width %d not instantiated", R);
}

// Width of the chunks that R vectors are processed in, at most cap (even) a chunk: the
// vectors spread evenly over the fewest chunks, rounded up to a lane's two vectors
// (complex64, double-float).  A width close to a power of two takes it: those kernels
// know their width at compile time (honeycomb 701x600, complex64: 20 vectors 80.9 us
// a step at width 20 against 107.8 at 32; with vacancies 83.5 against 108.8, FP64 braket
// 334 against 484).
int step_width(int prec, int R, int cap) {
  const int chunks = (R + cap - 1) / cap;
  int w = (R + chunks - 1) / chunks;
  if (prec != TBK_PREC_FP64 && w > 1) w = (w + 1) & ~1;
  int p = 1;
  while (p < w) p <<= 1;
  return p * 15 <= w * 16 ? p : w;
}

static int rows_per_tile(int prec, int Rc, int threads = kStepThreads) {
  const int vpl = prec != TBK_PREC_FP64 && Rc >= 2 ? 2 : 1;
  return threads / (Rc / vpl);
}

// ---------------------------------------------------------------- internal API
// (used by the Kubo block recursions in kubo.cu and the server)
// ELL value arrays of a precision: FP32, FP64 or double-float pairs.
const void* ell_vals(const EllDev& E, int prec) {
  return prec == TBK_PREC_MIXED ? E.val32.p : prec == TBK_PREC_DD ? E.valdd.p : E.val64.p;
}
const void* ell_diag(const EllDev& E, int prec) {
  return prec == TBK_PREC_MIXED ? E.diag32.p : prec == TBK_PREC_DD ? E.diagdd.p : E.diag64.p;
}

bool has_classes(const EllDev& E, int prec) {
  return E.cls_state == 1 || (prec == TBK_PREC_MIXED && E.cls32_state == 1);
}

bool has_row_classes(tbk_sparse_s* A, int prec) { return has_classes(A->ell, prec); }

static ClassTab class_tab32(const ClassSet32& c) {
  ClassTab t;
  t.cls = c.cls.as<uint8_t>();
  t.cnt = c.cnt.as<int32_t>();
  t.off = c.off.as<int32_t>();
  t.val = c.val[0].p;
  t.val2 = c.val[1].p;
  t.n_cls = c.n_cls;
  t.w = c.w;
  return t;
}

ClassTab class_tab(const EllDev& E, int prec) {
  ClassTab t;
  if (!has_classes(E, prec)) return t;
  if (E.cls_state != 1) return class_tab32(E.c32);
  t.cls = E.cls.as<uint8_t>();
  t.cnt = E.cls_cnt.as<int32_t>();
  t.off = E.cls_off.as<int32_t>();
  t.val = prec == TBK_PREC_MIXED ? E.cls_v32.p : prec == TBK_PREC_DD ? E.cls_vdd.p : E.cls_v64.p;
  t.n_cls = E.n_cls;
  t.w = E.cls_w;
  return t;
}

size_t class_smem(const EllDev& E, int prec) {
  const ClassTab t = class_tab(E, prec);
  const size_t ne = (size_t)t.n_cls * t.w;
  const size_t fb = prec == TBK_PREC_MIXED ? 4 : 8;         // float, double, double-float pair
  return ne * fb * (E.cplx ? 2 : 1) + ne * 4 + (size_t)t.n_cls * 4;
}

// Threads per CTA of the steps without sums: wide ones where every SM gets two waves of
// them (below that the smaller CTAs spread better).
static int step_threads(tbk_sparse_s* A, int Rc, int prec, int wide) {
  if (prec != TBK_PREC_MIXED || !has_classes(A->ell, prec)) return kStepThreads;
  const int64_t lanes = (int64_t)A->rows * (Rc >= 2 ? Rc / 2 : 1);
  return lanes >= (int64_t)wide * 2 * 2 * sm_count() ? wide : kStepThreads;
}

// CTAs per SM of A's form.  FP64: the smaller of both forms', so that they group their
// partial sums alike and give the same bits.
static int step_occupancy(tbk_sparse_s* A, int Rc, int prec, bool sums, int threads = kStepThreads) {
  const StepKind kind{sums, class_tab(A->ell, prec).w > 8};
  const bool cplx = A->ell.cplx != 0, cls = has_classes(A->ell, prec);
  const int oc = cls || prec == TBK_PREC_FP64
                     ? occupancy_cls_prec(prec, cplx, Rc, class_smem(A->ell, prec), kind, threads) : 64;
  const int oe = !cls || prec == TBK_PREC_FP64 ? occupancy_prec(prec, cplx, Rc, kind) : 64;
  return std::min(oc, oe);
}

static int tiles_of(tbk_sparse_s* A, int Rc, int prec, int threads) {
  const int rpt = rows_per_tile(prec, Rc, threads);
  return (A->rows + rpt - 1) / rpt;
}

int step_config(tbk_sparse_s* A, int Rc, int prec, int* grid, cudaStream_t st, bool wide) {
  TBK_TRY(ensure_ell(A, st));
  if (prec == TBK_PREC_DD) TBK_TRY(ensure_ell_dd(A, st));
  if (prec == TBK_PREC_MIXED) TBK_TRY(ensure_classes32(A, st));
  else TBK_TRY(ensure_classes(A, st));
  const int threads = wide ? step_threads(A, Rc, prec, kWideThreads<4>) : kStepThreads;
  *grid = std::max(1, std::min(tiles_of(A, Rc, prec, threads), sm_count() * step_occupancy(A, Rc, prec, false, threads)));
  return TBK_OK;
}

static int step_dispatch(tbk_sparse_s* A, int Rc, int prec, bool first, const StepArgs& a, int grid, cudaStream_t st);

static int pair_threads(tbk_sparse_s* A, int Rc) {
  const int64_t lanes = (int64_t)A->rows * (Rc >= 2 ? Rc / 2 : 1);
  return lanes >= (int64_t)kWideThreads<2> * 2 * 2 * sm_count() ? kWideThreads<2> : kStepThreads;
}

int pair_config(tbk_sparse_s* A, int Rc, const ClassSet32& pair, int* grid) {
  const int threads = pair_threads(A, Rc);
  // launch bounds: two CTAs of the wide size per SM
  const int per_sm = 2 * kWideThreads<2> / threads;
  *grid = std::max(1, std::min(tiles_of(A, Rc, TBK_PREC_MIXED, threads), sm_count() * per_sm));
  return TBK_OK;
}

int step_any(tbk_sparse_s* A, int Rc, int prec, const void* x, void* y, const void* pv, bool first, double* part,
             int grid, cudaStream_t st, const KStore* ks, bool store_y, tbk_sparse_s* vop, bool dots,
             const ClassSet32* pair, bool reverse) {
  StepArgs a;
  a.n = A->rows;
  a.n_slices = A->ell.n_slices;
  a.err = nullptr;
  a.soff = A->ell.slice_off.as<int32_t>();
  a.ecol = A->ell.col.as<int32_t>();
  a.eval = ell_vals(A->ell, prec);
  a.diag = ell_diag(A->ell, prec);
  a.x = x;
  a.y = y;
  a.pv = first ? y : pv;
  a.bras = nullptr;
  a.part = part;
  a.store = store_y ? 1 : 0;
  a.reverse = reverse ? 1 : 0;
  a.gather = 1;
  a.pf_dist = 1;
  a.pipe = A->ell.max_width > 4;
  if (ks) {
    a.ks = *ks;
    a.kst = ks->split ? 5 : 1;
    if (vop) {
      a.ks.vval[0] = ell_vals(vop->ell, prec);
      a.ks.vdiag[0] = ell_diag(vop->ell, prec);
      a.ks.usev[0] = 1;
      a.ks.vreal[0] = A->ell.cplx && !vop->ell.cplx;
      a.kst = 2;
      if (pair) {
        a.ct = class_tab32(*pair);
        a.threads = pair_threads(A, Rc);
      }
    }
  } else if (vop) {
    return fail(TBK_ERR_INVALID, "operator product without a store");
  } else if (!dots) {
    a.kst = 4;
  }
  return step_dispatch(A, Rc, prec, first, a, grid, st);
}

int step_ks(tbk_sparse_s* A, int Rc, int prec, const void* x, void* y, const void* pv, bool first, double* part,
            int grid, cudaStream_t st, const KStore& ks, int mode, bool reverse) {
  StepArgs a;
  a.n = A->rows;
  a.n_slices = A->ell.n_slices;
  a.err = nullptr;
  a.soff = A->ell.slice_off.as<int32_t>();
  a.ecol = A->ell.col.as<int32_t>();
  a.eval = ell_vals(A->ell, prec);
  a.diag = ell_diag(A->ell, prec);
  a.x = x;
  a.y = y;
  a.pv = first ? y : pv;
  a.bras = nullptr;
  a.part = part;
  a.store = 1;
  a.reverse = reverse ? 1 : 0;
  a.gather = 1;
  a.pf_dist = 1;
  a.ks = ks;
  a.kst = mode;
  a.pipe = A->ell.max_width > 4;
  return step_dispatch(A, Rc, prec, first, a, grid, st);
}

static int step_dispatch(tbk_sparse_s* A, int Rc, int prec, bool first, const StepArgs& a0, int grid, cudaStream_t st) {
  StepArgs a = a0;
  if (a.ct.val2) {                                          // joint classes with the operator
    a.cls = true;
  } else if (has_classes(A->ell, prec) && a.kst != 2) {     // the class form where it applies
    a.cls = true;
    a.ct = class_tab(A->ell, prec);
    if (a.kst != 0 && a.kst != 3) a.threads = step_threads(A, Rc, prec, kWideThreads<4>);   // kWideSteps
  }
  a.n_tiles = tiles_of(A, Rc, prec, a.threads);            // of the kernel that runs: the grid strides over any number
  return launch_step_prec(prec, A->ell.cplx != 0, Rc, a, first, false, grid, st);
}

int launch_step_f32(bool cplx, int R, const StepArgs& a, bool first, bool braket, int grid, cudaStream_t st);
int launch_step_f64(bool cplx, int R, const StepArgs& a, bool first, bool braket, int grid, cudaStream_t st);
int launch_step_dd(bool cplx, int R, const StepArgs& a, bool first, bool braket, int grid, cudaStream_t st);
int occupancy_f32(bool cplx, int R, StepKind kind);
int occupancy_f64(bool cplx, int R, StepKind kind);
int occupancy_dd(bool cplx, int R, StepKind kind);
int launch_step_cls_f32(bool cplx, int R, const StepArgs& a, bool first, bool braket, int grid, cudaStream_t st);
int launch_step_cls_f64(bool cplx, int R, const StepArgs& a, bool first, bool braket, int grid, cudaStream_t st);
int launch_step_cls_dd(bool cplx, int R, const StepArgs& a, bool first, bool braket, int grid, cudaStream_t st);
int occupancy_cls_f32(bool cplx, int R, size_t smem, StepKind kind, int threads);
int occupancy_cls_f64(bool cplx, int R, size_t smem, StepKind kind);
int occupancy_cls_dd(bool cplx, int R, size_t smem, StepKind kind);

int occupancy_cls_prec(int prec, bool cplx, int R, size_t smem, StepKind kind, int threads) {
  if (prec == TBK_PREC_FP64) return occupancy_cls_f64(cplx, R, smem, kind);
  if (prec == TBK_PREC_DD) return occupancy_cls_dd(cplx, R, smem, kind);
  return occupancy_cls_f32(cplx, R, smem, kind, threads);
}

int launch_step_prec(int prec, bool cplx, int R, const StepArgs& a, bool first, bool braket, int grid,
                     cudaStream_t st) {
  if (a.cls) {
    if (prec == TBK_PREC_FP64) return launch_step_cls_f64(cplx, R, a, first, braket, grid, st);
    if (prec == TBK_PREC_DD) return launch_step_cls_dd(cplx, R, a, first, braket, grid, st);
    return launch_step_cls_f32(cplx, R, a, first, braket, grid, st);
  }
  if (prec == TBK_PREC_FP64) return launch_step_f64(cplx, R, a, first, braket, grid, st);
  if (prec == TBK_PREC_DD) return launch_step_dd(cplx, R, a, first, braket, grid, st);
  return launch_step_f32(cplx, R, a, first, braket, grid, st);
}

int occupancy_prec(int prec, bool cplx, int R, StepKind kind) {
  if (prec == TBK_PREC_FP64) return occupancy_f64(cplx, R, kind);
  if (prec == TBK_PREC_DD) return occupancy_dd(cplx, R, kind);
  return occupancy_f32(cplx, R, kind);
}

int load_block_any(int prec, int32_t n, int32_t R, int32_t r0, int32_t Rp, const double2* src, void* dst,
                   cudaStream_t st) {
  dim3 g((unsigned)((n + 31) / 32), (unsigned)((Rp + 31) / 32)), b(32, 8);
  const int32_t rc = std::min(Rp, R - r0);
  if (prec == TBK_PREC_FP64) load_block_kernel<double><<<g, b, 0, st>>>(n, R, r0, rc, Rp, src, static_cast<double2*>(dst));
  else if (prec == TBK_PREC_DD) load_block_kernel<dd><<<g, b, 0, st>>>(n, R, r0, rc, Rp, src, static_cast<dd2*>(dst));
  else load_block_kernel<float><<<g, b, 0, st>>>(n, R, r0, rc, Rp, src, static_cast<float2*>(dst));
  TBK_CHECK_LAUNCH();
  return TBK_OK;
}

int random_block_any(int prec, int32_t n, int32_t R, int32_t r0, int32_t Rp, uint64_t seed, void* dst,
                     cudaStream_t st) {
  if (prec == TBK_PREC_FP64) random_block<double>(n, R, r0, Rp, seed, dst, st);
  else if (prec == TBK_PREC_DD) random_block<dd>(n, R, r0, Rp, seed, dst, st);
  else random_block<float>(n, R, r0, Rp, seed, dst, st);
  TBK_CHECK_LAUNCH();
  return TBK_OK;
}

}  // namespace tbk

using namespace tbk;

struct tbk_kpm_s {
  tbk_sparse_s* H = nullptr;
  int32_t R = 0, Rc = 0, n_chunks = 0, flags = 0, prec = 0;
  int64_t n = 0;
  size_t csize = 0;                 // bytes of one complex element
  DevBuf va, vb, bras, stage, part, sums, mu, err;
  int grid = 0, n_tiles = 0;        // legacy (one row group per warp) kernel
  int64_t n_pad = 0;                // rows of the work blocks (whole 32-row slices)
  bool use_tma = false;             // TMA-staged warp-specialised kernel
  TmaLayout lay_dbl{}, lay_brk{};   // stage layouts: doubling / braket
  int grid_dbl = 0, grid_brk = 0, tiles_tma = 0;
  int grid_max = 0;
  bool use_cls = false;             // one-pass kernel in the class form (translation-invariant H~)
  int pf_dist = 1;                  // L2 prefetch distance of the one-pass kernel (grid-stride waves)
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  cudaEvent_t tr[3] = {nullptr, nullptr, nullptr};   // TBK_TRACE: call start, after the upload, after the readback
  double last_ms = 0.0, last_bytes = 0.0;
  int32_t last_launches = 0;
  int32_t cap_steps = 0;            // partial buffer capacity (steps)
  // two-step passes (mixed precision, doubling): dependency tiles, deferred list, lag
  bool fused = false;
  int32_t lag = 0, n_def = 0, n_waves = 0, tpt = 4, n_tasks = 0;
  DevBuf dep, isdef, deflist, wave;
  // launch-bound plans (one chunk, small blocks): the recursion's launch
  // sequence is captured once per (steps, mode, buffers) and replayed
  cudaStream_t cap_st = nullptr;
  cudaGraphExec_t gexec = nullptr;
  struct GraphKey {
    int32_t n_steps = -1;
    bool braket = false;
    const void *va = nullptr, *vb = nullptr, *part = nullptr, *bras = nullptr;
    bool operator==(const GraphKey& o) const {
      return n_steps == o.n_steps && braket == o.braket && va == o.va && vb == o.vb && part == o.part &&
             bras == o.bras;
    }
  } gkey, seen;
  int small_state = 0;              // one-launch recursion: 0 undecided, 1 used, -1 not applicable
  SmallLayout slay{};
  bool cta = false;                 // the one-launch recursion is one CTA per vector (kpm_cta_kernel)
  int persist = 0;                  // cooperative recursion (kpm_persist_kernel): 0 undecided, 1 used, -1 not
  DevBuf meet;
  CtaLayout clay{};
};

// TBK_TRACE=1: every host-input solve prints its phases (upload, kets load,
// recursion, reduction and readback) in device milliseconds to stderr
static bool trace_on() {
  static const bool on = [] {
    const char* e = getenv("TBK_TRACE");
    return e && atoi(e) != 0;
  }();
  return on;
}

// Device view of a host pointer when it lies in pinned (registered) host
// memory, else null.
static const double2* mapped_host(const double* p) {
  cudaPointerAttributes at{};
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  if (at.type == cudaMemoryTypeHost && at.devicePointer) return static_cast<const double2*>(at.devicePointer);
  return nullptr;
}
// TBK_STAGE_UPLOAD=1: copy host inputs into a device staging buffer even when
// they are pinned (A/B of the in-place read)
static bool stage_uploads() {
  static const bool on = [] {
    const char* e = getenv("TBK_STAGE_UPLOAD");
    return e && atoi(e) != 0;
  }();
  return on;
}

// single-chunk plans whose work blocks fit in 64 MiB are launch-bound: replay
// their recursion as a graph
constexpr size_t kGraphBlockBytes = 64u << 20;

static int plan_partials(tbk_kpm_s* P, int32_t n_steps) {
  if (n_steps <= P->cap_steps) return TBK_OK;
  TBK_TRY(P->part.alloc(sizeof(double) * 2 * (size_t)n_steps * P->grid_max * P->n_chunks));
  TBK_TRY(P->sums.alloc(sizeof(double) * 2 * (size_t)n_steps));
  P->cap_steps = n_steps;
  return TBK_OK;
}

static int plan_mu(tbk_kpm_s* P, int32_t n_mom) {
  if (P->mu.bytes >= sizeof(double) * (size_t)n_mom) return TBK_OK;
  return P->mu.alloc(sizeof(double) * n_mom);
}

template <int R, bool C>
static void* fused_fn() { return reinterpret_cast<void*>(kpm_fused2_kernel<R, C>); }
static void* fused_kernel_ptr(int Rc, bool cplx) {
  switch (Rc) {
    case 1: return cplx ? fused_fn<1, true>() : fused_fn<1, false>();
    case 2: return cplx ? fused_fn<2, true>() : fused_fn<2, false>();
    case 4: return cplx ? fused_fn<4, true>() : fused_fn<4, false>();
    case 8: return cplx ? fused_fn<8, true>() : fused_fn<8, false>();
    case 16: return cplx ? fused_fn<16, true>() : fused_fn<16, false>();
    case 32: return cplx ? fused_fn<32, true>() : fused_fn<32, false>();
    case 64: return cplx ? fused_fn<64, true>() : fused_fn<64, false>();
  }
  return nullptr;
}

// Two-step passes: per-tile dependencies, far-reaching (wrap-around) tiles
// deferred, lag = the widest remaining reach + two waves of the grid.  Leaves
// P->fused false when the matrix does not suit (too many far tiles, lag >= size).
static int plan_fused(tbk_kpm_s* P, cudaStream_t st) {
  if (P->prec != TBK_PREC_MIXED || !(P->flags & TBK_FLAG_DOUBLING) || (P->flags & TBK_FLAG_STAGED) ||
      !(P->flags & TBK_FLAG_TWO_STEP))
    return TBK_OK;
  const EllDev& E = P->H->ell;
  const bool cplx = E.cplx != 0;
  void* fn = fused_kernel_ptr(P->Rc, cplx);
  if (!fn || P->n_tiles < 1) return TBK_OK;
  int occ = 0;
  TBK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kStepThreads, 0));
  if (occ < 1) return TBK_OK;
  int tpt = 4;                                          // base tiles per task
  if (const char* e = getenv("TBK_FUSE_TILES")) tpt = std::max(1, atoi(e));   // tuning override
  const int rpt = rows_per_tile(P->prec, P->Rc) * tpt;
  const int32_t nt = (int32_t)((P->n + rpt - 1) / rpt);   // tasks
  const int G = std::max(1, std::min(nt, std::min(P->grid, sm_count() * occ)));
  TBK_TRY(P->dep.alloc(sizeof(int32_t) * nt));
  iota_kernel<<<(nt + 255) / 256, 256, 0, st>>>(nt, P->dep.as<int32_t>());
  TBK_CHECK_LAUNCH();
  tile_dep_kernel<<<(unsigned)((P->n + 255) / 256), 256, 0, st>>>((int32_t)P->n, rpt, E.slice_off.as<int32_t>(),
                                                                  E.col.as<int32_t>(), P->dep.as<int32_t>());
  TBK_CHECK_LAUNCH();
  std::vector<int32_t> dep(nt);
  TBK_CUDA(cudaMemcpyAsync(dep.data(), P->dep.p, sizeof(int32_t) * nt, cudaMemcpyDeviceToHost, st));
  TBK_CUDA(cudaStreamSynchronize(st));
  const int32_t far = 8 * G;
  std::vector<uint8_t> isdef(nt, 0);
  std::vector<int32_t> defl;
  int32_t reach = 0;
  for (int32_t j = 0; j < nt; ++j) {
    const int32_t d = dep[j] - j;
    if (d > far) { isdef[j] = 1; defl.push_back(j); }
    else reach = std::max(reach, d);
  }
  const int32_t lag = reach + G + G / 2;
  if ((int64_t)defl.size() * 8 > nt || lag >= nt) return TBK_OK;
  TBK_TRY(P->isdef.alloc(nt));
  TBK_CUDA(cudaMemcpyAsync(P->isdef.p, isdef.data(), nt, cudaMemcpyHostToDevice, st));
  TBK_TRY(P->deflist.alloc(sizeof(int32_t) * (defl.size() + 1)));
  if (!defl.empty())
    TBK_CUDA(cudaMemcpyAsync(P->deflist.p, defl.data(), sizeof(int32_t) * defl.size(), cudaMemcpyHostToDevice, st));
  P->n_waves = (nt + G - 1) / G;
  TBK_TRY(P->wave.alloc(sizeof(unsigned int) * P->n_waves));
  TBK_CUDA(cudaStreamSynchronize(st));
  P->lag = lag;
  P->tpt = tpt;
  P->n_tasks = nt;
  P->n_def = (int32_t)defl.size();
  P->grid = G;                                          // both kernels write partials for this grid
  P->fused = true;
  return TBK_OK;
}

static int launch_fused(tbk_kpm_s* P, void* A, void* B, double* part1, double* part2, bool first, bool dot2,
                        cudaStream_t st) {
  const EllDev& E = P->H->ell;
  void* fn = fused_kernel_ptr(P->Rc, E.cplx != 0);
  TBK_CUDA(cudaMemsetAsync(P->wave.p, 0, sizeof(unsigned int) * P->n_waves, st));
  int32_t n = (int32_t)P->n, nt = P->n_tasks, tpt = P->tpt, ndef = P->n_def, lag = P->lag;
  const int32_t* soff = E.slice_off.as<int32_t>();
  const int32_t* ecol = E.col.as<int32_t>();
  const float* ev = E.val32.as<float>();
  const float* dg = E.diag32.as<float>();
  float2* a = static_cast<float2*>(A);
  float2* b = static_cast<float2*>(B);
  const int32_t* dep = P->dep.as<int32_t>();
  const uint8_t* isdef = P->isdef.as<uint8_t>();
  const int32_t* defl = P->deflist.as<int32_t>();
  unsigned int* wave = P->wave.as<unsigned int>();
  int fi = first ? 1 : 0, d2 = dot2 ? 1 : 0;
  int* err = P->err.as<int>();
  void* args[] = {&n, &nt, &tpt, &soff, &ecol, &ev, &dg, &a, &b, &dep, &isdef, &defl, &ndef, &lag, &wave, &part1,
                  &part2, &fi, &d2, &err};
  TBK_CUDA(cudaLaunchCooperativeKernel(fn, dim3(P->grid), dim3(kStepThreads), args, 0, st));
  return TBK_OK;
}

// one-launch recursion (kpm_small.cuh): one thread-block cluster per random
// vector keeps the vector and its slice of H~ in shared memory
constexpr int32_t kSmallSmemBytes = 200 << 10;

template <typename F, bool CPLX_H>
static void* small_kernel_ptr(bool braket) {
  return braket ? reinterpret_cast<void*>(kpm_cluster_kernel<F, CPLX_H, true>)
                : reinterpret_cast<void*>(kpm_cluster_kernel<F, CPLX_H, false>);
}
static void* small_kernel(int prec, bool cplx, bool braket) {
  if (prec == TBK_PREC_FP64) return cplx ? small_kernel_ptr<double, true>(braket) : small_kernel_ptr<double, false>(braket);
  if (prec == TBK_PREC_DD) return cplx ? small_kernel_ptr<dd, true>(braket) : small_kernel_ptr<dd, false>(braket);
  return cplx ? small_kernel_ptr<float, true>(braket) : small_kernel_ptr<float, false>(braket);
}

template <typename F, bool CPLX_H>
static void* cta_kernel_ptr(bool braket) {
  return braket ? reinterpret_cast<void*>(kpm_cta_kernel<F, CPLX_H, true>)
                : reinterpret_cast<void*>(kpm_cta_kernel<F, CPLX_H, false>);
}
static void* cta_kernel(bool cplx, bool braket) {
  return cplx ? cta_kernel_ptr<float, true>(braket) : cta_kernel_ptr<float, false>(braket);
}

// decides once per plan whether the one-launch recursion (TBK_FLAG_PERSISTENT)
// applies and lays out its shared memory.  Complex64 vectors of a matrix with
// row classes that fit one SM: one CTA per vector (kpm_cta_kernel; the
// 4,096-site, 8-vector solve: 0.40 ms against 0.63 ms for the per-step
// launches replayed as a graph).  Otherwise a cluster per vector: rows per CTA
// a power of two >= 32, at most 8 CTAs per cluster, at most 2 rows per
// thread.  (One CTA per double-float vector measured 0.91 ms against 0.74 ms:
// one SM's FP32 pipe sets the pace.)  Opt-in: the one-launch forms group the
// moment sums per vector, so their bits differ from the per-step kernels'
// (which the class and ELL forms share).
static int plan_small(tbk_kpm_s* P, bool tma) {
  if (P->small_state != 0) return TBK_OK;
  P->small_state = -1;
  if (!(P->flags & TBK_FLAG_PERSISTENT) || P->n_chunks != 1 || tma || (P->flags & TBK_FLAG_TWO_STEP)) return TBK_OK;
  const EllDev& E = P->H->ell;
  const int32_t n = (int32_t)P->n;
  if (P->use_cls && P->prec == TBK_PREC_MIXED) {
    CtaLayout C;
    C.n = n;
    const ClassTab ct = class_tab(E, P->prec);
    C.n_cls = ct.n_cls;
    C.w = ct.w;
    C.csz = (int32_t)P->csize;
    C.vb = (P->prec == TBK_PREC_MIXED ? 4 : 8) * (E.cplx ? 2 : 1);
    if ((int64_t)C.bytes() <= kSmallSmemBytes) {
      bool ok = true;
      for (int b = 0; b < 2 && ok; ++b)
        if (cudaFuncSetAttribute(cta_kernel(E.cplx != 0, b == 1), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 C.bytes()) != cudaSuccess) {
          cudaGetLastError();
          ok = false;
        }
      if (ok) {
        P->clay = C;
        P->cta = true;
        P->slay = SmallLayout{};
        P->slay.cs = 1;                   // partials: one pair per vector and step
        P->small_state = 1;
        if (P->R > P->grid_max) {
          P->grid_max = P->R;
          P->cap_steps = 0;
        }
        return TBK_OK;
      }
    }
  }
  int32_t rpc = 32, lg = 5;
  while ((int64_t)rpc * kClusterMax < n) { rpc <<= 1; ++lg; }
  if (rpc > 2 * kSmallThreadsMax) return TBK_OK;
  SmallLayout L;
  L.rpc = rpc;
  L.lg_rpc = lg;
  L.cs = (n + rpc - 1) / rpc;
  L.threads = std::min(rpc, kSmallThreadsMax);
  const bool cplx = E.cplx != 0;
  const int fb = P->prec == TBK_PREC_MIXED ? 4 : 8;      // float, double, dd (hi, lo)
  L.vb = fb * (cplx ? 2 : 1);
  L.csz = (int32_t)P->csize;
  std::vector<int32_t> so((size_t)E.n_slices + 1);
  TBK_CUDA(cudaMemcpy(so.data(), E.slice_off.p, sizeof(int32_t) * so.size(), cudaMemcpyDeviceToHost));
  int32_t max_ne = 0;
  for (int q = 0; q < L.cs; ++q) {
    const int32_t a = std::min(q * (rpc >> 5), E.n_slices), b = std::min((q + 1) * (rpc >> 5), E.n_slices);
    max_ne = std::max(max_ne, so[b] - so[a]);
  }
  L.max_ne = max_ne;
  if (L.bytes() > kSmallSmemBytes) return TBK_OK;
  void* fn[2] = {small_kernel(P->prec, cplx, false), small_kernel(P->prec, cplx, true)};
  for (void* f : fn) {
    TBK_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, L.bytes()));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = L.cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(P->R * L.cs);
    cfg.blockDim = dim3(L.threads);
    cfg.dynamicSmemBytes = L.bytes();
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, f, &cfg) != cudaSuccess || clusters < 1) {
      cudaGetLastError();
      return TBK_OK;
    }
  }
  P->slay = L;
  P->small_state = 1;
  if (P->R * L.cs > P->grid_max) {         // partials: one pair per CTA and step
    P->grid_max = P->R * L.cs;
    P->cap_steps = 0;
  }
  return TBK_OK;
}

template <typename F, bool CPLX_H>
static int launch_small_t(tbk_kpm_s* P, bool braket, int32_t n_steps, cudaStream_t st) {
  using CT = typename C2<F>::T;
  const EllDev& E = P->H->ell;
  const SmallLayout L = P->slay;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = L.cs;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(P->R * L.cs);
  cfg.blockDim = dim3(L.threads);
  cfg.dynamicSmemBytes = L.bytes();
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const int32_t n = (int32_t)P->n;
  const int32_t* so = E.slice_off.as<int32_t>();
  const int32_t* co = E.col.as<int32_t>();
  const F* ev = static_cast<const F*>(ell_vals(E, P->prec));
  const F* dg = static_cast<const F*>(ell_diag(E, P->prec));
  const CT* k = static_cast<const CT*>(P->va.p);
  const CT* b = braket ? static_cast<const CT*>(P->bras.p) : nullptr;
  double* pt = P->part.as<double>();
  if (braket)
    TBK_CUDA(cudaLaunchKernelEx(&cfg, kpm_cluster_kernel<F, CPLX_H, true>, n, E.n_slices, n_steps, P->Rc, L, so, co,
                                ev, dg, k, b, pt));
  else
    TBK_CUDA(cudaLaunchKernelEx(&cfg, kpm_cluster_kernel<F, CPLX_H, false>, n, E.n_slices, n_steps, P->Rc, L, so, co,
                                ev, dg, k, b, pt));
  return TBK_OK;
}

template <typename F, bool CPLX_H>
static int launch_cta_t(tbk_kpm_s* P, bool braket, int32_t n_steps, cudaStream_t st) {
  using CT = typename C2<F>::T;
  const EllDev& E = P->H->ell;
  const CtaLayout C = P->clay;
  const ClassTab ct = class_tab(E, P->prec);
  const F* dg = static_cast<const F*>(ell_diag(E, P->prec));
  const CT* k = static_cast<const CT*>(P->va.p);
  const CT* b = braket ? static_cast<const CT*>(P->bras.p) : nullptr;
  double* pt = P->part.as<double>();
  if (braket)
    kpm_cta_kernel<F, CPLX_H, true><<<P->R, cta_threads<F>(), C.bytes(), st>>>(n_steps, P->Rc, C, ct, dg, k, b, pt);
  else
    kpm_cta_kernel<F, CPLX_H, false><<<P->R, cta_threads<F>(), C.bytes(), st>>>(n_steps, P->Rc, C, ct, dg, k, b, pt);
  TBK_CHECK_LAUNCH();
  return TBK_OK;
}

static int launch_small(tbk_kpm_s* P, bool braket, int32_t n_steps, cudaStream_t st) {
  const bool c = P->H->ell.cplx != 0;
  if (P->cta) return c ? launch_cta_t<float, true>(P, braket, n_steps, st) : launch_cta_t<float, false>(P, braket, n_steps, st);
  if (P->prec == TBK_PREC_FP64) return c ? launch_small_t<double, true>(P, braket, n_steps, st)
                                         : launch_small_t<double, false>(P, braket, n_steps, st);
  if (P->prec == TBK_PREC_DD) return c ? launch_small_t<dd, true>(P, braket, n_steps, st)
                                       : launch_small_t<dd, false>(P, braket, n_steps, st);
  return c ? launch_small_t<float, true>(P, braket, n_steps, st) : launch_small_t<float, false>(P, braket, n_steps, st);
}

template <typename F>
static void* persist_kernel_t(bool cplx, bool braket, bool cls) {
  if (cplx) {
    if (braket) return cls ? (void*)kpm_persist_kernel<F, true, true, true> : (void*)kpm_persist_kernel<F, true, true, false>;
    return cls ? (void*)kpm_persist_kernel<F, true, false, true> : (void*)kpm_persist_kernel<F, true, false, false>;
  }
  if (braket) return cls ? (void*)kpm_persist_kernel<F, false, true, true> : (void*)kpm_persist_kernel<F, false, true, false>;
  return cls ? (void*)kpm_persist_kernel<F, false, false, true> : (void*)kpm_persist_kernel<F, false, false, false>;
}
static void* persist_kernel(const tbk_kpm_s* P, bool braket) {
  const bool cplx = P->H->ell.cplx != 0;
  if (P->prec == TBK_PREC_FP64) return persist_kernel_t<double>(cplx, braket, P->use_cls);
  if (P->prec == TBK_PREC_DD) return persist_kernel_t<dd>(cplx, braket, P->use_cls);
  return persist_kernel_t<float>(cplx, braket, P->use_cls);
}

// Decides once per plan whether the cooperative recursion applies: one chunk of whole
// lanes, one tile per CTA in the step kernels' own grid (so that the partial sums are
// the same), all CTAs resident at once in both modes.
static int plan_persist(tbk_kpm_s* P) {
  if (P->persist != 0) return TBK_OK;
  P->persist = -1;
  const bool lanes = P->prec == TBK_PREC_FP64 || P->Rc % 2 == 0;
  if (P->n_chunks != 1 || !lanes || P->n_tiles != P->grid ||
      (P->flags & (TBK_FLAG_STAGED | TBK_FLAG_TWO_STEP | TBK_FLAG_PERSISTENT | TBK_FLAG_NO_GRAPH)))
    return TBK_OK;
  // double-float: two CTAs an SM at most (honeycomb 200x200, R = 2, 313 tiles: 6.57 us a step, 5.89 in
  // launches of their own)
  if (P->prec == TBK_PREC_DD && P->grid > 2 * sm_count()) return TBK_OK;
  const size_t smem = P->use_cls ? class_smem(P->H->ell, P->prec) : 0;
  for (int b = 0; b < 2; ++b) {
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, persist_kernel(P, b == 1), kStepThreads, smem) !=
        cudaSuccess) {
      cudaGetLastError();
      return TBK_OK;
    }
    if (P->grid > nb * sm_count()) return TBK_OK;
  }
  TBK_TRY(P->meet.alloc(sizeof(unsigned int)));
  P->persist = 1;
  return TBK_OK;
}

// *launched false: the stream has fewer SMs than the plan counted on (a green context)
static int launch_persist(tbk_kpm_s* P, bool braket, int32_t n_steps, double* part, cudaStream_t st, bool* launched) {
  const EllDev& E = P->H->ell;
  const ClassTab ct = class_tab(E, P->prec);
  const size_t smem = P->use_cls ? class_smem(E, P->prec) : 0;
  TBK_CUDA(cudaMemsetAsync(P->meet.p, 0, sizeof(unsigned int), st));
  int32_t n = (int32_t)P->n, lpr = P->prec == TBK_PREC_FP64 ? P->Rc : P->Rc / 2;
  const int32_t* so = E.slice_off.as<int32_t>();
  const int32_t* co = E.col.as<int32_t>();
  const void* ev = ell_vals(E, P->prec);
  const void* dg = ell_diag(E, P->prec);
  void *va = P->va.p, *vb = P->vb.p, *br = braket ? P->bras.p : nullptr;
  unsigned int* meet = P->meet.as<unsigned int>();
  int* err = P->err.as<int>();
  uint32_t lim = g_wait_limit.load(std::memory_order_relaxed);
  void* args[] = {&n, &n_steps, &lpr, &so, &co, &ev, &dg, const_cast<ClassTab*>(&ct), &va, &vb, &br, &part, &meet, &err, &lim};
  const cudaError_t e = cudaLaunchCooperativeKernel(persist_kernel(P, braket), dim3(P->grid), dim3(kStepThreads), args, smem, st);
  *launched = e == cudaSuccess;
  if (e == cudaErrorCooperativeLaunchTooLarge) cudaGetLastError();
  else TBK_CUDA(e);
  return TBK_OK;
}

// Runs all chunks.  kets_loader(r0, dst) fills the chunk's v0 (site-major);
// bras_loader(r0, dst) fills the chunk's bras block (braket mode only).
template <typename KL, typename BL>
static int kpm_run_impl(tbk_kpm_s* P, int32_t n_mom, bool braket, KL&& kets_loader, BL&& bras_loader,
                        double* mu_out, bool mu_device, cudaStream_t st) {
  if (n_mom < 2) return fail(TBK_ERR_INVALID, "n must be greater than or equal to 2");
  const bool doubling = !braket;
  // doubling: step s yields mu_2s and mu_2s-1, so steps 0 .. n_mom/2 are needed
  const int32_t n_steps = doubling ? (n_mom <= 2 ? 1 : n_mom / 2 + 1) : n_mom - 1;
  const bool tma = P->use_tma && (P->flags & TBK_FLAG_STAGED);
  TBK_TRY(plan_small(P, tma));
  TBK_TRY(plan_persist(P));
  TBK_TRY(plan_partials(P, n_steps));
  TBK_TRY(plan_mu(P, n_mom));
  if (braket && P->bras.bytes < P->va.bytes) {
    TBK_TRY(P->bras.alloc(P->va.bytes));
    TBK_CUDA(cudaMemsetAsync(P->bras.p, 0, P->bras.bytes, st));
  }
  const EllDev& E = P->H->ell;
  const int G = tma ? (braket ? P->grid_brk : P->grid_dbl) : P->grid;
  const TmaLayout& lay = braket ? P->lay_brk : P->lay_dbl;
  TBK_CUDA(cudaMemsetAsync(P->err.p, 0, sizeof(int), st));
  const bool mixed = P->prec == TBK_PREC_MIXED;
  const bool cplx = P->H->ell.cplx != 0;
  float ms_total = 0.f;
  int32_t launches = 0;
  bool mirror = false;
  const bool small = P->small_state == 1;
  const int32_t nblk = small ? P->R * P->slay.cs : G;    // partials per (step, slot)
  for (int32_t ch = 0; ch < P->n_chunks; ++ch) {
    const int32_t r0 = ch * P->Rc;
    TBK_TRY(kets_loader(r0, P->va.p));
    if (braket) TBK_TRY(bras_loader(r0, P->bras.p));
    TBK_CUDA(cudaEventRecord(P->ev0, st));
    void* x = P->va.p;
    void* y = P->vb.p;
    int32_t s = 0;
    if (doubling && P->fused && !tma) {
      // pairs of steps per pass: x keeps v_s (then v_{s+2}), y keeps v_{s-1} (then v_{s+1})
      for (; s + 1 < n_steps; s += 2) {
        double* p1 = P->part.as<double>() + (((int64_t)ch * n_steps + s) * 2) * G;
        double* p2 = P->part.as<double>() + (((int64_t)ch * n_steps + s + 1) * 2) * G;
        const bool dot2 = s + 1 == n_steps - 1;
        TBK_TRY(launch_fused(P, x, y, p1, p2, s == 0, dot2, st));
        ++launches;
      }
    }
    auto issue = [&](cudaStream_t q, int32_t s_begin, void* xx, void* yy) -> int {
    for (int32_t s = s_begin; s < n_steps; ++s) {
      StepArgs a;
      a.n = (int32_t)P->n;
      a.n_tiles = tma ? P->tiles_tma : P->n_tiles;
      a.n_slices = E.n_slices;
      a.err = P->err.as<int>();
      a.pf_dist = P->pf_dist;
      a.soff = E.slice_off.as<int32_t>();
      a.ecol = E.col.as<int32_t>();
      a.eval = ell_vals(E, P->prec);
      a.diag = ell_diag(E, P->prec);
      a.x = xx;
      a.y = yy;
      a.pv = yy;
      a.bras = braket ? P->bras.p : nullptr;
      a.part = P->part.as<double>() + (((int64_t)ch * n_steps + s) * 2) * G;
      const bool last_dot = doubling && s == n_steps - 1 && s > 0;   // dots only, no product
      a.store = last_dot ? 0 : 1;
      a.gather = last_dot ? 0 : 1;
      a.reverse = (P->flags & TBK_FLAG_NO_L2_ZIGZAG) ? 0 : (s & 1);
      a.pipe = E.max_width > 4;
      if (P->use_cls && !tma) {
        a.cls = true;
        a.ct = class_tab(E, P->prec);
      }
      const bool first = s == 0;
      int rc;
      if (tma) {
        if (mixed) rc = cplx ? launch_tma<float, true>(P->Rc, a, lay, first, braket, G, q)
                             : launch_tma<float, false>(P->Rc, a, lay, first, braket, G, q);
        else rc = cplx ? launch_tma<double, true>(P->Rc, a, lay, first, braket, G, q)
                       : launch_tma<double, false>(P->Rc, a, lay, first, braket, G, q);
      } else {
        rc = launch_step_prec(P->prec, cplx, P->Rc, a, first, braket, G, q);
      }
      if (rc != TBK_OK) return rc;
      std::swap(xx, yy);   // yy now holds v_{n+1}; it becomes xx, xx (v_n) becomes the next v_{n-1}
    }
    return TBK_OK;
    };
    const bool graphable = P->n_chunks == 1 && s == 0 && !tma && !(P->flags & TBK_FLAG_NO_GRAPH) &&
                           P->va.bytes <= kGraphBlockBytes;
    bool issued = small;
    if (small) {
      TBK_TRY(launch_small(P, braket, n_steps, st));
      launches += 1;
    } else if (P->persist == 1 && (int64_t)n_steps * P->grid < (int64_t)INT32_MAX) {
      TBK_TRY(launch_persist(P, braket, n_steps, P->part.as<double>(), st, &issued));
      mirror = issued && !(P->flags & TBK_FLAG_NO_L2_ZIGZAG);
      launches += issued ? n_steps : 0;
    }
    if (!issued && graphable) {
      tbk_kpm_s::GraphKey key;
      key.n_steps = n_steps;
      key.braket = braket;
      key.va = P->va.p;
      key.vb = P->vb.p;
      key.part = P->part.p;
      key.bras = braket ? P->bras.p : nullptr;
      if (!(P->gexec && P->gkey == key) && P->seen == key) {
        // second identical run: capture the launch sequence on the plan's own
        // stream (thread-local mode: other threads' launches are unaffected)
        if (!P->cap_st) TBK_CUDA(cudaStreamCreateWithFlags(&P->cap_st, cudaStreamNonBlocking));
        if (P->gexec) {
          cudaGraphExecDestroy(P->gexec);
          P->gexec = nullptr;
        }
        cudaGraph_t g = nullptr;
        TBK_CUDA(cudaStreamBeginCapture(P->cap_st, cudaStreamCaptureModeThreadLocal));
        const int rc = issue(P->cap_st, 0, x, y);
        const cudaError_t ec = cudaStreamEndCapture(P->cap_st, &g);
        if (rc != TBK_OK) {
          if (g) cudaGraphDestroy(g);
          return rc;
        }
        if (ec != cudaSuccess) return fail(TBK_ERR_CUDA, "recursion graph capture: %s", cudaGetErrorString(ec));
        const cudaError_t ei = cudaGraphInstantiate(&P->gexec, g, 0);
        cudaGraphDestroy(g);
        if (ei != cudaSuccess) {
          P->gexec = nullptr;
          return fail(TBK_ERR_CUDA, "recursion graph instantiate: %s", cudaGetErrorString(ei));
        }
        P->gkey = key;
      }
      P->seen = key;
      if (P->gexec && P->gkey == key) {
        TBK_CUDA(cudaGraphLaunch(P->gexec, st));
        launches += n_steps;
      } else {
        TBK_TRY(issue(st, 0, x, y));
        launches += n_steps;
      }
    } else if (!issued) {
      TBK_TRY(issue(st, s, x, y));
      launches += n_steps - s;
    }
    TBK_CUDA(cudaEventRecord(P->ev1, st));
    TBK_CUDA(cudaEventSynchronize(P->ev1));
    float ms = 0.f;
    TBK_CUDA(cudaEventElapsedTime(&ms, P->ev0, P->ev1));
    ms_total += ms;
  }
  reduce_partials_kernel<<<dim3(n_steps, 2), 256, 0, st>>>(P->part.as<double>(), P->n_chunks, n_steps, nblk,
                                                          mirror ? 1 : 0, P->sums.as<double>());
  TBK_CHECK_LAUNCH();
  assemble_moments_kernel<<<(n_mom + 255) / 256, 256, 0, st>>>(P->sums.as<double>(), n_mom, doubling ? 1 : 0,
                                                               P->mu.as<double>());
  TBK_CHECK_LAUNCH();
  if (mu_device) TBK_CUDA(cudaMemcpyAsync(mu_out, P->mu.p, sizeof(double) * n_mom, cudaMemcpyDeviceToDevice, st));
  else TBK_CUDA(cudaMemcpyAsync(mu_out, P->mu.p, sizeof(double) * n_mom, cudaMemcpyDeviceToHost, st));
  int herr = 0;
  TBK_CUDA(cudaMemcpyAsync(&herr, P->err.p, sizeof(int), cudaMemcpyDeviceToHost, st));
  if (P->tr[2]) TBK_CUDA(cudaEventRecord(P->tr[2], st));
  TBK_CUDA(cudaStreamSynchronize(st));
  if (P->tr[2] && P->n_chunks == 1) {
    float up = 0.f, ld = 0.f, rec = 0.f, tail = 0.f;
    cudaEventElapsedTime(&up, P->tr[0], P->tr[1]);
    cudaEventElapsedTime(&ld, P->tr[1], P->ev0);
    cudaEventElapsedTime(&rec, P->ev0, P->ev1);
    cudaEventElapsedTime(&tail, P->ev1, P->tr[2]);
    fprintf(stderr, "tbk trace: upload %.3f ms, kets load %.3f ms, recursion %.3f ms, reduce+readback %.3f ms\n", up,
            ld, rec, tail);
  }
  if (herr) return fail(TBK_ERR_TIMEOUT, "recursion kernel gave up waiting (code %d)", herr);
  // algorithmic DRAM bytes per recursion launch (average over the launches)
  const double vec = (double)P->n * P->Rc * P->csize;
  const double hv = (mixed ? 4.0 : 8.0) * (cplx ? 2.0 : 1.0);
  // class form: the row's class byte and its diagonal value (the table is in shared memory)
  const double mat_ell = (double)E.n_entries * (4.0 + hv) + (double)E.n_rows * hv + 4.0 * (E.n_slices + 1);
  const double mat = (P->use_cls && !tma) ? (double)E.n_rows * (1.0 + hv) : mat_ell;
  double per_chunk = 0.0;
  int32_t s0 = 0;
  if (doubling && P->fused && !tma) {
    // a pass reads v_s, v_{s-1} and H~ once and writes v_{s+1}, v_{s+2}; v_{s+1}
    // and v_s are read again from L2 by the second step
    for (; s0 + 1 < n_steps; s0 += 2) {
      const bool dot2 = s0 + 1 == n_steps - 1;
      per_chunk += (s0 > 0 ? 2 : 1) * vec + vec + (dot2 ? 0.0 : vec) + mat_ell;
    }
  }
  for (int32_t s = s0; s < n_steps; ++s) {
    const bool last_dot = doubling && s == n_steps - 1 && s > 0;
    double b = vec;                                        // x
    if (s > 0) b += vec;                                   // v_{n-1}
    if (!last_dot) b += vec + mat;                         // y store + H~
    if (braket) b += vec;                                  // bras
    per_chunk += b;
  }
  P->last_ms = ms_total;
  P->last_launches = launches;
  P->last_bytes = launches ? per_chunk * P->n_chunks / launches : 0.0;
  return TBK_OK;
}

extern "C" {

int tbk_kpm_create(tbk_kpm* out, tbk_sparse Ht, int32_t R, int32_t flags) {
  if (!out || !Ht) return fail(TBK_ERR_INVALID, "tbk_kpm_create: null argument");
  *out = nullptr;
  if (R < 1) return fail(TBK_ERR_INVALID, "R must be >= 1");
  const int prec = flags & TBK_FLAG_PREC_MASK;
  if (prec != TBK_PREC_FP64 && prec != TBK_PREC_MIXED && prec != TBK_PREC_DD)
    return fail(TBK_ERR_INVALID, "unknown precision %d", prec);
  cudaStream_t st = nullptr;
  ScratchScope scope(st);
  TBK_TRY(ensure_ell(Ht, st));
  if (prec == TBK_PREC_DD) TBK_TRY(ensure_ell_dd(Ht, st));
  auto* P = new tbk_kpm_s();
  P->H = Ht;
  P->R = R;
  P->flags = flags;
  P->prec = prec;
  P->n = Ht->rows;
  P->csize = prec == TBK_PREC_MIXED ? 8 : 16;
  const int rmax = prec == TBK_PREC_MIXED ? 64 : 32;
  int rc = 1;
  while (rc < R && rc < rmax) rc <<= 1;
  // the opt-in forms exist for powers of two only
  if (!(flags & (TBK_FLAG_STAGED | TBK_FLAG_TWO_STEP | TBK_FLAG_PERSISTENT))) rc = step_width(prec, R, rmax);
  P->Rc = rc;
  P->n_chunks = (R + rc - 1) / rc;
  const int rpt = rows_per_tile(prec, rc);
  P->n_tiles = (int)((P->n + rpt - 1) / rpt);
  int occ = 1;
  const bool cplx = Ht->ell.cplx != 0;
  {
    const int s0 = prec == TBK_PREC_MIXED ? ensure_classes32(Ht, st) : ensure_classes(Ht, st);
    if (s0 != TBK_OK) {
      delete P;
      return s0;
    }
  }
  P->use_cls = has_classes(Ht->ell, prec);
  occ = step_occupancy(Ht, rc, prec, true);
  P->grid = std::max(1, std::min(P->n_tiles, sm_count() * occ));
  P->grid_max = P->grid;
  if (const char* e = getenv("TBK_PREFETCH")) P->pf_dist = atoi(e);   // tuning override
  P->n_pad = (int64_t)Ht->ell.n_slices * 32;
  // TMA-staged kernel: tiles of whole slices, ~8 KB of vector rows per stream
  if (flags & TBK_FLAG_STAGED) {
    const int row_bytes = rc * (int)P->csize;
    int TR = 8192 / row_bytes;
    if (const char* e = getenv("TBK_TMA_ROWS")) TR = atoi(e);   // tuning override (rows per tile)
    TR = std::max(32, std::min(512, TR)) & ~31;
    const int hsize = (prec == TBK_PREC_MIXED ? 4 : 8) * (cplx ? 2 : 1);
    const int wmax = std::max(1, Ht->ell.max_width);
    P->lay_dbl = make_tma_layout(TR, wmax, rc, (int)P->csize, hsize, false);
    P->lay_brk = make_tma_layout(TR, wmax, rc, (int)P->csize, hsize, true);
    const int smem_brk = P->lay_brk.stage_bytes * kTmaStages;
    // FP64 on GB300 is bound by the FP64 pipe, where more resident warps of the
    // one-pass kernel beat the staged ring; the staged kernel serves complex64.
    if (prec == TBK_PREC_MIXED && smem_brk <= 200 * 1024 && Ht->ell.n_slices > 0) {
      int occ_d = 0, occ_b = 0, st1, st2;
      if (prec == TBK_PREC_MIXED) {
        st1 = cplx ? tma_setup<float, true>(rc, false, P->lay_dbl.stage_bytes * kTmaStages, &occ_d)
                   : tma_setup<float, false>(rc, false, P->lay_dbl.stage_bytes * kTmaStages, &occ_d);
        st2 = cplx ? tma_setup<float, true>(rc, true, smem_brk, &occ_b) : tma_setup<float, false>(rc, true, smem_brk, &occ_b);
      } else {
        st1 = cplx ? tma_setup<double, true>(rc, false, P->lay_dbl.stage_bytes * kTmaStages, &occ_d)
                   : tma_setup<double, false>(rc, false, P->lay_dbl.stage_bytes * kTmaStages, &occ_d);
        st2 = cplx ? tma_setup<double, true>(rc, true, smem_brk, &occ_b) : tma_setup<double, false>(rc, true, smem_brk, &occ_b);
      }
      if (st1 == TBK_OK && st2 == TBK_OK && occ_d > 0 && occ_b > 0) {
        P->tiles_tma = (int)((P->n_pad + TR - 1) / TR);
        P->grid_dbl = std::max(1, std::min(P->tiles_tma, sm_count() * occ_d));
        P->grid_brk = std::max(1, std::min(P->tiles_tma, sm_count() * occ_b));
        P->grid_max = std::max(P->grid_max, std::max(P->grid_dbl, P->grid_brk));
        P->use_tma = true;
      }
    }
  }
  const size_t blk = (size_t)P->n_pad * rc * P->csize;
  int s;
  if ((s = P->va.alloc(blk)) != TBK_OK || (s = P->vb.alloc(blk)) != TBK_OK || (s = P->err.alloc(sizeof(int))) != TBK_OK) {
    delete P;
    return s;
  }
  if (cudaMemset(P->va.p, 0, blk) != cudaSuccess || cudaMemset(P->vb.p, 0, blk) != cudaSuccess) {
    delete P;
    return fail(TBK_ERR_CUDA, "cudaMemset of the work blocks failed");
  }
  if (cudaEventCreate(&P->ev0) != cudaSuccess || cudaEventCreate(&P->ev1) != cudaSuccess) {
    delete P;
    return fail(TBK_ERR_CUDA, "cudaEventCreate failed");
  }
  if ((s = plan_fused(P, st)) != TBK_OK) {
    delete P;
    return s;
  }
  if (cudaStreamSynchronize(st) != cudaSuccess) {          // the blocks are ready for any stream
    delete P;
    return fail(TBK_ERR_CUDA, "tbk_kpm_create: work blocks");
  }
  *out = P;
  return TBK_OK;
}

void tbk_kpm_destroy(tbk_kpm P) {
  if (!P) return;
  cudaDeviceSynchronize();
  if (P->ev0) cudaEventDestroy(P->ev0);
  if (P->ev1) cudaEventDestroy(P->ev1);
  for (auto e : P->tr)
    if (e) cudaEventDestroy(e);
  if (P->gexec) cudaGraphExecDestroy(P->gexec);
  if (P->cap_st) cudaStreamDestroy(P->cap_st);
  delete P;
}

int tbk_kpm_run(tbk_kpm P, int32_t n_mom, const double* bras, const double* kets, double* mu_out,
                void* stream) {
  if (!P || !kets || !bras || !mu_out) return fail(TBK_ERR_INVALID, "tbk_kpm_run: null argument");
  cudaStream_t st = as_stream(stream);
  ScratchScope scope(st);
  const bool dev = (P->flags & TBK_FLAG_DEVICE_PTRS) != 0;
  const bool doubling = (P->flags & TBK_FLAG_DOUBLING) != 0;
  if (doubling && bras != kets) return fail(TBK_ERR_INVALID, "TBK_FLAG_DOUBLING needs bras == kets");
  const bool same = bras == kets;
  const size_t in_bytes = sizeof(double2) * (size_t)P->n * P->R;
  // Host inputs.  Pinned (page-locked, registered) host memory is mapped into
  // the device's address space: the load kernel then reads its columns in
  // place over the host link (NVLink-C2C on GB300), with no staging buffer and
  // no separate copy.  Other host memory is copied into a device staging
  // buffer first (one copy each); every chunk transposes its columns from there.
  const double2* kets_dev = reinterpret_cast<const double2*>(kets);
  const double2* bras_dev = reinterpret_cast<const double2*>(bras);
  bool mapped = false;
  if (!dev && !stage_uploads()) {
    const double2* km = mapped_host(kets);
    const double2* bm = same ? km : mapped_host(bras);
    if (km && bm) {
      kets_dev = km;
      bras_dev = bm;
      mapped = true;
      if (trace_on() && !P->tr[0])
        for (auto& e : P->tr) TBK_CUDA(cudaEventCreate(&e));
      if (P->tr[0]) {
        TBK_CUDA(cudaEventRecord(P->tr[0], st));
        TBK_CUDA(cudaEventRecord(P->tr[1], st));
      }
    }
  }
  if (!dev && !mapped) {
    const size_t need = same ? in_bytes : 2 * in_bytes;
    if (P->stage.bytes < need) TBK_TRY(P->stage.alloc(need));
    if (trace_on() && !P->tr[0])
      for (auto& e : P->tr) TBK_CUDA(cudaEventCreate(&e));
    if (P->tr[0]) TBK_CUDA(cudaEventRecord(P->tr[0], st));
    TBK_CUDA(cudaMemcpyAsync(P->stage.p, kets, in_bytes, cudaMemcpyHostToDevice, st));
    kets_dev = P->stage.as<double2>();
    bras_dev = kets_dev;
    if (!same) {
      TBK_CUDA(cudaMemcpyAsync(P->stage.as<char>() + in_bytes, bras, in_bytes, cudaMemcpyHostToDevice, st));
      bras_dev = reinterpret_cast<const double2*>(P->stage.as<char>() + in_bytes);
    }
    if (P->tr[1]) TBK_CUDA(cudaEventRecord(P->tr[1], st));
  }
  const bool mixed = P->prec == TBK_PREC_MIXED;
  auto load_from = [&](const double2* src) {
    return [&, src](int32_t r0, void* dst) -> int {
      dim3 g((unsigned)((P->n + 31) / 32), (unsigned)((P->Rc + 31) / 32)), b(32, 8);
      int32_t rc = std::min(P->Rc, P->R - r0);
      if (mixed) load_block_kernel<float><<<g, b, 0, st>>>((int32_t)P->n, P->R, r0, rc, P->Rc, src, static_cast<float2*>(dst));
      else if (P->prec == TBK_PREC_DD) load_block_kernel<dd><<<g, b, 0, st>>>((int32_t)P->n, P->R, r0, rc, P->Rc, src, static_cast<dd2*>(dst));
      else load_block_kernel<double><<<g, b, 0, st>>>((int32_t)P->n, P->R, r0, rc, P->Rc, src, static_cast<double2*>(dst));
      TBK_CHECK_LAUNCH();
      return TBK_OK;
    };
  };
  return kpm_run_impl(P, n_mom, !doubling, load_from(kets_dev), load_from(bras_dev), mu_out, dev, st);
}

int tbk_kpm_run_random(tbk_kpm P, int32_t n_mom, uint64_t seed, double* mu_out, void* stream) {
  if (!P || !mu_out) return fail(TBK_ERR_INVALID, "tbk_kpm_run_random: null argument");
  cudaStream_t st = as_stream(stream);
  ScratchScope scope(st);
  const bool dev = (P->flags & TBK_FLAG_DEVICE_PTRS) != 0;
  const bool mixed = P->prec == TBK_PREC_MIXED;
  const bool doubling = (P->flags & TBK_FLAG_DOUBLING) != 0;
  auto gen = [&](int32_t r0, void* dst) -> int {
    int64_t tot = P->n * P->Rc;
    TBK_TRY(random_block_any(P->prec, (int32_t)P->n, P->R, r0, P->Rc, seed, dst, st));
    (void)mixed; (void)tot;
    TBK_CHECK_LAUNCH();
    return TBK_OK;
  };
  return kpm_run_impl(P, n_mom, !doubling, gen, gen, mu_out, dev, st);
}

int tbk_kpm_last_timing(tbk_kpm P, double* ms, int32_t* launches, double* bytes) {
  if (!P) return fail(TBK_ERR_INVALID, "tbk_kpm_last_timing: null plan");
  if (ms) *ms = P->last_ms;
  if (launches) *launches = P->last_launches;
  if (bytes) *bytes = P->last_bytes;
  return TBK_OK;
}

}  // extern "C"

namespace {

// Drop-in plan cache.  The reference's callers (GreenFunctionImag,
// TB/lattice.h:605-615) call Cheb_first_kind_seq_braket again and again with
// the same rescaled matrix; every call still uploads the CSC arrays (the
// reference's contract: host inputs), and a device comparison against the
// arrays of the previous call decides whether the matrix, its ELL and row
// classes and the recursion plans (work blocks, captured graphs) can be
// reused.  A different matrix replaces the cached one; tbk_cheb_braket_release
// frees everything; TBK_FLAG_NO_CACHE builds and frees per call.
struct DropinCache {
  std::mutex mu;
  tbk_sparse H = nullptr;
  int32_t rows = -1, cplx = -1;
  int64_t nnz = -1;
  DevBuf stage, flag;
  struct Plan {
    int32_t R, flags;
    tbk_kpm P;
  };
  std::vector<Plan> plans;
  void drop_plans() {
    for (auto& q : plans) tbk_kpm_destroy(q.P);
    plans.clear();
  }
  void drop() {
    drop_plans();
    if (H) tbk_sparse_destroy(H);
    H = nullptr;
    rows = cplx = -1;
    nnz = -1;
    stage.release();
    flag.release();
  }
};
DropinCache g_dropin;
constexpr size_t kDropinPlans = 4;

__global__ void words_differ_kernel(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, int64_t nw,
                                    int* __restrict__ flag) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < nw; q += (int64_t)gridDim.x * blockDim.x)
    if (a[q] != b[q]) {
      atomicOr(flag, 1);
      return;
    }
}

int words_differ(const void* a, const void* b, size_t bytes, int* flag, cudaStream_t st) {
  const int64_t nw = (int64_t)(bytes / 4);
  if (nw == 0) return TBK_OK;
  const unsigned g = (unsigned)std::min<int64_t>((nw + 255) / 256, 4096);
  words_differ_kernel<<<g, 256, 0, st>>>(static_cast<const uint32_t*>(a), static_cast<const uint32_t*>(b), nw, flag);
  TBK_CHECK_LAUNCH();
  return TBK_OK;
}

size_t align16(size_t b) { return (b + 15) & ~size_t(15); }

int cheb_braket_cached(int32_t n_rows, int64_t nnz, const int32_t* cp, const int32_t* ri, const double* v, int cplx,
                       int32_t n, const double* bras, const double* kets, int32_t R, int32_t flags,
                       double* mu_out) {
  DropinCache& C = g_dropin;
  std::lock_guard<std::mutex> lock(C.mu);
  cudaStream_t st = nullptr;                               // synchronous, as the reference
  ScratchScope scope(st);
  const size_t bcp = sizeof(int32_t) * ((size_t)n_rows + 1), bri = sizeof(int32_t) * (size_t)nnz;
  const size_t bv = sizeof(double) * (cplx ? 2 : 1) * (size_t)nnz;
  const size_t o_ri = align16(bcp), o_v = o_ri + align16(bri), need = o_v + align16(bv);
  if (C.stage.bytes < need) TBK_TRY(C.stage.alloc(need));
  if (!C.flag.p) TBK_TRY(C.flag.alloc(sizeof(int)));
  char* sb = C.stage.as<char>();
  TBK_CUDA(cudaMemcpyAsync(sb, cp, bcp, cudaMemcpyHostToDevice, st));
  if (nnz) {
    TBK_CUDA(cudaMemcpyAsync(sb + o_ri, ri, bri, cudaMemcpyHostToDevice, st));
    TBK_CUDA(cudaMemcpyAsync(sb + o_v, v, bv, cudaMemcpyHostToDevice, st));
  }
  bool same = C.H && C.rows == n_rows && C.nnz == nnz && C.cplx == cplx;
  if (same) {
    TBK_CUDA(cudaMemsetAsync(C.flag.p, 0, sizeof(int), st));
    TBK_TRY(words_differ(sb, C.H->col_ptr.p, bcp, C.flag.as<int>(), st));
    TBK_TRY(words_differ(sb + o_ri, C.H->row_idx.p, bri, C.flag.as<int>(), st));
    TBK_TRY(words_differ(sb + o_v, C.H->values.p, bv, C.flag.as<int>(), st));
    int h = 1;
    TBK_CUDA(cudaMemcpyAsync(&h, C.flag.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    TBK_CUDA(cudaStreamSynchronize(st));
    same = h == 0;
  }
  if (!same) {
    C.drop_plans();
    if (C.H) tbk_sparse_destroy(C.H);
    C.H = nullptr;
    C.rows = C.cplx = -1;
    C.nnz = -1;
    tbk_sparse H = nullptr;
    TBK_TRY(tbk_sparse_from_csc(&H, n_rows, n_rows, nnz, reinterpret_cast<const int32_t*>(sb),
                                reinterpret_cast<const int32_t*>(sb + o_ri), reinterpret_cast<const double*>(sb + o_v),
                                cplx, 1, nullptr));
    C.H = H;
    C.rows = n_rows;
    C.nnz = nnz;
    C.cplx = cplx;
  }
  const int32_t pf = flags & ~TBK_FLAG_DEVICE_PTRS;
  tbk_kpm P = nullptr;
  for (auto& q : C.plans)
    if (q.R == R && q.flags == pf) P = q.P;
  if (!P) {
    if (C.plans.size() >= kDropinPlans) {
      tbk_kpm_destroy(C.plans.front().P);
      C.plans.erase(C.plans.begin());
    }
    TBK_TRY(tbk_kpm_create(&P, C.H, R, pf));
    C.plans.push_back({R, pf, P});
  }
  return tbk_kpm_run(P, n, bras, kets, mu_out, nullptr);
}

}  // namespace

extern "C" {

static int cheb_braket_common(int32_t n_rows, int64_t nnz, const int32_t* cp, const int32_t* ri,
                              const double* v, int cplx, int32_t n, const double* bras, const double* kets,
                              int32_t R, int32_t flags, double* mu_out) {
  if (!cp || !bras || !kets || !mu_out || (nnz > 0 && (!ri || !v)))
    return fail(TBK_ERR_INVALID, "Cheb_first_kind_seq_braket: null argument");
  if (n < 2) return fail(TBK_ERR_INVALID, "n must be greater than or equal to 2");
  if (n_rows < 1 || R < 1) return fail(TBK_ERR_INVALID, "Cheb_first_kind_seq_braket: empty input");
  if (nnz < 0 || nnz > INT32_MAX) return fail(TBK_ERR_INVALID, "Cheb_first_kind_seq_braket: bad nnz");
  if ((flags & TBK_FLAG_DOUBLING) && bras != kets)
    return fail(TBK_ERR_INVALID, "TBK_FLAG_DOUBLING needs bras == kets");
  if (!(flags & TBK_FLAG_NO_CACHE))
    return cheb_braket_cached(n_rows, nnz, cp, ri, v, cplx, n, bras, kets, R, flags & ~TBK_FLAG_NO_CACHE, mu_out);
  tbk_sparse H = nullptr;
  TBK_TRY(tbk_sparse_from_csc(&H, n_rows, n_rows, nnz, cp, ri, v, cplx, 0, nullptr));
  tbk_kpm P = nullptr;
  int s = tbk_kpm_create(&P, H, R, flags & ~(TBK_FLAG_DEVICE_PTRS | TBK_FLAG_NO_CACHE));
  if (s == TBK_OK) s = tbk_kpm_run(P, n, bras, kets, mu_out, nullptr);
  tbk_kpm_destroy(P);
  tbk_sparse_destroy(H);
  return s;
}

int tbk_set_wait_limit(int64_t polls) {
  if (polls > (int64_t)kWaitLimit) return fail(TBK_ERR_INVALID, "wait limit above %u polls", kWaitLimit);
  g_wait_limit.store(polls < 0 ? kWaitLimit : (uint32_t)polls, std::memory_order_relaxed);
  return TBK_OK;
}

void tbk_cheb_braket_release(void) {
  std::lock_guard<std::mutex> lock(g_dropin.mu);
  g_dropin.drop();
  scratch_trim();
}

int tbk_cheb_braket_real(int32_t n_rows, int64_t nnz, const int32_t* cp, const int32_t* ri, const double* v,
                         int32_t n, const double* bras, const double* kets, int32_t R, int32_t flags,
                         double* mu_out) {
  return cheb_braket_common(n_rows, nnz, cp, ri, v, 0, n, bras, kets, R, flags, mu_out);
}

int tbk_cheb_braket_complex(int32_t n_rows, int64_t nnz, const int32_t* cp, const int32_t* ri, const double* v,
                            int32_t n, const double* bras, const double* kets, int32_t R, int32_t flags,
                            double* mu_out) {
  return cheb_braket_common(n_rows, nnz, cp, ri, v, 1, n, bras, kets, R, flags, mu_out);
}

}  // extern "C"
