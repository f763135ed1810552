// kpm_step.cuh — the one-pass recursion step kernel and its launch templates.
// Instantiated per vector precision in kpm_step_f32.cu, kpm_step_f64.cu and
// kpm_step_dd.cu (compiled in parallel); everything else calls
// launch_step_prec / occupancy_prec.
#pragma once
#include <cuda_runtime.h>

#include "kpm_device.cuh"
#include "split_store.cuh"
#include "tbk_internal.h"

namespace tbk {

constexpr int kStepThreads = 256;
constexpr int kStepWarps = kStepThreads / 32;

// Row classes of a translation-invariant matrix (EllDev::cls*): class of each
// row, and per class its entry count, column offsets (column - row) and values
// in the recursion's precision, w entries per class.
struct ClassTab {
  const uint8_t* cls = nullptr;
  const int32_t* cnt = nullptr;
  const int32_t* off = nullptr;
  const void* val = nullptr;
  const void* val2 = nullptr;   // values of a second matrix with the same columns (KST = 2)
  int32_t n_cls = 0, w = 0;
};
// shared-memory table of the class form: values, offsets, counts
template <typename F, bool CPLX_H>
constexpr int class_value_bytes() { return (CPLX_H ? 2 : 1) * (int)sizeof(F); }
// Four consecutive class values in FP32 (o a multiple of 4, as the tables' width is).
template <bool CPLX_H>
__device__ __forceinline__ void load_smem4(const float* p, int32_t o, HVal<float, CPLX_H> (&h)[4]) {
  if constexpr (CPLX_H) {
    const float4 a = reinterpret_cast<const float4*>(p)[o / 2], b = reinterpret_cast<const float4*>(p)[o / 2 + 1];
    h[0] = {a.x, a.y};
    h[1] = {a.z, a.w};
    h[2] = {b.x, b.y};
    h[3] = {b.z, b.w};
  } else {
    const float4 a = reinterpret_cast<const float4*>(p)[o / 4];
    h[0] = {a.x};
    h[1] = {a.y};
    h[2] = {a.z};
    h[3] = {a.w};
  }
}
template <typename F, bool CPLX_H>
inline size_t class_smem_bytes(const ClassTab& ct) {
  const size_t ne = (size_t)ct.n_cls * ct.w;
  return ne * class_value_bytes<F, CPLX_H>() * (ct.val2 ? 2 : 1) + ne * 4 + (size_t)ct.n_cls * 4;
}

// The moment sums of a step, part[slot][CTA].  FP64 from here on, and an FP64
// instruction holds its quarter of the SM for 64 clocks: steps without moments do no
// sums at all, braket steps after the first (kTwo false) sum one value, and two values
// share one shuffle tree (warp_pair_sum).  Against two full trees per warp and 16
// serial adds per CTA in every step: square 64x64, R = 8, FP64 braket 4.66 -> 4.06 us a
// step; honeycomb 301x253, R = 4: complex64 doubling 9.86 -> 6.77 us, FP64 doubling
// 29.2 -> 23.9 us; square 500x333 with a flux, R = 6, double-float braket 28.0 -> 23.1 us.
template <typename F, bool kTwo>
__device__ __forceinline__ void step_sums(F m0, F m1, double* __restrict__ part) {
  __shared__ double sh[2][kStepWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if constexpr (kTwo) {
    const double d = warp_pair_sum((double)m0, (double)m1);
    if ((lane & 15) == 0) sh[lane >> 4][warp] = d;
  } else {
    const double d = warp_sum((double)m0);
    if (lane == 0) sh[0][warp] = d;
  }
  __syncthreads();
  if (threadIdx.x < 2 * kStepWarps) {
    const int slot = threadIdx.x / kStepWarps;
    double d = (kTwo || slot == 0) ? sh[slot][threadIdx.x % kStepWarps] : 0.0;
#pragma unroll
    for (int o = kStepWarps / 2; o > 0; o >>= 1) d += __shfl_xor_sync((1u << 2 * kStepWarps) - 1u, d, o);
    if (threadIdx.x % kStepWarps == 0) part[slot * gridDim.x + blockIdx.x] = d;
  }
}
// Complex64 steps call it out of line, but for the brakets below: inlined, its FP64 registers change
// how the row loop is scheduled (doubling: honeycomb 701x600 with vacancies, ELL form, R = 32 122.0 ->
// 108.8 us a step; honeycomb 1024x1024, class form, R = 32 249.7 -> 239.2; braket with a flux, R = 32,
// square 900x900 185 -> 163).  The wider types run 2-6% faster with it inlined.
template <bool kTwo>
__device__ __noinline__ void step_sums_call(float m0, float m1, double* __restrict__ part) {
  step_sums<float, kTwo>(m0, m1, part);
}

// operator value o, real (vreal) or of H's type
template <typename F, bool CPLX_H>
__device__ __forceinline__ HVal<F, CPLX_H> op_value(const F* __restrict__ p, int64_t o, bool vreal) {
  if constexpr (CPLX_H) {
    if (vreal) return HVal<F, true>{HVal<F, false>::load(p, o).v, F(0)};
  }
  return HVal<F, CPLX_H>::load(p, o);
}

// the lane's values k .. into block m of a complex64 or an FP16-pair K-tiled store
template <typename F, int VPL>
__device__ __forceinline__ void store_c64(float2* __restrict__ dst, int32_t M, int32_t m, int64_t k0,
                                          const LaneV<F, VPL>& v) {
#pragma unroll
  for (int q = 0; q < VPL; ++q) {
    const int64_t k = k0 + q;
    dst[((k >> 4) * M + m) * 16 + (k & 15)] = make_float2(to_f32(v.re[q]), to_f32(v.im[q]));
  }
}
template <typename F, int VPL>
__device__ __forceinline__ void store_split(float2* __restrict__ dst, int32_t M, int32_t m, int64_t k,
                                            const LaneV<F, VPL>& v, float s, int* __restrict__ bad) {
  __half* d = reinterpret_cast<__half*>(dst);
  if constexpr (VPL == 2)
    split_put2(d, M, m, k, to_f32(v.re[0]), to_f32(v.im[0]), to_f32(v.re[1]), to_f32(v.im[1]), s, bad);
  else
    split_put(d, M, m, k, to_f32(v.re[0]), to_f32(v.im[0]), s, bad);
}

// acc += (2) p[o] x for a matrix value in memory
template <typename F, int VPL, bool CPLX_H, bool FOLD>
__device__ __forceinline__ void ell_entry(const F* __restrict__ p, int64_t o, const LaneV<F, VPL>& xs,
                                          LaneV<F, VPL>& acc) {
  const HVal<F, CPLX_H> h = HVal<F, CPLX_H>::load(p, o);
  if constexpr (FOLD) h.twice().template fma<VPL>(xs, acc);
  else h.template fma<VPL>(xs, acc);
}

// Class-form complex64 steps that feed stores or an operator product may run with up to
// kWideThreads threads per CTA.  On 3D lattices the neighbours' rows come from L2, and a
// CTA of consecutive rows shares their lines in L1: FCC 128^3 with 4 vectors has 128 rows
// to a lattice line, so that 256 threads hold one line, 768 three: a step with an FP16-pair
// store 71.6 -> 61.0 us.
template <typename F, int KST, bool CLS>
constexpr bool kWideSteps = CLS && sizeof(F) == 4 && KST != 0 && KST != 3;
template <int KST>
constexpr int kWideThreads = KST == 2 ? 512 : 768;

// Rows of more than 8 entries in the double-float class form (PIPE there)
template <typename F, int R, bool CLS>
constexpr bool kWideRows = CLS && is_dd<F> && R >= 16;
// CTAs per SM that the registers must leave room for (0: not stated).  What is best is between
// the number of warps and the gathers that each has in flight, and left to itself the compiler
// swings either way with small changes around the row loop.  us a step:
// FP64: 4 in both forms, which then keep one grid and so the same bits (honeycomb 1024x1024, R = 32,
//   braket 1,483 -> 1,364; 3 would give the class form 1,227, the ELL form 577 against 484).
// Double-float, class form: 3 (not stated, as before 60-64 registers, | 1: 88-106 | 3): honeycomb
//   512x512, R = 8, braket 48.5 | 56.3 | 50.5; 1024x1024, R = 32, doubling 791 | 753 | 737, braket 889
//   | 799 | 729; R = 4, doubling 97 | 106 | 101.  Rows of more than 8 entries, R >= 16: 1 (FCC 100^3,
//   R = 32, doubling 843 | 673 | 708).  ELL form of real matrices: 3 (FCC 64^3 with vacancies, R = 32,
//   doubling 242 not stated, 187 with 3), but for short rows of run-time widths (square 900x900 with
//   vacancies, R = 6, 60 -> 67); complex ones not stated.
// Complex64 braket: 6, which is 40 registers, where the compiler takes 32 (class form, and the ELL form
//   with few entries a row: FCC 64^3, R = 32, 61.4 -> 56; square 900x900 with a flux, R = 32, 164 -> 147, with
//   vacancies 148 -> 127), but for widths 1, 2 and run-time ones (flux, R = 2, 11.3 -> 14.4 with it).
template <typename F, int R, bool CPLX_H, bool BRAKET, int KST, bool PIPE, bool CLS>
constexpr int min_ctas() {
  if (kWideSteps<F, KST, CLS>) return 2;
  if (is_f64<F>) return 4;
  if (KST != 0) return 0;
  if (is_dd<F>) return CLS ? (PIPE ? 1 : 3) : CPLX_H || (R == 0 && !PIPE) ? 0 : 3;
  if (BRAKET) return CLS || (!PIPE && R >= 4) ? 6 : 0;
  return 0;
}

// One recursion step over all rows, x = v_s, y = v_{s-1} on entry.
//   FIRST: y = H x                    else: y = 2 H x - y  (v_{s+1} over v_{s-1})
//   doubling (BRAKET false): part[0] += <x|x>; part[1] += <x|y_in> (= <v_s|v_{s-1}>),
//                            FIRST: part[1] += <x|H x> (= <v_0|v_1>)
//   braket:                  part[0] += <b|v_{s+1}>;  FIRST also part[1] += <b|x>
//   gather == 0: no product at all (the last doubling step only needs the dots).
//   KST: 3 = add c v to the output (a Clenshaw step of a Chebyshev expansion,
//   ks.addc / ks.addv); otherwise also write complex64 K-tiled stores (Kubo
//   blocks, KStore): 1 = the output into one store; 2 = per column group the
//   output or V x for an
//   operator V with H's ELL structure, formed from the same gathered x (the
//   operator product of the previous block fused into the step), so that the
//   two sides of a Kubo pair can run as one recursion of twice the width.  A
//   template parameter because even an untaken runtime branch there costs the
//   moments recursion ~8% of its bandwidth.
//   KST = 5: as 1, into an FP16-pair store (ks.split; KST = 2 looks at it itself).
//   KST = 4: a plain step whose moments nothing reads (the Kubo recursion
//   ahead of an operator product).  Only KST = 0 forms the moment sums.
//   PIPE (of the ELL form; see kWideRows): rows wider than one group of 4 gathers (ELL width > 4, e.g. FCC's
//   12 neighbours) load the next group's columns while this group's gathers
//   are in flight: 4 dependent memory round trips per 12-neighbour row instead
//   of 6 (1.8x on the FCC Kubo recursion).  Narrow rows keep the plain loop,
//   whose extra predicated loads would cost the honeycomb recursion 8%.
//   CLS: rows of a translation-invariant matrix come in a few classes (ct);
//   each neighbour is row + offset from the class table in shared memory and
//   its value comes from there too, so no column index or value is loaded and
//   the only index read (the row's class byte) is issued one grid-stride
//   iteration ahead.  Same entries in the same order as the ELL: the same sums.
//   R: vectors per row, a power of two; 0: any other width, LPR lanes per row given
//   at run time (rows stay whole within a CTA, a few threads at its end idle).
template <typename F, int R, bool CPLX_H, bool FIRST, bool BRAKET, int KST = 0, bool PIPE = false, bool CLS = false>
__global__ void __launch_bounds__(kWideSteps<F, KST, CLS> ? kWideThreads<KST> : kStepThreads, min_ctas<F, R, CPLX_H, BRAKET, KST, PIPE, CLS>())
kpm_step_kernel(
    int32_t n, int32_t n_tiles, const int32_t* __restrict__ soff, const int32_t* __restrict__ ecol,
    const F* __restrict__ eval, const F* __restrict__ diag, const typename C2<F>::T* __restrict__ x,
    typename C2<F>::T* y, const typename C2<F>::T* pv, const typename C2<F>::T* __restrict__ bras,
    double* __restrict__ part, int store, int reverse, int gather, int pf_dist, const KStore ks, const ClassTab ct, int32_t lpr) {
  using CT = typename C2<F>::T;
  constexpr int VPL = (R == 0 || R >= VecW<F>::max_vpl) ? VecW<F>::max_vpl : 1;
  static_assert(R == 0 || (R / VPL >= 1 && R / VPL <= 32 && (32 % (R / VPL)) == 0), "R out of range");
  const int LPR = R > 0 ? R / VPL : lpr;   // lanes per row
  const int RW = LPR * VPL;                // vectors per row
  const int ROWS_PER_TILE = (kWideSteps<F, KST, CLS> ? (int)blockDim.x : kStepThreads) / LPR;
  const int trow = threadIdx.x / LPR;      // this thread's row in a tile (none: past n)
  const bool idle = R == 0 && trow >= ROWS_PER_TILE;
  using Acc = F;                           // per-thread sums in the vector precision

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = threadIdx.x % LPR;
  Acc m0 = 0, m1 = 0;
  constexpr bool FOLD = kFoldStep<F> && !FIRST;
  static_assert(!(CLS && KST == 2 && sizeof(F) != 4), "class form: operator products in FP32 only");

  // class form: the table in shared memory (4-byte words: values, offsets, counts)
  extern __shared__ __align__(16) unsigned char cls_smem[];
  const F* s_val = reinterpret_cast<const F*>(cls_smem);
  const F* s_val2 = nullptr;               // the operator's values (KST = 2)
  const int32_t* s_off = nullptr;
  const int32_t* s_cnt = nullptr;
  uint32_t c_next = 0;                     // class of this thread's row in the next iteration
  if constexpr (CLS) {
    const int32_t ne = ct.n_cls * ct.w;
    const int32_t v1 = ne * (class_value_bytes<F, CPLX_H>() / 4), vw = KST == 2 ? 2 * v1 : v1;
    uint32_t* sw = reinterpret_cast<uint32_t*>(cls_smem);
    const uint32_t* gv = static_cast<const uint32_t*>(ct.val);
    if constexpr (FOLD) {
      F* dv = reinterpret_cast<F*>(cls_smem);
      for (int32_t q = threadIdx.x; q < ne * (CPLX_H ? 2 : 1); q += blockDim.x)
        dv[q] = times2(static_cast<const F*>(ct.val)[q]);
    } else {
      for (int32_t q = threadIdx.x; q < v1; q += blockDim.x) sw[q] = gv[q];
    }
    if constexpr (KST == 2) {
      const uint32_t* gw = static_cast<const uint32_t*>(ct.val2);
      for (int32_t q = threadIdx.x; q < v1; q += blockDim.x) sw[v1 + q] = gw[q];
      s_val2 = reinterpret_cast<const F*>(sw + v1);
    }
    for (int32_t q = threadIdx.x; q < ne; q += blockDim.x) sw[vw + q] = (uint32_t)ct.off[q];
    for (int32_t q = threadIdx.x; q < ct.n_cls; q += blockDim.x) sw[vw + ne + q] = (uint32_t)ct.cnt[q];
    s_off = reinterpret_cast<const int32_t*>(sw + vw);
    s_cnt = reinterpret_cast<const int32_t*>(sw + vw + ne);
    __syncthreads();
    const int32_t t0 = blockIdx.x;
    if (t0 < n_tiles) {
      const int32_t r0 = (reverse ? (n_tiles - 1 - t0) : t0) * ROWS_PER_TILE + trow;
      if (r0 < n && !idle) c_next = __ldg(ct.cls + r0);
    }
  }

  float scale0 = 1.f, scale1 = 1.f;        // of FP16-pair stores
  if constexpr (KST == 5 || KST == 2) {
    if (ks.split) {
      scale0 = __ldg(ks.scale[0]);
      if (KST == 2 && ks.halves == 2) scale1 = __ldg(ks.scale[1]);
    }
  }
  HVal<F, true> add_c{F(0), F(0)};         // c_k of a Clenshaw step
  if constexpr (KST == 3) {
    const double f = is_dd<F> ? 0.5 : 1.0;
    add_c = HVal<F, true>{F(f * ks.addc[0]), F(f * ks.addc[1])};
  }

  const CT* xl = x + sub * VPL;            // this lane's column of x
  const uint32_t row_bytes = (uint32_t)(RW * sizeof(CT));
  auto nb = [&](uint32_t c) { return ld_row<F, VPL>(xl, c, row_bytes); };
  // rows are verified equal to their class, so r + offset is the row's column; the clamp only
  // keeps a bad table inside the block
  auto clamp = [&](int32_t c) { return min((uint32_t)c, (uint32_t)(n - 1)); };
  for (int32_t t = blockIdx.x; t < n_tiles; t += gridDim.x) {
    const uint32_t c_cur = c_next;
    if constexpr (CLS) {
      const int32_t tn = t + (int32_t)gridDim.x;
      c_next = 0;
      if (tn < n_tiles) {
        const int32_t rn = (reverse ? (n_tiles - 1 - tn) : tn) * ROWS_PER_TILE + trow;
        if (rn < n && !idle) c_next = __ldg(ct.cls + rn);
      }
    }
    const int32_t tile = reverse ? (n_tiles - 1 - t) : t;
    if (pf_dist > 0 && threadIdx.x == 0) {
      // bring the streams of the tile this CTA reaches pf_dist iterations later
      // into L2 ahead of time: its own rows of v_n and v_{n-1} (and the bras)
      const int32_t tf = t + pf_dist * (int32_t)gridDim.x;
      if (tf < n_tiles) {
        const int32_t tilef = reverse ? (n_tiles - 1 - tf) : tf;
        const int64_t rf = (int64_t)tilef * ROWS_PER_TILE;
        const int32_t nr = (int32_t)min((int64_t)ROWS_PER_TILE, (int64_t)n - rf);
        if (nr > 0) {
          const uint32_t vb = (uint32_t)nr * (uint32_t)(RW * sizeof(CT));
          if ((vb & 15u) == 0) {
            bulk_prefetch_l2(x + rf * RW, vb);
            if (!FIRST) bulk_prefetch_l2(pv + rf * RW, vb);
            if (BRAKET) bulk_prefetch_l2(bras + rf * RW, vb);
          }
          if constexpr (!CLS) {
            if (gather) {
              // and the ELL columns and values of its slices, so that the rows'
              // column loads find them in L2 (slice offsets are whole 32-entry
              // columns: 128-byte aligned, whole 128-byte multiples)
              constexpr uint32_t VB = (CPLX_H ? 2u : 1u) * (uint32_t)sizeof(F);
              const int32_t s0 = (int32_t)(rf >> 5), s1 = (int32_t)((rf + nr - 1) >> 5);
              const int32_t o0 = soff[s0], o1 = soff[s1 + 1];
              if (o1 > o0) {
                bulk_prefetch_l2(ecol + o0, (uint32_t)(o1 - o0) * 4u);
                bulk_prefetch_l2(reinterpret_cast<const char*>(eval) + (int64_t)o0 * VB, (uint32_t)(o1 - o0) * VB);
              }
            }
          }
        }
      }
    }
    const int32_t r = tile * ROWS_PER_TILE + trow;
    if (r >= n || idle) continue;
    const int64_t me = (int64_t)r * LPR + sub;
    const LaneV<F, VPL> xs = ld_ro<F, VPL>(x + me * VPL);
    LaneV<F, VPL> prev;
    if constexpr (!FIRST) prev = ld_stream<F, VPL>(pv + me * VPL);   // pv == y: in place
    LaneV<F, VPL> acc, vacc;
#pragma unroll
    for (int q = 0; q < VPL; ++q) {
      if constexpr (FOLD) { acc.re[q] = negate(prev.re[q]); acc.im[q] = negate(prev.im[q]); }
      else { acc.re[q] = 0; acc.im[q] = 0; }
    }
    // column group of this lane (its VPL columns never straddle two groups)
    const int grp = (KST == 2 && ks.halves == 2 && sub * VPL >= RW / 2) ? 1 : 0;
    const F* vval = nullptr;
    const F* vdiag = nullptr;
    bool vreal = false;
    if constexpr (KST == 2) {
      vreal = CPLX_H && (grp ? ks.vreal[1] : ks.vreal[0]) != 0;
      const void* vv = grp ? ks.vval[1] : ks.vval[0];      // selects, not an indexed parameter array
      const void* vd = grp ? ks.vdiag[1] : ks.vdiag[0];
      vval = vv ? static_cast<const F*>(vv) : eval;
      vdiag = vd ? static_cast<const F*>(vd) : diag;
#pragma unroll
      for (int q = 0; q < VPL; ++q) { vacc.re[q] = 0; vacc.im[q] = 0; }
    }
    if (gather && CLS) {
      ell_entry<F, VPL, CPLX_H, FOLD>(diag, r, xs, acc);
      if constexpr (KST == 2) HVal<F, CPLX_H>::load(vdiag, r).template fma<VPL>(xs, vacc);
      const int32_t cnt = s_cnt[c_cur];
      const int32_t tb = (int32_t)c_cur * ct.w;
      // a class's tail entries up to the table width (a multiple of 4) are
      // (offset 0, value 0): 0 x (own row), exactly what a predicated-off entry
      // adds.  FP32 vectors take whole groups without predicates (fewer
      // instructions and registers); the wider types keep the predicates,
      // whose unconditional form holds more gathers in registers
      constexpr bool WHOLE = sizeof(F) == 4;
      // the table read four entries at a time where the launch bound leaves registers
      // for it (FCC 64^3 Kubo blocks 8.8 -> 8.1 us; the moments step spills: honeycomb
      // 1024^2, R = 32: 242 -> 277)
      constexpr bool VEC = CLS && KST == 2;
      int k0 = 0;
      if constexpr (is_f64<F>) {
        // FP64: whole groups, then single entries (a predicated product still
        // takes its turn on the FP64 pipe)
        for (; k0 + 4 <= cnt; k0 += 4) {
          LaneV<F, VPL> xv[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            xv[u] = nb(clamp(r + s_off[tb + k0 + u]));
#pragma unroll
          for (int u = 0; u < 4; ++u) HVal<F, CPLX_H>::load_smem(s_val, tb + k0 + u).template fma<VPL>(xv[u], acc);
        }
#pragma unroll 1
        for (; k0 < cnt; ++k0)
          HVal<F, CPLX_H>::load_smem(s_val, tb + k0).template fma<VPL>(nb(clamp(r + s_off[tb + k0])), acc);
      }
      for (int k = k0; k < cnt; k += 4) {
        HVal<F, CPLX_H> h[4];
        LaneV<F, VPL> xv[4];
        if constexpr (VEC) {
          const int4 o = *reinterpret_cast<const int4*>(s_off + tb + k);
          xv[0] = nb(clamp(r + o.x));
          xv[1] = nb(clamp(r + o.y));
          xv[2] = nb(clamp(r + o.z));
          xv[3] = nb(clamp(r + o.w));
          load_smem4<CPLX_H>(s_val, tb + k, h);
        } else if constexpr (WHOLE) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            h[u] = HVal<F, CPLX_H>::load_smem(s_val, tb + k + u);
            xv[u] = nb(clamp(r + s_off[tb + k + u]));
          }
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const bool v = k + u < cnt;
            h[u] = v ? HVal<F, CPLX_H>::load_smem(s_val, tb + k + u) : HVal<F, CPLX_H>::zero();
            xv[u] = v ? ld_ro<F, VPL>(x + ((int64_t)clamp(r + s_off[tb + k + u]) * LPR + sub) * VPL) : xs;
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) h[u].template fma<VPL>(xv[u], acc);
        if constexpr (VEC) {
          load_smem4<CPLX_H>(s_val2, tb + k, h);
#pragma unroll
          for (int u = 0; u < 4; ++u) h[u].template fma<VPL>(xv[u], vacc);
        }
      }
    } else if (gather) {
      ell_entry<F, VPL, CPLX_H, FOLD>(diag, r, xs, acc);
      if constexpr (KST == 2) op_value<F, CPLX_H>(vdiag, r, vreal).template fma<VPL>(xs, vacc);
      const int32_t s = r >> 5, l = r & 31;
      const int32_t off = soff[s];
      const int32_t w = (soff[s + 1] - off) >> 5;
      const int32_t* cp = ecol + off + l;
      int32_t cn[4];
      if constexpr (PIPE && !(is_f64<F> && KST != 2)) {
#pragma unroll
        for (int u = 0; u < 4; ++u) cn[u] = u < w ? __ldg(cp + u * 32) : r;
      }
      int k0 = 0;
      if constexpr (is_f64<F> && KST != 2) {                        // as in the class form
        for (; k0 + 4 <= w; k0 += 4) {
          LaneV<F, VPL> xv[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            xv[u] = nb(__ldg(cp + (k0 + u) * 32));
#pragma unroll
          for (int u = 0; u < 4; ++u)
            ell_entry<F, VPL, CPLX_H, FOLD>(eval, off + l + (int64_t)(k0 + u) * 32, xv[u], acc);
        }
#pragma unroll 1
        for (; k0 < w; ++k0)
          ell_entry<F, VPL, CPLX_H, FOLD>(eval, off + l + (int64_t)k0 * 32,
                                          nb(__ldg(cp + k0 * 32)), acc);
      }
      // all of a row's gathers in flight together: predicated groups of 4
      for (int k = k0; k < w; k += 4) {
        int32_t c[4];
        HVal<F, CPLX_H> h[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const bool v = k + u < w;
          if constexpr (PIPE) c[u] = cn[u];
          else c[u] = v ? __ldg(cp + (k + u) * 32) : r;             // padding: own row
          h[u] = v ? HVal<F, CPLX_H>::load(eval, off + l + (int64_t)(k + u) * 32) : HVal<F, CPLX_H>::zero();
        }
        if constexpr (PIPE) {                                       // next group's columns
#pragma unroll
          for (int u = 0; u < 4; ++u) cn[u] = k + 4 + u < w ? __ldg(cp + (k + 4 + u) * 32) : r;
        }
        LaneV<F, VPL> xv[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          // complex FP32 values: square 700x512 with a flux, R = 4: 9.4 us a step, 10.1 by rows
          if constexpr (CPLX_H && sizeof(F) == 4 && KST == 0 && R > 0) xv[u] = ld_ro<F, VPL>(x + ((int64_t)c[u] * LPR + sub) * VPL);
          else xv[u] = nb(c[u]);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if constexpr (FOLD) {
            h[u].twice().template fma<VPL>(xv[u], acc);
          } else {
            h[u].template fma<VPL>(xv[u], acc);
          }
        }
        if constexpr (KST == 2) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const HVal<F, CPLX_H> hv = k + u < w ? op_value<F, CPLX_H>(vval, off + l + (int64_t)(k + u) * 32, vreal)
                                                 : HVal<F, CPLX_H>::zero();
            hv.template fma<VPL>(xv[u], vacc);
          }
        }
      }
    }
    if constexpr (KST == 3 && sizeof(F) == 8) {
      // Clenshaw step of a Chebyshev expansion: b_k = 2 H b_{k+1} - b_{k+2} + c_k v, the
      // last term summed with the row's (add_c = c_k / 2 where the sum is doubled after)
      add_c.template fma<VPL>(ld_ro<F, VPL>(static_cast<const CT*>(ks.addv) + me * VPL), acc);
    }
    finish_acc<F, VPL>(acc);
    if constexpr (KST == 2) finish_acc<F, VPL>(vacc);
    LaneV<F, VPL> out;
    if constexpr (FIRST || FOLD) out = acc;
    else recur_out<F, VPL>(acc, prev, out);
    if constexpr (KST == 3 && sizeof(F) == 4) {
      const LaneV<F, VPL> vv = ld_ro<F, VPL>(static_cast<const CT*>(ks.addv) + me * VPL);
#pragma unroll
      for (int q = 0; q < VPL; ++q) {
        out.re[q] = out.re[q] + (add_c.r * vv.re[q] - add_c.i * vv.im[q]);
        out.im[q] = out.im[q] + (add_c.r * vv.im[q] + add_c.i * vv.re[q]);
      }
    }
    // moment partial sums (before the store, from registers only); steps that
    // feed stores, expansions or an operator product need none
    if constexpr (KST != 0) {
    } else if constexpr (BRAKET) {
      const LaneV<F, VPL> b = ld_ro<F, VPL>(bras + me * VPL);
      dot_acc<F, VPL>(b, out, m0);
      if constexpr (FIRST) dot_acc<F, VPL>(b, xs, m1);
    } else {
      dot_acc<F, VPL>(xs, xs, m0);
      if constexpr (FIRST) dot_acc<F, VPL>(xs, out, m1);
      else dot_acc<F, VPL>(xs, prev, m1);
    }
    if (store) st_v<F, VPL>(y + me * VPL, out);
    if constexpr (KST == 1) {
      // block km[0] of the K-tiled store: one rounding per value
      store_c64<F, VPL>(ks.store[0], ks.kM, ks.km[0], (int64_t)r * RW + sub * VPL, out);
    } else if constexpr (KST == 5) {
      store_split<F, VPL>(ks.store[0], ks.kM, ks.km[0], (int64_t)r * RW + sub * VPL, out, scale0, ks.bad);
    } else if constexpr (KST == 2) {
      const int32_t kmg = grp ? ks.km[1] : ks.km[0];
      if (kmg >= 0) {
        const int32_t Rg = RW / ks.halves;
        const LaneV<F, VPL>& sv = (grp ? ks.usev[1] : ks.usev[0]) ? vacc : out;
        float2* dst = grp ? ks.store[1] : ks.store[0];
        const int64_t k = (int64_t)r * Rg + sub * VPL - grp * Rg;
        if (ks.split) store_split<F, VPL>(dst, ks.kM, kmg, k, sv, grp ? scale1 : scale0, ks.bad);
        else store_c64<F, VPL>(dst, ks.kM, kmg, k, sv);
      }
    }
  }
  if constexpr (KST == 0) {
    if constexpr (sizeof(F) == 4 && !(BRAKET && (CLS || (!CPLX_H && !PIPE && R >= 4)))) step_sums_call<!BRAKET || FIRST>(m0, m1, part);
    else step_sums<F, !BRAKET || FIRST>(m0, m1, part);
  }
}


// ----------------------------------------------------------------- dispatch
struct StepArgs {
  int32_t n, n_tiles, n_slices;
  int* err;
  const int32_t* soff;
  const int32_t* ecol;
  const void* eval;
  const void* diag;
  const void* x;
  void* y;
  const void* pv;      // v_{n-1}; equal to y for the in-place recursion
  const void* bras;
  double* part;
  int store, reverse, gather, pf_dist;
  KStore ks;                   // optional complex64 K-tiled stores (Kubo blocks)
  int kst = 0;                 // 0 moments, 1 output into ks.store[0], 2 per-group output / V x,
                               // 3 Clenshaw term, 4 plain step without moment sums, 5 as 1 in FP16 pairs
  bool pipe = false;           // ELL wider than 4: pipelined column loads
  bool cls = false;            // row classes (ct) instead of the ELL's columns and values
  ClassTab ct;
  int32_t threads = kStepThreads;   // per CTA (class-form complex64 steps without sums)
  int32_t lpr = 0;             // lanes per row of a width without its own instantiation (R = 0)
};

template <typename F, int R, bool CPLX_H, bool CLS>
inline int launch_step_r(const StepArgs& a, bool first, bool braket, int grid, cudaStream_t st) {
  using CT = typename C2<F>::T;
  const size_t smem = CLS ? class_smem_bytes<F, CPLX_H>(a.ct) : 0;
  auto x = static_cast<const CT*>(a.x);
  auto y = static_cast<CT*>(a.y);
  auto pv = static_cast<const CT*>(a.pv ? a.pv : a.y);
  auto b = static_cast<const CT*>(a.bras);
  auto ev = static_cast<const F*>(a.eval);
  auto dg = static_cast<const F*>(a.diag);
#define TBK_STEP(FI, BR, KS)                                                                          \
  do {                                                                                                \
    if constexpr (kWideRows<F, R, CLS> && KS == 0 && !FI) {                                           \
      if (a.ct.w > 8) {                                                                               \
        kpm_step_kernel<F, R, CPLX_H, FI, BR, KS, true, true><<<grid, kStepThreads, smem, st>>>(      \
            a.n, a.n_tiles, a.soff, a.ecol, ev, dg, x, y, pv, b, a.part, a.store, a.reverse, a.gather, a.pf_dist, a.ks, \
            a.ct, a.lpr);                                                                             \
        break;                                                                                        \
      }                                                                                               \
    }                                                                                                 \
    if constexpr (CLS)                                                                                \
      kpm_step_kernel<F, R, CPLX_H, FI, BR, KS, false, true><<<grid, kWideSteps<F, KS, true> ? a.threads : kStepThreads, smem, st>>>( \
          a.n, a.n_tiles, a.soff, a.ecol, ev, dg, x, y, pv, b, a.part, a.store, a.reverse, a.gather, a.pf_dist, a.ks, \
          a.ct, a.lpr);                                                                                      \
    else if (a.pipe)                                                                                  \
      kpm_step_kernel<F, R, CPLX_H, FI, BR, KS, true><<<grid, kStepThreads, 0, st>>>(                 \
          a.n, a.n_tiles, a.soff, a.ecol, ev, dg, x, y, pv, b, a.part, a.store, a.reverse, a.gather, a.pf_dist, a.ks, \
          a.ct, a.lpr);                                                                                      \
    else                                                                                              \
      kpm_step_kernel<F, R, CPLX_H, FI, BR, KS, false><<<grid, kStepThreads, 0, st>>>(                \
          a.n, a.n_tiles, a.soff, a.ecol, ev, dg, x, y, pv, b, a.part, a.store, a.reverse, a.gather, a.pf_dist, a.ks, \
          a.ct, a.lpr);                                                                                      \
  } while (0)
  if (a.kst != 0) {
    if (braket) return fail(TBK_ERR_UNSUPPORTED, "K-tiled store with a braket step");
    constexpr int VPLR = (R == 0 || R >= VecW<F>::max_vpl) ? VecW<F>::max_vpl : 1;
    const int rw = R > 0 ? R : a.lpr * VPLR;
    if (a.kst == 2 && a.ks.halves == 2 && (rw / 2) % VPLR != 0)
      return fail(TBK_ERR_UNSUPPORTED, "column groups narrower than a lane's vectors");
    if (a.kst == 3) {
      if (first) return fail(TBK_ERR_UNSUPPORTED, "Clenshaw term on a first step");
      TBK_STEP(false, false, 3);
    } else if (a.kst == 4) {
      if (first) TBK_STEP(true, false, 4); else TBK_STEP(false, false, 4);
    } else if (a.kst == 5) {
      if (first) TBK_STEP(true, false, 5); else TBK_STEP(false, false, 5);
    } else if (a.kst == 2) {
      if constexpr (CLS && sizeof(F) != 4) {
        return fail(TBK_ERR_UNSUPPORTED, "operator products in the class form are complex64");
      } else {
        if (CLS && !a.ct.val2) return fail(TBK_ERR_UNSUPPORTED, "operator product without its class values");
        if (first) TBK_STEP(true, false, 2); else TBK_STEP(false, false, 2);
      }
    }
    else { if (first) TBK_STEP(true, false, 1); else TBK_STEP(false, false, 1); }
  } else if (first) { if (braket) TBK_STEP(true, true, 0); else TBK_STEP(true, false, 0); }
  else { if (braket) TBK_STEP(false, true, 0); else TBK_STEP(false, false, 0); }
#undef TBK_STEP
  TBK_CHECK_LAUNCH();
  return TBK_OK;
}

template <typename F, bool CPLX_H, bool CLS = false>
inline int launch_step(int R, const StepArgs& a, bool first, bool braket, int grid, cudaStream_t st) {
  switch (R) {
    case 1: return launch_step_r<F, 1, CPLX_H, CLS>(a, first, braket, grid, st);
    case 2: return launch_step_r<F, 2, CPLX_H, CLS>(a, first, braket, grid, st);
    case 4: return launch_step_r<F, 4, CPLX_H, CLS>(a, first, braket, grid, st);
    case 8: return launch_step_r<F, 8, CPLX_H, CLS>(a, first, braket, grid, st);
    case 16: return launch_step_r<F, 16, CPLX_H, CLS>(a, first, braket, grid, st);
    case 32: return launch_step_r<F, 32, CPLX_H, CLS>(a, first, braket, grid, st);
    case 64:
      if constexpr (sizeof(F) == 4) return launch_step_r<F, 64, CPLX_H, CLS>(a, first, braket, grid, st);
      break;
  }
  if (R > 0 && R < 64 && R % VecW<F>::max_vpl == 0) {
    StepArgs b = a;
    b.lpr = R / VecW<F>::max_vpl;
    return launch_step_r<F, 0, CPLX_H, CLS>(b, first, braket, grid, st);
  }
  return fail(TBK_ERR_UNSUPPORTED, "chunk width %d not instantiated", R);
}


// of the steps that form moment sums or not; in rows of more than 8 entries
struct StepKind { bool sums = false, wide = false; };
// threads: of a wide step (kWideSteps)
template <typename F, bool CPLX_H, int R, bool CLS = false>
inline int occupancy_blocks(size_t smem, StepKind kind, int threads = kStepThreads) {
  int nb = 0;
  if (kind.sums && kind.wide && kWideRows<F, R, CLS>)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &nb, kpm_step_kernel<F, R, CPLX_H, false, false, 0, kWideRows<F, R, CLS>, CLS>, kStepThreads, smem);
  else if (kind.sums)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kpm_step_kernel<F, R, CPLX_H, false, false, 0, false, CLS>,
                                                  kStepThreads, smem);
  else
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kpm_step_kernel<F, R, CPLX_H, false, false, 4, false, CLS>,
                                                  threads, smem);
  return nb > 0 ? nb : 1;
}

template <typename F, bool CLS>
inline int occupancy_r(bool cplx, int R, size_t smem, StepKind kind, int threads = kStepThreads) {
  switch (R) {
    case 1: return cplx ? occupancy_blocks<F, true, 1, CLS>(smem, kind, threads) : occupancy_blocks<F, false, 1, CLS>(smem, kind, threads);
    case 2: return cplx ? occupancy_blocks<F, true, 2, CLS>(smem, kind, threads) : occupancy_blocks<F, false, 2, CLS>(smem, kind, threads);
    case 4: return cplx ? occupancy_blocks<F, true, 4, CLS>(smem, kind, threads) : occupancy_blocks<F, false, 4, CLS>(smem, kind, threads);
    case 8: return cplx ? occupancy_blocks<F, true, 8, CLS>(smem, kind, threads) : occupancy_blocks<F, false, 8, CLS>(smem, kind, threads);
    case 16: return cplx ? occupancy_blocks<F, true, 16, CLS>(smem, kind, threads) : occupancy_blocks<F, false, 16, CLS>(smem, kind, threads);
    case 32: case 64: return cplx ? occupancy_blocks<F, true, 32, CLS>(smem, kind, threads) : occupancy_blocks<F, false, 32, CLS>(smem, kind, threads);
    default: return cplx ? occupancy_blocks<F, true, 0, CLS>(smem, kind, threads) : occupancy_blocks<F, false, 0, CLS>(smem, kind, threads);
  }
}

// per-precision entry points (TBK_PREC_*); a.cls selects the class form
int launch_step_prec(int prec, bool cplx, int R, const StepArgs& a, bool first, bool braket, int grid,
                     cudaStream_t st);
// CTAs per SM
int occupancy_prec(int prec, bool cplx, int R, StepKind kind);
// the same of the class-form kernel with its shared-memory table
int occupancy_cls_prec(int prec, bool cplx, int R, size_t smem, StepKind kind, int threads = kStepThreads);
// whether a matrix runs in the class form in a precision
bool has_classes(const EllDev& E, int prec);
// the class table of a matrix in a precision (ct.n_cls == 0: no class form)
ClassTab class_tab(const EllDev& E, int prec);
size_t class_smem(const EllDev& E, int prec);

}  // namespace tbk
