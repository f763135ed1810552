// kpm_persist.cuh — a whole small recursion in one cooperative launch.
//
// Vectors of at most one 256-thread tile per resident CTA: every thread keeps its own
// elements of v_s, v_{s-1} and the bras, its diagonal and its row class in registers, the
// class table stays in shared memory, and a step reads only the neighbours' elements
// (through L2, where the other CTAs wrote them) and writes v_{s+1}.  Between steps the CTAs
// meet at a counter in global memory; the step's moment sums run between a CTA's
// arrival and its wait.  The arithmetic, its order and the partial sums are those of
// kpm_step_kernel with one tile per CTA: the same bits.  (That sweeps odd steps from the last
// tile to the first, so its CTA b has the sums of the last tile but b: the reduction reads these
// backwards.)
// What bounds a step: the L2 round trip of the gathers, the FP64 pipe and the meeting.
// us a step against one launch per step (graph replay): square 64x64, R = 8, braket FP64
// 3.99 -> 2.52, double-float 3.78 -> 2.65, complex64 3.65 -> 2.28; 170x160, R = 8, complex64
// 4.51 -> 2.83; with one tile per CTA and four CTAs per SM in FP64 (128x128, R = 8, at the
// end of its range) 7.23 -> 6.21.
// The waits are bounded (wait_limit polls): a CTA that gives up records an error, and
// all leave.
#pragma once
#include <cuda_runtime.h>

#include "kpm_device.cuh"
#include "kpm_step.cuh"

namespace tbk {

constexpr int kErrMeet = 0x400;

template <typename F, int VPL>
__device__ __forceinline__ LaneV<F, VPL> ld_cg(const typename C2<F>::T* p) {
  LaneV<F, VPL> o;
  if constexpr (is_dd<F>) {
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      const float4 q = __ldcg(reinterpret_cast<const float4*>(p) + v);
      o.re[v] = dd(q.x, q.y); o.im[v] = dd(q.z, q.w);
    }
  } else if constexpr (sizeof(F) == 4 && VPL == 2) {
    const float4 q = __ldcg(reinterpret_cast<const float4*>(p));
    o.re[0] = q.x; o.im[0] = q.y; o.re[1] = q.z; o.im[1] = q.w;
  } else {
    const auto q = __ldcg(p);
    o.re[0] = q.x; o.im[0] = q.y;
  }
  return o;
}

// acc += sum of h_k x_k over one row's entries, value(k) and neighbour(k) giving them, in the
// groups and order of kpm_step_kernel
template <typename F, int VPL, bool CPLX_H, typename Val, typename Nb>
__device__ __forceinline__ void row_entries(int cnt, LaneV<F, VPL>& acc, const LaneV<F, VPL>& own, Val&& value,
                                            Nb&& neighbour) {
  int k = 0;
  if constexpr (is_f64<F>) {
    for (; k + 4 <= cnt; k += 4) {
      LaneV<F, VPL> xv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) xv[u] = neighbour(k + u);
#pragma unroll
      for (int u = 0; u < 4; ++u) value(k + u).template fma<VPL>(xv[u], acc);
    }
#pragma unroll 1
    for (; k < cnt; ++k) value(k).template fma<VPL>(neighbour(k), acc);
  } else {
    for (; k < cnt; k += 4) {
      LaneV<F, VPL> xv[4];
      HVal<F, CPLX_H> h[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool v = k + u < cnt;
        h[u] = v ? value(k + u) : HVal<F, CPLX_H>::zero();
        xv[u] = v ? neighbour(k + u) : own;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) h[u].template fma<VPL>(xv[u], acc);
    }
  }
}

template <typename F, bool CPLX_H, bool BRAKET, bool CLS>
__global__ void __launch_bounds__(kStepThreads) kpm_persist_kernel(
    int32_t n, int32_t n_steps, int32_t lpr, const int32_t* __restrict__ soff, const int32_t* __restrict__ ecol,
    const F* __restrict__ eval, const F* __restrict__ diag, const ClassTab ct, typename C2<F>::T* va,
    typename C2<F>::T* vb, const typename C2<F>::T* __restrict__ bras, double* __restrict__ part,
    unsigned int* __restrict__ meet, int* __restrict__ err, uint32_t wait_limit) {
  using CT = typename C2<F>::T;
  using HV = HVal<F, CPLX_H>;
  constexpr int VPL = VecW<F>::max_vpl;
  constexpr bool FOLD = kFoldStep<F>;
  extern __shared__ __align__(16) unsigned char ps_smem[];
  __shared__ int gave_up;
  F* s_val = reinterpret_cast<F*>(ps_smem);
  const int32_t ne = CLS ? ct.n_cls * ct.w : 0, nv = ne * (CPLX_H ? 2 : 1);
  int32_t* s_off = reinterpret_cast<int32_t*>(ps_smem + (size_t)nv * sizeof(F));
  int32_t* s_cnt = s_off + ne;
  if constexpr (CLS) {
    for (int32_t q = threadIdx.x; q < nv; q += kStepThreads) s_val[q] = static_cast<const F*>(ct.val)[q];
    for (int32_t q = threadIdx.x; q < ne; q += kStepThreads) s_off[q] = ct.off[q];
    for (int32_t q = threadIdx.x; q < ct.n_cls; q += kStepThreads) s_cnt[q] = ct.cnt[q];
  }
  if (threadIdx.x == 0) gave_up = 0;
  __syncthreads();

  const int rows = kStepThreads / lpr, trow = threadIdx.x / lpr, sub = threadIdx.x % lpr;
  const int32_t r = blockIdx.x * rows + trow;
  const bool act = trow < rows && r < n;
  const int64_t me = act ? ((int64_t)r * lpr + sub) * VPL : 0;
  LaneV<F, VPL> xs{}, prev{}, b{}, out{};
  HV hd = HV::zero();
  int32_t tb = 0, cnt = 0;
  int64_t eb = 0;
  if (act) {
    xs = ld_cg<F, VPL>(va + me);
    if constexpr (BRAKET) b = ld_cg<F, VPL>(bras + me);
    hd = HV::load(diag, r);
    if constexpr (CLS) {
      const int32_t c = ct.cls[r];
      tb = c * ct.w;
      cnt = s_cnt[c];
    } else {
      const int32_t o = soff[r >> 5];
      cnt = (soff[(r >> 5) + 1] - o) >> 5;
      eb = (int64_t)o + (r & 31);
    }
  }
  for (int32_t s = 0; s < n_steps; ++s) {
    const CT* x = (s & 1) ? vb : va;
    CT* y = (s & 1) ? va : vb;
    const bool first = s == 0, dots_only = !BRAKET && s == n_steps - 1 && s > 0;
    F m0 = 0, m1 = 0;
    if (act) {
      if (!dots_only) {
        LaneV<F, VPL> acc;
#pragma unroll
        for (int q = 0; q < VPL; ++q) {
          if constexpr (FOLD) {
            acc.re[q] = first ? 0 : negate(prev.re[q]);
            acc.im[q] = first ? 0 : negate(prev.im[q]);
          } else {
            acc.re[q] = 0;
            acc.im[q] = 0;
          }
        }
        hd.template fma<VPL>(xs, acc);                       // doubled after the first step (FOLD)
        if constexpr (CLS) {
          row_entries<F, VPL, CPLX_H>(
              cnt, acc, xs, [&](int k) { return HV::load_smem(s_val, tb + k); },
              [&](int k) {
                return ld_cg<F, VPL>(x + ((int64_t)min(max(r + s_off[tb + k], 0), n - 1) * lpr + sub) * VPL);
              });
        } else {
          row_entries<F, VPL, CPLX_H>(
              cnt, acc, xs,
              [&](int k) {
                const HV h = HV::load(eval, eb + (int64_t)k * 32);
                if constexpr (FOLD) return first ? h : h.twice();
                else return h;
              },
              [&](int k) { return ld_cg<F, VPL>(x + ((int64_t)__ldg(ecol + eb + (int64_t)k * 32) * lpr + sub) * VPL); });
        }
        finish_acc<F, VPL>(acc);
        if (FOLD || first) out = acc;
        else recur_out<F, VPL>(acc, prev, out);
        st_v<F, VPL>(y + me, out);
      }
      if constexpr (BRAKET) {
        dot_acc<F, VPL>(b, out, m0);
        if (first) dot_acc<F, VPL>(b, xs, m1);
      } else {
        dot_acc<F, VPL>(xs, xs, m0);
        if (first) dot_acc<F, VPL>(xs, out, m1);
        else dot_acc<F, VPL>(xs, prev, m1);
      }
      prev = xs;
      xs = out;
    }
    const bool more = s + 1 < n_steps;
    __syncthreads();                                          // the CTA's stores precede its arrival
    if (more && threadIdx.x == 0) {
      __threadfence();
      atomicAdd(meet, 1u);
    }
    double* p = part + (int64_t)s * 2 * gridDim.x;
    if (!BRAKET || first) step_sums<F, true>(m0, m1, p);
    else step_sums<F, false>(m0, m1, p);
    if constexpr (FOLD) {
      if (first) {                                            // from here on with 2 H
        hd = hd.twice();
        if constexpr (CLS)
          for (int32_t q = threadIdx.x; q < nv; q += kStepThreads) s_val[q] = times2(s_val[q]);
      }
    }
    if (!more) break;
    if (threadIdx.x == 0) {
      const unsigned int want = (unsigned int)(s + 1) * gridDim.x;
      uint32_t it = 0;
      unsigned int seen;
      do {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(meet) : "memory");
      } while (seen < want && ++it < wait_limit);
      if (seen < want) {
        atomicOr(err, kErrMeet);
        gave_up = 1;
      }
    }
    __syncthreads();
    if (gave_up) return;
  }
}

}  // namespace tbk
