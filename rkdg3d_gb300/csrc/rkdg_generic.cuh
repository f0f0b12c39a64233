// What the kernels share: float-pair arithmetic, row loads, conversions, the
// wave-speed reductions, the map of a batch's active work and the Runge-Kutta
// epilogue; and the kernels of one thread per element: the FP32 element pass, the
// Shu indicator's limiter and the cell means.
#pragma once

#include "rkdg_common.h"
#include "rkdg_physics.cuh"
#include "rkdg_speed_bound.h"

namespace rkdg {

// Largest CTA of the kernels of one thread per element or face point.
constexpr int kGenericMaxBlock = 256;
// The element pass and the Shu limiter of FP32 elements of at most 16 values (Q1
// quads, P1 triangles) are latency bound at the occupancy their registers allow:
// they run at most 128 threads per CTA and are compiled for six (element pass, 80
// registers) or five (limiter, 96 registers) CTAs per SM with a few spilled values,
// which measured 7-8% faster on the batched and triangle workloads than the 12-16
// warps of their uncapped registers.  Larger elements would spill kilobytes at that
// cap and keep the default.
template <typename R, int NVAL>
__host__ __device__ constexpr bool generic_small() {
  return std::is_same<R, float>::value && NVAL <= 16;
}
template <typename R, int NVAL>
__host__ __device__ constexpr int generic_max_block() {
  return generic_small<R, NVAL>() ? 128 : kGenericMaxBlock;
}
template <typename R, int NVAL, bool LIMITER>
__host__ __device__ constexpr int generic_min_blocks() {
  return generic_small<R, NVAL>() ? (LIMITER ? 5 : 6) : 1;
}

// ---- double-single (float pair) helpers for the FP32-bulk path --------------
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}
__device__ __forceinline__ void ds_add(float& hi, float& lo, float bh, float bl) {
  float s, e;
  two_sum(hi, bh, s, e);
  e += lo + bl;
  hi = s + e;
  lo = e - (hi - s);
}
// (ch, cl) * k as a float pair
__device__ __forceinline__ void ds_mul_f(float ch, float cl, float k, float& ph, float& pl) {
  ph = ch * k;
  pl = fmaf(ch, k, -ph) + cl * k;
}

// ---- vector access to the element rows of float arrays ------------------------
// An element's ND values of one variable are contiguous (byNODES layout, offset
// (k * ne + e) * ND).  The float arrays the FP32-bulk path reads and writes are
// the library's own allocations (256-byte aligned), so a row is 16-byte
// aligned when ND % 4 == 0 and 8-byte aligned when ND % 2 == 0.  Double
// arrays may be the caller's and are accessed element by element.
template <typename T, int ND>
struct RowVec {
  static constexpr int W = std::is_same<T, float>::value ? (ND % 4 == 0 ? 4 : (ND % 2 == 0 ? 2 : 1)) : 1;
};
template <int W, typename T>
__device__ __forceinline__ void ld_vec(const T* __restrict__ p, T* v) {
  if constexpr (W == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
  } else if constexpr (W == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    v[0] = t.x; v[1] = t.y;
  } else {
    v[0] = p[0];
  }
}
template <int W, typename T>
__device__ __forceinline__ void st_vec(T* __restrict__ p, const T* v) {
  if constexpr (W == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  } else if constexpr (W == 2) {
    *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
  } else {
    p[0] = v[0];
  }
}
// a whole row of N values
template <int N, typename T>
__device__ __forceinline__ void ld_row(const T* __restrict__ p, T* v) {
  constexpr int W = RowVec<T, N>::W;
#pragma unroll
  for (int i = 0; i < N; i += W) ld_vec<W>(p + i, v + i);
}
template <int N, typename T>
__device__ __forceinline__ void st_row(T* __restrict__ p, const T* v) {
  constexpr int W = RowVec<T, N>::W;
#pragma unroll
  for (int i = 0; i < N; i += W) st_vec<W>(p + i, v + i);
}

// The plain read first: thousands of CTAs end on one address, and once a large
// value is there most of them need no atomic.
__device__ __forceinline__ void atomic_max_nonneg(unsigned long long* addr, double v) {
  if (!(v > 0.0) || (unsigned long long)__double_as_longlong(v) <= *(volatile unsigned long long*)addr) return;
  atomicMax(addr, (unsigned long long)__double_as_longlong(v));
}

// Block-wide max of a per-thread wave speed, committed with one atomicMax per
// block (the MPI_Allreduce(MAX) of main.cpp:543 on one device).
// SQUARE: v is the square of a speed.
template <typename R, bool SQUARE = false>
__device__ __forceinline__ void block_max_commit(R v, unsigned long long* dst) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __shared__ R redd[32];
  if (lane == 0) redd[w] = v;
  __syncthreads();
  if (w == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    R x = lane < nw ? redd[lane] : R(0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = fmax(x, __shfl_xor_sync(0xffffffffu, x, o));
    if (lane == 0) atomic_max_nonneg(dst, SQUARE ? sqrt((double)x) : (double)x);
  }
}

// A double cut to FP32 (towards zero) by bit operations: the conversion
// instruction runs at the FP64 rate.
__device__ __forceinline__ float cut_f32(double x) {
  const int hi = __double2hiint(x);
  if ((unsigned)((hi & 0x7fffffff) - 0x38100000) >= 0x0fe00000u) return __double2float_rz(x);
  const unsigned t = __funnelshift_l((unsigned)__double2loint(x), (unsigned)hi, 3);
  return __uint_as_float(((t ^ 0x40000000u) & 0x7fffffffu) | ((unsigned)hi & 0x80000000u));
}

// FP64 <-> float pair.  The conversion instructions run at the FP64 rate, so
// normal numbers take bit operations instead: the rounded high word and the
// remainder, an integer of at most 29 bits in units of the double's last place.
// 4.4 M values: split 12 us against 49.
__device__ __forceinline__ void split_value(double v, float& h, float& l) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const int ex = (int)((hi >> 20) & 0x7ff) - 1023;
  if (ex < -60 || ex > 100) {  // zero, tiny, huge, not finite
    h = (float)v;
    l = (float)(v - (double)h);
    return;
  }
  // 23 mantissa bits below the exponent, then 29 bits of remainder
  unsigned t = (__funnelshift_l(lo, hi, 3) ^ 0x40000000u) & 0x7fffffffu;
  const int rest = (int)(lo & 0x1fffffffu);
  const bool up = rest > 0x10000000 || (rest == 0x10000000 && (t & 1u));
  t += up;  // the carry moves into the exponent
  const int r = up ? rest - 0x20000000 : rest;
  const unsigned sign = hi & 0x80000000u;
  h = __uint_as_float(t | sign);
  // 2^(ex - 52), negative for negative v
  l = (float)r * __uint_as_float((unsigned)((ex - 52 + 127) << 23) | sign);
}
__device__ __forceinline__ double widen(float x) {
  const unsigned b = __float_as_uint(x), e = (b >> 23) & 0xff;
  if (e == 0 || e == 0xff) return (double)x;
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(b << 29));
}

// The bound of a face point's speed (rkdg_speed_bound.h) lies below the largest
// FP64 speed so far.
__device__ __forceinline__ bool speed_below(float bound, const unsigned long long* mcs) {
  const double top = __longlong_as_double((long long)*(const volatile unsigned long long*)mcs);
  return bound < (float)top * 0.999999f;
}

__device__ __forceinline__ void flag_error(int* err, int code, int where) {
  if (atomicCAS(&err[0], 0, code) == 0) err[1] = where;
}

// The reference aborts when a face wave speed is negative
// (face_integrator.cpp:214-218).  That is how its solvers report a
// non-physical state (-1), but HLLC's signed max(SL, SR) (rs_hllc.cpp:98) is
// also negative in supersonic flow against the normal.  With quirk bit 0 only
// the -1 of a non-physical state is an error; the speed enters the max as 0.
// In a batch of independent problems (pb >= 0) a non-physical state stops
// only its own problem: the problem is marked failed and the others go on.
template <typename R>
__device__ __forceinline__ R checked_speed(const RhsParams& prm, R sp, int e, int pb = -1) {
  if constexpr (std::is_same<R, double>::value)
    if (__double2hiint(sp) >= 0) return sp;  // the sign on the integer pipe
  if (sp < R(0)) {
    if (!(prm.quirks & 1) || sp == R(-1)) {
      if (pb >= 0 && prm.pfail)
        prm.pfail[pb] = 1;
      else
        flag_error(prm.err, 2, e);
    }
    return R(0);
  }
  return sp;
}

// Per-problem max wave speed for batched problems: elements of one problem
// are contiguous, so a warp holds a few contiguous runs; a segmented shuffle
// reduction leaves each run's max in its first lane, which commits it.
template <typename R, bool SQUARE = false>
__device__ __forceinline__ void segmented_max_commit(R v, int pb, unsigned long long* pmcs) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const R o = __shfl_down_sync(0xffffffffu, v, off);
    const int opb = __shfl_down_sync(0xffffffffu, pb, off);
    if (lane + off < 32 && opb == pb) v = fmax(v, o);
  }
  const int prev = __shfl_up_sync(0xffffffffu, pb, 1);
  if (pb >= 0 && (lane == 0 || prev != pb)) atomic_max_nonneg(&pmcs[pb], SQUARE ? sqrt((double)v) : (double)v);
}

// Batched problems with a map of the active work: the i-th element of the
// active problems (in problem order), and its problem pb.  While every problem
// is active the map is the identity: one load instead of a chain of six to nine.
__device__ __forceinline__ int active_element(const int* cum, const int* pid, const int* poff, int na,
                                              int i, int ne, const int* prob, int& pb) {
  if (cum[na] == ne) {
    pb = prob[i];
    return i;
  }
  int lo = 0, hi = na;  // cum[lo] <= i < cum[lo + 1]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (cum[mid] <= i)
      lo = mid;
    else
      hi = mid;
  }
  pb = pid[lo];
  return poff[pb] + (i - cum[lo]);
}

// Likewise the i-th face of the active problems: each problem's interior faces,
// then its others.
__device__ __forceinline__ int active_face(const RhsParams& prm, int na, int i) {
  const int* cum = prm.act_fcum;
  if (cum[na] == prm.nface) return i;
  int lo = 0, hi = na;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (cum[mid] <= i)
      lo = mid;
    else
      hi = mid;
  }
  const int pb = prm.act_pid[lo], j = i - cum[lo], f = prm.pfi[pb] + j, end = prm.pfi[pb + 1];
  return f < end ? f : prm.pfb[pb] + (f - end);
}

// (ch, cl) * (sh, sl) as a float pair: a tableau coefficient times a
// problem's dt, both float pairs.
__device__ __forceinline__ void ds_mul(float ch, float cl, float sh, float sl, float& ph, float& pl) {
  const float p = ch * sh;
  float e = fmaf(ch, sh, -p);
  e = fmaf(ch, sl, e);
  e = fmaf(cl, sh, e);
  ph = p + e;
  pl = e - (ph - p);
}

// Epilogue for one element and one equation: y[i], i < ND.  dts scales the
// coefficients of batched problems (1 otherwise): a double for a double
// state, a float pair (dts2) for the float path.
template <int ND, typename R>
__device__ __forceinline__ void epilogue(const EpiParams<R>& ep, long long base_idx,
                                         const R* y, const R* wmean, int ne, int e, int k,
                                         double dts, float2 dts2) {
  if (ep.mode == 0) {
#pragma unroll
    for (int i = 0; i < ND; ++i) ep.out64[base_idx + i] = (double)y[i];
    return;
  }
  if constexpr (std::is_same<R, double>::value) {
    double m = 0.0;
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      const long long idx = base_idx + i;
      double v = ep.base ? ep.base[idx] : 0.0;
      for (int j = 0; j < ep.nprev; ++j) v += (ep.cprev[j] * dts) * ep.kprev[j][idx];
      v += (ep.ccur * dts) * y[i];
      if (ep.kout) ep.kout[idx] = y[i];
      if (ep.out64) ep.out64[idx] = v;
      if (ep.out32) ep.out32[idx] = (float)v;
      m += wmean[i] * v;
    }
    if (ep.means || ep.means32) store_mean(ep, (long long)k * ne + e, m);
  } else {
    // rows in vectors of W values; at most three previous stages (the
    // tableaux have up to four stages), unrolled so the coefficients stay in
    // registers
    constexpr int W = RowVec<float, ND>::W;
    float mh = 0.0f, ml = 0.0f;
    float ch[3], cl[3], cch = ep.ccur_hi, ccl = ep.ccur_lo;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      ch[j] = ep.cprev_hi[j];
      cl[j] = ep.cprev_lo[j];
    }
    if (ep.pdt || ep.pdt2) {  // unscaled tableau coefficients times the problem's dt
#pragma unroll
      for (int j = 0; j < 3; ++j)
        if (j < ep.nprev) ds_mul(ch[j], cl[j], dts2.x, dts2.y, ch[j], cl[j]);
      ds_mul(cch, ccl, dts2.x, dts2.y, cch, ccl);
    }
    if (!ep.final_stage) {
#pragma unroll
      for (int i0 = 0; i0 < ND; i0 += W) {
        const long long idx = base_idx + i0;
        float inc[W], bh[W], kp[W], v[W];
        ld_vec<W>(ep.baselo + idx, inc);
        ld_vec<W>(ep.basehi + idx, bh);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          if (j < ep.nprev) {
            ld_vec<W>(ep.kprev[j] + idx, kp);
#pragma unroll
            for (int w = 0; w < W; ++w) inc[w] = fmaf(ch[j], kp[w], inc[w]);
          }
        }
#pragma unroll
        for (int w = 0; w < W; ++w) {
          inc[w] = fmaf(cch, y[i0 + w], inc[w]);
          v[w] = bh[w] + inc[w];
        }
        if (ep.kout) st_vec<W>(ep.kout + idx, y + i0);
        st_vec<W>(ep.out32 + idx, v);
#pragma unroll
        for (int w = 0; w < W; ++w) {
          float ph, pl;
          ds_mul_f(wmean[i0 + w], 0.0f, v[w], ph, pl);
          ds_add(mh, ml, ph, pl);
        }
      }
    } else {
#pragma unroll
      for (int i0 = 0; i0 < ND; i0 += W) {
        const long long idx = base_idx + i0;
        float sh[W], sl[W], kp[W], h[W], l[W];
#pragma unroll
        for (int w = 0; w < W; ++w) sh[w] = sl[w] = 0.0f;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          if (j < ep.nprev) {
            ld_vec<W>(ep.kprev[j] + idx, kp);
#pragma unroll
            for (int w = 0; w < W; ++w) {
              float ph, pl;
              ds_mul_f(ch[j], cl[j], kp[w], ph, pl);
              ds_add(sh[w], sl[w], ph, pl);
            }
          }
        }
        ld_vec<W>(ep.basehi + idx, h);
        ld_vec<W>(ep.baselo + idx, l);
#pragma unroll
        for (int w = 0; w < W; ++w) {
          float ph, pl;
          ds_mul_f(cch, ccl, y[i0 + w], ph, pl);
          ds_add(sh[w], sl[w], ph, pl);
          ds_add(h[w], l[w], sh[w], sl[w]);
        }
        st_vec<W>(ep.out32 + idx, h);
        st_vec<W>(ep.outlo + idx, l);
#pragma unroll
        for (int w = 0; w < W; ++w) {
          float ph, pl;
          ds_mul_f(wmean[i0 + w], 0.0f, h[w], ph, pl);
          ds_add(mh, ml, ph, pl);
          ds_add(mh, ml, wmean[i0 + w] * l[w], 0.0f);
        }
      }
    }
    // (mh, ml) stays normalised through ds_add: it is the float pair of the
    // mean as it stands
    if (ep.means32)
      ep.means32[(long long)k * ne + e] = make_float2(mh, ml);
    else if (ep.means)
      ep.means[(long long)k * ne + e] = (double)mh + (double)ml;
  }
}

// ---- element pass of the planar right-hand side --------------------------------
// One thread per element, for FP32 elements of at most 16 values: the faces'
// fluxes come from the face pass (rkdg_planar.cuh), the element's own rows are
// loaded once.  524,288 P1 triangles: 59 us against 76 for a thread per node;
// 253,064 Q1 quads of a batch: 45 + 48 us for the two passes against 96 for one
// kernel that evaluated every face from both sides.  Q1 quads keep the arithmetic
// and the order of the sums of a kernel that evaluated its faces itself, see
// riemann().
template <int G, int P, typename R>
__global__ void __launch_bounds__(generic_max_block<R, El<G, P>::NEQ * El<G, P>::ND>(),
                                  generic_min_blocks<R, El<G, P>::NEQ * El<G, P>::ND, false>())
    k_elem_planar(const __grid_constant__ RhsParams prm, const R* __restrict__ u,
                  const __grid_constant__ EpiParams<R> ep) {
  using E = El<G, P>;
  constexpr int DIM = E::DIM, ND = E::ND, NEQ = E::NEQ, NFPE = E::NFPE, NQF = E::NQF;
  __shared__ R sB[NFPE][NQF][ND];
  __shared__ R sD[DIM][ND][ND];
  __shared__ R sMinv[ND][ND];
  __shared__ R sWm[ND];
  const RefTables* T = prm.tab;
  // batched problems with a map of the active work: CTAs past it are idle
  if (prm.act_cum && (int)(blockIdx.x * blockDim.x) >= prm.act_cum[*prm.act_n]) return;
  const PlanarOps<R>& H = prm.pops->f;
  for (int t = threadIdx.x; t < NFPE * NQF * ND; t += blockDim.x) (&sB[0][0][0])[t] = H.eb[t];
  for (int t = threadIdx.x; t < DIM * ND * ND; t += blockDim.x) (&sD[0][0][0])[t] = H.ed[t];
  for (int t = threadIdx.x; t < ND * ND; t += blockDim.x) (&sMinv[0][0])[t] = H.em[t];
  for (int t = threadIdx.x; t < ND; t += blockDim.x) sWm[t] = H.wm[t];
  __syncthreads();

  const int ne = prm.ne;
  const long long NDa = prm.ndofs;
  R gamma = (R)prm.gamma, cov = (R)prm.covolume;
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  R lmax = R(0);
  bool live = e < ne;
  int pb = -1;
  double dts = 1.0;
  float2 dts2 = make_float2(1.0f, 0.0f);
  if (prm.act_cum) {
    const int na = *prm.act_n;
    live = e < prm.act_cum[na];
    if (live) e = active_element(prm.act_cum, prm.act_pid, prm.poff, na, e, prm.ne, prm.prob, pb);
  }
  if (live && prm.prob) {
    live = prm.pactive[pb] != 0;
    if constexpr (std::is_same<R, float>::value) {
      // FP32 copies: no FP64 conversions per element
      gamma = prm.pgamma32 ? prm.pgamma32[pb] : (R)prm.pgamma[pb];
      cov = prm.pcov32 ? prm.pcov32[pb] : (R)prm.pcov[pb];
      if (ep.pdt2) {
        dts2 = ep.pdt2[pb];
      } else if (ep.pdt) {
        dts = ep.pdt[pb];
        const float h = (float)dts;
        dts2 = make_float2(h, (float)(dts - (double)h));
      }
    } else {
      gamma = (R)prm.pgamma[pb];
      cov = (R)prm.pcov[pb];
      if (ep.pdt) dts = ep.pdt[pb];
    }
  }
  if (live) {
    R acc[NEQ][ND];
#pragma unroll
    for (int k = 0; k < NEQ; ++k)
#pragma unroll
      for (int s = 0; s < ND; ++s) acc[k][s] = R(0);
    R own[NEQ][ND];
#pragma unroll
    for (int k = 0; k < NEQ; ++k) ld_row<ND>(u + k * NDa + (long long)e * ND, own[k]);
    const long long nf = (long long)prm.nface * NQF;
#pragma unroll
    for (int lf = 0; lf < NFPE; ++lf) {
      const int ref = prm.fref[lf * ne + e];
      const R* fx = (const R*)prm.fslot + (long long)ref_face(ref) * NQF;
      const R sg = (ref & 2) ? R(1) : R(-1);
      R fl[NEQ][NQF];
#pragma unroll
      for (int k = 0; k < NEQ; ++k) ld_row<NQF>(fx + k * nf, fl[k]);
      // Elem1's points in order; this element may run through them backwards
#pragma unroll
      for (int q = 0; q < NQF; ++q) {
        const R* Bo = sB[lf][(ref & 1) ? NQF - 1 - q : q];
#pragma unroll
        for (int k = 0; k < NEQ; ++k) {
          const R t = sg * fl[k][q];
#pragma unroll
          for (int j = 0; j < ND; ++j) acc[k][j] += t * Bo[j];
        }
      }
    }
    {
      const R* eg = (const R*)prm.egeo;
      const R* ng = (const R*)prm.ngeo;  // per-node geometry (bilinear quads) or null
      R adj[DIM][DIM];
#pragma unroll
      for (int r = 0; r < DIM; ++r)
#pragma unroll
        for (int d = 0; d < DIM; ++d) adj[r][d] = eg[(long long)(r * DIM + d) * ne + e];
      const R idet = eg[(long long)(DIM * DIM) * ne + e];
#pragma unroll
      for (int m = 0; m < ND; ++m) {
        if (ng) {
#pragma unroll
          for (int r = 0; r < DIM; ++r)
#pragma unroll
            for (int d = 0; d < DIM; ++d) adj[r][d] = ng[((long long)(r * DIM + d) * ND + m) * ne + e];
        }
        R st[NEQ];
#pragma unroll
        for (int k = 0; k < NEQ; ++k) st[k] = own[k][m];
        R F[NEQ][DIM];
        const R sp = flux_and_speed<DIM>(st, F, gamma, cov);
        lmax = fmax(lmax, sp);
#pragma unroll
        for (int k = 0; k < NEQ; ++k)
#pragma unroll
          for (int r = 0; r < DIM; ++r) {
            R gc = R(0);
#pragma unroll
            for (int d = 0; d < DIM; ++d) gc += adj[r][d] * F[k][d];
#pragma unroll
            for (int j = 0; j < ND; ++j) acc[k][j] += sD[r][j][m] * gc;
          }
      }
      if (prm.ncidx) {  // hanging faces of a nonconforming mesh
        const int ix = prm.ncidx[e];
        if (ix >= 0) {
          const R* xf = (const R*)prm.xface + (long long)ix * NEQ * ND;
#pragma unroll
          for (int k = 0; k < NEQ; ++k)
#pragma unroll
            for (int j = 0; j < ND; ++j) acc[k][j] += xf[k * ND + j];
        }
      }
#pragma unroll
      for (int k = 0; k < NEQ; ++k) {
        R y[ND];
#pragma unroll
        for (int i = 0; i < ND; ++i) {
          R v = R(0);
#pragma unroll
          for (int j = 0; j < ND; ++j) v += sMinv[i][j] * acc[k][j];
          // the collocated mass of a quad is diagonal, so a per-node 1/det J
          // (bilinear quads) applies row by row
          y[i] = v * (ng ? ng[((long long)(DIM * DIM) * ND + i) * ne + e] : idet);
        }
        if (T->wmn_e) {  // this element's own cell-mean weights
          R wl[ND];
#pragma unroll
          for (int i = 0; i < ND; ++i) wl[i] = (R)T->wmn_e[(long long)e * ND + i];
          epilogue<ND, R>(ep, k * NDa + (long long)e * ND, y, wl, ne, e, k, dts, dts2);
        } else {
          epilogue<ND, R>(ep, k * NDa + (long long)e * ND, y, sWm, ne, e, k, dts, dts2);
        }
      }
    }
  }
  if (prm.prob)
    segmented_max_commit<R>(lmax, live ? pb : -1, prm.pmcs);
  else
    block_max_commit<R>(lmax, prm.mcs);
}

// ---- limiter ------------------------------------------------------------------
// Cell means for the limiter: FP64, or the FP32 path's float pairs.
__device__ __forceinline__ bool mean_lt(double a, double b) { return a < b; }
__device__ __forceinline__ bool mean_lt(float2 a, float2 b) {
  return a.x < b.x || (a.x == b.x && a.y < b.y);
}
template <bool F32>
__device__ __forceinline__ typename std::conditional<F32, float2, double>::type load_mean(
    const LimParams& prm, long long i) {
  if constexpr (F32)
    return prm.means32[i];
  else
    return prm.means[i];
}
// a mean as a double (either representation)
__device__ __forceinline__ double mean_value(const LimParams& prm, long long i) {
  if (prm.means32) {
    const float2 m = prm.means32[i];
    return (double)m.x + (double)m.y;
  }
  return prm.means[i];
}

// Nodal basis of the reference element at an arbitrary reference point (the
// tensor GL Lagrange basis, or the triangle basis from its monomial expansion).
template <int G, int P>
__device__ __forceinline__ void basis_at(const RefTables* T, const double* xi,
                                         double (&phi)[El<G, P>::ND]) {
  using E = El<G, P>;
  constexpr int DIM = E::DIM, ND = E::ND;
  if constexpr (G == 2) {
    double px[P + 1], py[P + 1];
    px[0] = py[0] = 1.0;
#pragma unroll
    for (int a = 1; a <= P; ++a) {
      px[a] = px[a - 1] * xi[0];
      py[a] = py[a - 1] * xi[1];
    }
#pragma unroll
    for (int j = 0; j < ND; ++j) phi[j] = 0.0;
#pragma unroll
    for (int m = 0; m < ND; ++m) {
      const double mv = px[T->tmono[m][0]] * py[T->tmono[m][1]];
#pragma unroll
      for (int j = 0; j < ND; ++j) phi[j] += T->tcoef[m][j] * mv;
    }
  } else {
    constexpr int N1 = P + 1;
    double l[DIM][N1];
#pragma unroll
    for (int d = 0; d < DIM; ++d)
#pragma unroll
      for (int i = 0; i < N1; ++i) {
        double v = 1.0;
#pragma unroll
        for (int m = 0; m < N1; ++m)
          if (m != i) v *= (xi[d] - T->x1n[m]) / (T->x1n[i] - T->x1n[m]);
        l[d][i] = v;
      }
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      double v = l[0][j % N1] * l[1][(j / N1) % N1];
      if constexpr (DIM == 3) v *= l[2][j / (N1 * N1)];
      phi[j] = v;
    }
  }
}

// IndicatorShu::checkDiscontinuity (indicator_shu.cpp:13-74) for element e:
// for every cell k of the stencil (e, then its face neighbours) the average
// over e of k's polynomial extrapolated there (Averager::
// computeStencilExtrapAverages, averager.cpp:154-273: the element rule of
// order p + OrderW on e mapped into k's reference frame), and
//   value = min(1, Ck max|mean_e| / (sum_k |mean_e - extrap_k| + eps)),
// Ck = 0.03, eps = 1e-6, or 1 where both are below eps.  The maximum runs over
// the stencil but reads e's own mean every time, as the reference does.
template <int G, int P, bool DS, typename R>
__device__ __forceinline__ void shu_indicator(const LimParams& prm, const R* __restrict__ u,
                                              const float* __restrict__ ulo, int e,
                                              R (&val)[El<G, P>::NEQ]) {
  using E = El<G, P>;
  constexpr int DIM = E::DIM, ND = E::ND, NEQ = E::NEQ, NFPE = E::NFPE;
  const RefTables* T = prm.tab;
  const int ne = prm.ne;
  const long long NDa = prm.ndofs;
  const double* ea = prm.eaff;
  double Je[DIM][DIM], xe[DIM], ume[NEQ], sum[NEQ];
#pragma unroll
  for (int i = 0; i < DIM; ++i) {
#pragma unroll
    for (int r = 0; r < DIM; ++r) Je[i][r] = ea[(long long)(i * DIM + r) * ne + e];
    xe[i] = ea[(long long)(DIM * DIM + i) * ne + e];
  }
#pragma unroll
  for (int k = 0; k < NEQ; ++k) {
    ume[k] = mean_value(prm, (long long)k * ne + e);
    sum[k] = 0.0;
  }
  double wsum = 0.0;
  for (int q = 0; q < T->nqs; ++q) wsum += T->ws[q];
  // stencil: the cell, its face neighbours, then the elements across its
  // hanging faces (ElementToElementTable, limiter.cpp:118-123)
  const int ncrow = prm.ncidx ? prm.ncidx[e] : -1;
  const int nnc = ncrow >= 0 ? prm.nc_ptr[ncrow + 1] - prm.nc_ptr[ncrow] : 0;
  for (int s = -1; s < NFPE + nnc; ++s) {
    int kc;
    if (s < 0) {
      kc = e;
    } else if (s < NFPE) {
      kc = prm.fnbr[s * ne + e];
    } else {
      const int ent = prm.nc_ent[prm.nc_ptr[ncrow] + s - NFPE];
      kc = prm.nc_face[(ent >> 1) * 4 + ((ent & 1) ? 0 : 2)];
    }
    if (kc < 0) continue;  // boundary faces are not in the stencil
    // e's reference point xi -> k's reference point A xi + b
    double A[DIM][DIM], b[DIM];
    if (kc == e) {
#pragma unroll
      for (int i = 0; i < DIM; ++i) {
#pragma unroll
        for (int r = 0; r < DIM; ++r) A[i][r] = i == r ? 1.0 : 0.0;
        b[i] = 0.0;
      }
    } else {
      double Jk[DIM][DIM], Ki[DIM][DIM], dx[DIM];
#pragma unroll
      for (int i = 0; i < DIM; ++i) {
#pragma unroll
        for (int r = 0; r < DIM; ++r) Jk[i][r] = ea[(long long)(i * DIM + r) * ne + kc];
        dx[i] = xe[i] - ea[(long long)(DIM * DIM + i) * ne + kc];
      }
      if constexpr (DIM == 2) {
        const double id = 1.0 / (Jk[0][0] * Jk[1][1] - Jk[0][1] * Jk[1][0]);
        Ki[0][0] = Jk[1][1] * id;
        Ki[0][1] = -Jk[0][1] * id;
        Ki[1][0] = -Jk[1][0] * id;
        Ki[1][1] = Jk[0][0] * id;
      } else {
        const double c00 = Jk[1][1] * Jk[2][2] - Jk[1][2] * Jk[2][1];
        const double c01 = Jk[0][2] * Jk[2][1] - Jk[0][1] * Jk[2][2];
        const double c02 = Jk[0][1] * Jk[1][2] - Jk[0][2] * Jk[1][1];
        const double id = 1.0 / (Jk[0][0] * c00 + Jk[1][0] * c01 + Jk[2][0] * c02);
        Ki[0][0] = c00 * id;
        Ki[0][1] = c01 * id;
        Ki[0][2] = c02 * id;
        Ki[1][0] = (Jk[1][2] * Jk[2][0] - Jk[1][0] * Jk[2][2]) * id;
        Ki[1][1] = (Jk[0][0] * Jk[2][2] - Jk[0][2] * Jk[2][0]) * id;
        Ki[1][2] = (Jk[0][2] * Jk[1][0] - Jk[0][0] * Jk[1][2]) * id;
        Ki[2][0] = (Jk[1][0] * Jk[2][1] - Jk[1][1] * Jk[2][0]) * id;
        Ki[2][1] = (Jk[0][1] * Jk[2][0] - Jk[0][0] * Jk[2][1]) * id;
        Ki[2][2] = (Jk[0][0] * Jk[1][1] - Jk[0][1] * Jk[1][0]) * id;
      }
#pragma unroll
      for (int i = 0; i < DIM; ++i) {
        b[i] = 0.0;
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
          double a = 0.0;
#pragma unroll
          for (int m = 0; m < DIM; ++m) a += Ki[i][m] * Je[m][r];
          A[i][r] = a;
          b[i] += Ki[i][r] * dx[r];
        }
      }
    }
    // W_j = mean over e of k's basis function j
    double W[ND];
#pragma unroll
    for (int j = 0; j < ND; ++j) W[j] = 0.0;
    for (int q = 0; q < T->nqs; ++q) {
      double xk[DIM];
#pragma unroll
      for (int i = 0; i < DIM; ++i) {
        double v = b[i];
#pragma unroll
        for (int r = 0; r < DIM; ++r) v += A[i][r] * T->xs[q][r];
        xk[i] = v;
      }
      double phi[ND];
      basis_at<G, P>(T, xk, phi);
      const double wq = T->ws[q] / wsum;
#pragma unroll
      for (int j = 0; j < ND; ++j) W[j] += wq * phi[j];
    }
#pragma unroll
    for (int k = 0; k < NEQ; ++k) {
      double ex = 0.0;
#pragma unroll
      for (int j = 0; j < ND; ++j) {
        const long long idx = k * NDa + (long long)kc * ND + j;
        double v = (double)u[idx];
        if constexpr (DS) v += (double)ulo[idx];
        ex += v * W[j];
      }
      sum[k] += fabs(ume[k] - ex);
    }
  }
#pragma unroll
  for (int k = 0; k < NEQ; ++k) {
    const double mx = fabs(ume[k]);
    const double v = (mx < 1e-6 && sum[k] < 1e-6) ? 1.0 : fmin(1.0, 0.03 * mx / (sum[k] + 1e-6));
    val[k] = (R)v;
  }
}

// LimiterFinDiff::limit (limiter_findiff.cpp:3-33) with the Shu indicator, one
// thread per element: the element becomes its mean where the last equation's
// indicator is below 0.999 (the Multi limiter is rejected with Shu).
template <int G, int P, typename R, bool DS>
__global__ void __launch_bounds__(generic_max_block<R, El<G, P>::NEQ * El<G, P>::ND>(),
                                  generic_min_blocks<R, El<G, P>::NEQ * El<G, P>::ND, true>())
    k_limit_shu(const LimParams prm, R* __restrict__ u, float* __restrict__ ulo) {
  using E = El<G, P>;
  constexpr int ND = E::ND, NEQ = E::NEQ;
  int e = blockIdx.x * blockDim.x + threadIdx.x, pmap = -1;
  if (prm.act_cum) {  // batched problems: the i-th element of the active ones
    const int na = *prm.act_n;
    if (e >= prm.act_cum[na]) return;
    e = active_element(prm.act_cum, prm.act_pid, prm.poff, na, e, prm.ne, prm.prob, pmap);
  }
  if (e >= prm.ne) return;
  if (prm.prob && !prm.pactive[prm.act_cum ? pmap : prm.prob[e]]) return;
  R sv[NEQ];
  shu_indicator<G, P, DS>(prm, u, ulo, e, sv);
  if (!(sv[NEQ - 1] < R(0.999))) return;
#pragma unroll
  for (int k = 0; k < NEQ; ++k) {
    R h;
    float l = 0.0f;
    if constexpr (std::is_same<R, float>::value) {
      const float2 m = prm.means32[(long long)k * prm.ne + e];
      h = m.x;
      l = m.y;
    } else {
      h = prm.means[(long long)k * prm.ne + e];
    }
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      const long long i = k * prm.ndofs + (long long)e * ND + j;
      u[i] = h;
      if constexpr (DS) ulo[i] = l;
    }
  }
}

// ---- cell means (Averager::computeMeanValues, averager.cpp:84-109) -----------
// GridFunction::GetElementAverages = (int u) / (int 1); for affine elements the
// Jacobian cancels and the weights are the reference integrals of the basis
// functions normalised to sum 1.  lo (optional) is the low word of a float pair.
template <int G, int P, typename T>
__global__ void k_means_generic(int ne, long long ndofs, const RefTables* tab,
                                const T* __restrict__ u, const float* __restrict__ ulo,
                                double* __restrict__ means) {
  using E = El<G, P>;
  constexpr int ND = E::ND, NEQ = E::NEQ;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
#pragma unroll
  for (int k = 0; k < NEQ; ++k) {
    double m = 0.0;
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      double v = (double)u[k * ndofs + (long long)e * ND + j];
      if (ulo) v += (double)ulo[k * ndofs + (long long)e * ND + j];
      m += (tab->wmn_e ? tab->wmn_e[(long long)e * ND + j] : tab->wmean[j]) * v;
    }
    means[(long long)k * ne + e] = m;
  }
}

}  // namespace rkdg
