// Right-hand side on hexahedra as a face pass and a node pass.
//
// FE_Evolution::Mult (fe_evolution.cpp:102-216) in two launches.
//   1. k_face_hex, FB faces per CTA: a thread per (face, side, variable) forms
//      the trace at the (p+2)^2 face points (contraction along the normal, then
//      the 2D interpolation, sum-factorised), a thread per face point the
//      numerical flux (FaceIntegrator::AssembleFaceVector,
//      face_integrator.cpp:11-276: Elem1, Elem2 argument order, the
//      Elem1-outward normal) or a boundary condition's, and a thread per
//      (face, variable) the flux's moments with the (p+1)^2 tangential basis
//      functions, which both elements of the face share up to the face's
//      orientation.  (k_speed_hex: the wave speeds only, for the initial time
//      step.)
//   2. k_node_hex, a thread per element node: the node's Euler flux
//      (FE_Evolution::GetFlux, fe_evolution.cpp:219-245) and its three
//      contravariant components through shared memory, then one line of each
//      direction's collocated derivative, one moment of each face, and the
//      Runge-Kutta epilogue.  The mass matrix of the Gauss-Legendre basis is
//      diagonal; its inverse sits in the 1D tables.
// Every trace, flux and moment is formed once; the state's traffic is coalesced.
//
// FP32 keeps the arithmetic, and the order of the sums, that the team (Q1) and
// tile (Q2) kernels have: their results to the bit on meshes whose elements
// index their common faces alike (see riemann() for what other rounding does to
// limited runs).  The face pass stages its elements by rows (a warp per row, all
// loads in flight); it is bound by issue (64% of the slots), the node pass by the
// latency of its loads at 36 warps per SM.  Per RK step: 48^3 Q2 0.94 ms against
// 1.04 (tiles) and 1.5 (rows read by the trace threads), 48x45x51 Q1 with HLL
// 0.46 ms against 0.78 (team), with the limiter 0.62 against 1.12, 31x29x23 Q2
// limited 0.30 against 0.53.
//
// FP64, per RK step: 32^3 Q2 2.91 ms against 4.9 with the shared-face team
// kernel (the FP64 pipe is active 84-87% of the time); 33x27x21 Q1 limited
// 0.83 ms against 1.5 with the team face and element passes, which wrote the
// fluxes once per side and applied a dense mass inverse.
#pragma once

#include "rkdg_common.h"
#include "rkdg_generic.cuh"
#include "rkdg_hex_team.cuh"
#include "rkdg_physics.cuh"
#include "rkdg_planar.cuh"

namespace rkdg {

template <int P>
struct HexFaces {
  static constexpr int N1 = P + 1, NQ1 = P + 2, ND = N1 * N1 * N1, NQF = NQ1 * NQ1, NF2 = N1 * N1,
                       NEQ = 5;
  static constexpr int FB = P == 2 ? 16 : 24, NT = 256;  // faces and threads of a face-pass CTA
  static constexpr int QS = NQF | 1, NDS = ND | 1;       // odd row strides in shared memory
  // node pass: elements and threads (whole warps) per CTA
  static constexpr int EPB = P == 2 ? 7 : 24, NTN = 192;
  static_assert(FB * 2 * NEQ <= NT && FB * NQF <= NT && EPB * ND <= NTN && NTN % 32 == 0, "one round each");
};

// Orientation code of a square face seen from the other element: bit 0 swaps
// the two tangential indices, bits 1 and 2 then reverse the first and second.
__device__ __forceinline__ int square_op(int op, int i, int j, int n) {
  const int a = (op & 1) ? j : i, b = (op & 1) ? i : j;
  return ((op & 2) ? n - 1 - a : a) + n * ((op & 4) ? n - 1 - b : b);
}

template <int P, typename R>
__global__ void __launch_bounds__(HexFaces<P>::NT)
    k_face_hex(const __grid_constant__ RhsParams prm, const R* __restrict__ u) {
  using S = HexFaces<P>;
  constexpr int N1 = S::N1, NQ1 = S::NQ1, NQF = S::NQF, NF2 = S::NF2, NEQ = S::NEQ, FB = S::FB,
                ND = S::ND, QS = S::QS;
  // float: the faces' elements are staged coalesced (a thread per value); with
  // FP64 the loads hide behind the FP64 pipe and the threads read their rows
  constexpr bool STAGE = std::is_same<R, float>::value;
  constexpr int NROW = FB * 2 * NEQ;  // (variable, side, face)
  __shared__ R sT[2][NEQ][FB][QS];
  __shared__ R sU[STAGE ? NROW * S::NDS : 1];
  __shared__ int4 sF[FB];
  // float: the normal and |J_f|, and the plain arithmetic (see riemann())
  constexpr bool F32 = std::is_same<R, float>::value;
  __shared__ typename std::conditional<F32, R[3], Frame<3, R>>::type sFr[FB];
  __shared__ R sJ[FB];
  const HexOps<R>& H = hex_ops<R>(prm.hops);
  const int tid = threadIdx.x, f0 = blockIdx.x * FB, nface = prm.nface, ne = prm.ne;
  const long long NDa = prm.ndofs;
  auto face_at = [&](int fl) {
    return f0 + fl < nface ? __ldg(prm.flist + f0 + fl) : make_int4(-1, -1, 0, 0);
  };
  // the faces and their frames, by the last threads; their loads and the
  // staged rows' are in flight together
  const int fo = tid - (S::NT - FB);
  R fn[4];
  if (fo >= 0) {
    const int4 fc = face_at(fo);
    sF[fo] = fc;
    const R* fg = (const R*)prm.fgeo + (long long)((fc.z & 7) * 4) * ne + max(fc.x, 0);
#pragma unroll
    for (int c = 0; c < 4; ++c) fn[c] = __ldg(fg + (long long)c * ne);
  }
  if constexpr (STAGE) {
    // one row of ND values per warp and load (Q1: four)
    constexpr int RPW = 32 / ND, NG = 2 * FB / RPW, IT = (NG + S::NT / 32 - 1) / (S::NT / 32);
    const int warp = tid >> 5, lane = tid & 31, sub = lane / ND, i = lane - sub * ND;
    R tmp[IT][NEQ];
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int g = warp + it * (S::NT / 32), r = g * RPW + sub;
      int e = -1;
      if (g < NG && sub < RPW) {
        const int4 fc = face_at(r >= FB ? r - FB : r);
        e = r >= FB ? fc.y : fc.x;
      }
      const R* p = u + (long long)e * ND + i;
#pragma unroll
      for (int k = 0; k < NEQ; ++k) tmp[it][k] = e >= 0 ? __ldg(p + k * NDa) : R(0);
    }
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int g = warp + it * (S::NT / 32), r = g * RPW + sub;
      if (g < NG && sub < RPW) {
#pragma unroll
        for (int k = 0; k < NEQ; ++k) sU[(k * 2 * FB + r) * S::NDS + i] = tmp[it][k];
      }
    }
  }
  if (fo >= 0) {
    if constexpr (F32) {
#pragma unroll
      for (int c = 0; c < 3; ++c) sFr[fo][c] = fn[c];
    } else {
      sFr[fo] = make_frame<3, R>(fn);
    }
    sJ[fo] = fn[3];
  }
  __syncthreads();
  // traces, in each side's own tensor order a + NQ1 b; the face list is sorted
  // by the faces' normal axis, so a warp takes one of the three orders
  if (tid < NROW) {
    const int k = tid / (2 * FB), r = tid - k * 2 * FB, side = r / FB, fl = r - side * FB;
    const int4 fc = sF[fl];
    const int e = side ? fc.y : fc.x;
    if (e >= 0) {
      const int lf = side ? (fc.z >> 3) & 7 : fc.z & 7;
      R v[NF2];
      team_contract_s_axis<P>(lf, STAGE ? sU + tid * S::NDS : u + k * NDa + (long long)e * ND, H.lend, v);
      team_interp<P, 1>(v, H.l1d, &sT[side][k][fl][0]);
    }
  }
  __syncthreads();
  R lmax = R(0);
  if (tid < FB * NQF) {
    const int fl = tid / NQF, t1 = tid - fl * NQF;
    if (f0 + fl < nface) {
      const int4 fc = sF[fl];
      const int lf1 = fc.z & 7;
      R s1[NEQ], s2[NEQ], F[NEQ];
      const R gamma = (R)prm.gamma, cov = (R)prm.covolume;
#pragma unroll
      for (int k = 0; k < NEQ; ++k) s1[k] = sT[0][k][fl][t1];
      bool none = false;
      if (fc.y >= 0) {
        const int op = fc.z >> 6, t2 = op ? square_op(op, t1 % NQ1, t1 / NQ1, NQ1) : t1;
#pragma unroll
        for (int k = 0; k < NEQ; ++k) s2[k] = sT[1][k][fl][t2];
      } else {
        const int nb = prm.fnbr[lf1 * ne + fc.x];
        none = nb == -1;  // no integrator
        if (!none) {
          const BCSlot& bc = prm.bc[-2 - nb];
          const R* n;
          if constexpr (F32) n = sFr[fl]; else n = sFr[fl].n;
          right_state<3>(bc.type, bc.state, s1, s2, n, gamma, cov, (R)prm.rgas);
        }
      }
      // no integrator, or a non-physical state: no flux
#pragma unroll
      for (int k = 0; k < NEQ; ++k) F[k] = R(0);
      if (!none) {
        R sp;
        if constexpr (F32) {
          const R n[3] = {sFr[fl][0], sFr[fl][1], sFr[fl][2]};
          sp = riemann<3, R, true>(s1, s2, n, F, gamma, cov, prm.rs, prm.avg);
        } else {
          sp = riemann<3>(s1, s2, sFr[fl], F, gamma, cov, prm.rs, prm.avg);
        }
        lmax = checked_speed(prm, sp, fc.x);
      }
      // this thread alone reads the point it overwrites
#pragma unroll
      for (int k = 0; k < NEQ; ++k) sT[0][k][fl][t1] = F32 ? H.wf[t1] * sJ[fl] * F[k] : F[k] * sJ[fl];
    }
  }
  __syncthreads();
  // moments with the tangential basis (FP64: weights and M1^-1 of both
  // directions included); the second side's traces are done with
  const R* tw = F32 ? H.l1d : H.lw;
  R* sO = &sT[1][0][0][0];  // [FB][NEQ][NF2]
  static_assert(NF2 <= QS, "moments fit the traces' place");
  if (tid < FB * NEQ) {
    const int k = tid / FB, fl = tid - k * FB;
    if (f0 + fl < nface) {
      const R* f = &sT[0][k][fl][0];
      R w[N1][NQ1];
#pragma unroll
      for (int b = 0; b < NQ1; ++b) {
        R fv[NQ1];
#pragma unroll
        for (int a = 0; a < NQ1; ++a) fv[a] = f[a + NQ1 * b];
#pragma unroll
        for (int i0 = 0; i0 < N1; ++i0) {
          R s = R(0);
#pragma unroll
          for (int a = 0; a < NQ1; ++a) s += tw[a * N1 + i0] * fv[a];
          w[i0][b] = s;
        }
      }
      R* out = sO + (fl * NEQ + k) * NF2;
#pragma unroll
      for (int i1 = 0; i1 < N1; ++i1)
#pragma unroll
        for (int i0 = 0; i0 < N1; ++i0) {
          R s = R(0);
#pragma unroll
          for (int b = 0; b < NQ1; ++b) s += tw[b * N1 + i1] * w[i0][b];
          out[i0 + N1 * i1] = s;
        }
    }
  }
  __syncthreads();
  const int nval = min(FB, nface - f0) * NEQ * NF2;
  R* out = (R*)prm.fslot + (long long)f0 * NEQ * NF2;
#pragma unroll
  for (int t0 = 0; t0 < NEQ * FB * NF2; t0 += S::NT)
    if (t0 + tid < nval) out[t0 + tid] = sO[t0 + tid];
  block_max_commit<R>(lmax, prm.mcs);
}

// The largest face wave speed of an FP64 state.  Every face point is bounded in
// FP32 first (rkdg_speed_bound.h); only faces with a point that could hold the
// maximum, or that has no bound, and boundary faces are evaluated in FP64.  A
// call on Gaussian pulses, 48x45x51 Q1, HLL with TRRS speeds: 0.35 ms against
// 1.32 with every point in FP64; 48^3 Q2 acoustic pulse, Rusanov: 0.46 against 1.65
// (planar: 524,288 P1 triangles 0.17 against 0.57, 317x211 quad Q3 0.09 against
// 0.15).
template <int P>
__global__ void __launch_bounds__(HexFaces<P>::NT)
    k_speed_hex(const __grid_constant__ RhsParams prm, const double* __restrict__ u) {
  using S = HexFaces<P>;
  constexpr int N1 = S::N1, NQ1 = S::NQ1, NQF = S::NQF, NF2 = S::NF2, NEQ = S::NEQ, FB = S::FB,
                ND = S::ND, QS = S::QS, NROW = FB * 2 * NEQ;
  struct Est {
    float u[NROW * S::NDS], t[2][NEQ][FB][QS], top[NROW];
  };
  union Buf {
    Est f;
    double t[2][NEQ][FB][QS];
  };
  __shared__ Buf sb;
  __shared__ int4 sF[FB];
  __shared__ int sNeed[FB];
  const int tid = threadIdx.x, f0 = blockIdx.x * FB, nface = prm.nface, ne = prm.ne;
  const long long NDa = prm.ndofs;
  auto face_at = [&](int fl) {
    return f0 + fl < nface ? __ldg(prm.flist + f0 + fl) : make_int4(-1, -1, 0, 0);
  };
  if (tid < FB) {
    const int4 fc = face_at(tid);
    sF[tid] = fc;
    sNeed[tid] = fc.x >= 0 && fc.y < 0;
  }
  {
    constexpr int RPW = 32 / ND, NG = 2 * FB / RPW, IT = (NG + S::NT / 32 - 1) / (S::NT / 32);
    const int warp = tid >> 5, lane = tid & 31, sub = lane / ND, i = lane - sub * ND;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int g = warp + it * (S::NT / 32), r = g * RPW + sub;
      if (g < NG && sub < RPW) {
        const int4 fc = face_at(r >= FB ? r - FB : r);
        const int e = r >= FB ? fc.y : fc.x;
        const double* p = u + (long long)e * ND + i;
#pragma unroll
        for (int k = 0; k < NEQ; ++k) sb.f.u[(k * 2 * FB + r) * S::NDS + i] = e >= 0 ? cut_f32(__ldg(p + k * NDa)) : 0.0f;
      }
    }
  }
  __syncthreads();
  if (tid < NROW) {
    const int k = tid / (2 * FB), r = tid - k * 2 * FB, side = r / FB, fl = r - side * FB;
    const int4 fc = sF[fl];
    if (fc.y >= 0) {
      const float* row = sb.f.u + tid * S::NDS;
      float v[NF2], top = 0.0f;
      team_contract_s_axis<P>(side ? (fc.z >> 3) & 7 : fc.z & 7, row, prm.hops.f.lend, v);
      team_interp<P, 1>(v, prm.hops.f.l1d, &sb.f.t[side][k][fl][0]);
#pragma unroll
      for (int j = 0; j < ND; ++j) top = fmaxf(top, fabsf(row[j]));
      sb.f.top[tid] = top;
    }
  }
  __syncthreads();
  if (tid < FB * NQF) {
    const int fl = tid / NQF, t1 = tid - fl * NQF;
    const int4 fc = sF[fl];
    if (fc.y >= 0) {
      const int op = fc.z >> 6, t2 = op ? square_op(op, t1 % NQ1, t1 / NQ1, NQ1) : t1;
      float s1[NEQ], s2[NEQ], n[3];
#pragma unroll
      for (int k = 0; k < NEQ; ++k) {
        s1[k] = sb.f.t[0][k][fl][t1];
        s2[k] = sb.f.t[1][k][fl][t2];
      }
#pragma unroll
      for (int c = 0; c < 3; ++c)
        n[c] = (float)__ldg((const double*)prm.fgeo + (long long)((fc.z & 7) * 4 + c) * ne + fc.x);
      const float g = (float)prm.gamma, b = (float)prm.covolume;
      SpeedSide A, B;
      const bool ok = speed_side<3>(s1, sb.f.top + fl, 2 * FB, n, g, b, A) &&
                      speed_side<3>(s2, sb.f.top + FB + fl, 2 * FB, n, g, b, B) &&
                      speed_below(speed_bound(A, B, g, prm.rs, prm.avg, prm.quirks & 1), prm.mcs);
      if (!ok) sNeed[fl] = 1;
    }
  }
  __syncthreads();
  int any = 0;
  for (int fl = 0; fl < FB; ++fl) any |= sNeed[fl];
  if (!any) return;  // the same for every thread
  __syncthreads();   // the estimates are done with
  if (tid < NROW) {
    const int k = tid / (2 * FB), r = tid - k * 2 * FB, side = r / FB, fl = r - side * FB;
    const int4 fc = sF[fl];
    const int e = side ? fc.y : fc.x;
    if (e >= 0 && sNeed[fl]) {
      double v[NF2];
      team_contract_s_axis<P>(side ? (fc.z >> 3) & 7 : fc.z & 7, u + k * NDa + (long long)e * ND, prm.hops.d.lend, v);
      team_interp<P, 1>(v, prm.hops.d.l1d, &sb.t[side][k][fl][0]);
    }
  }
  __syncthreads();
  double lmax = 0.0;
  if (tid < FB * NQF) {
    const int fl = tid / NQF, t1 = tid - fl * NQF;
    const int4 fc = sF[fl];
    if (fc.x >= 0 && sNeed[fl]) {
      const int lf1 = fc.z & 7, nb = fc.y >= 0 ? 0 : prm.fnbr[lf1 * ne + fc.x];
      if (nb != -1) {
        double s1[NEQ], s2[NEQ], F[NEQ], n[3];
#pragma unroll
        for (int c = 0; c < 3; ++c)
          n[c] = __ldg((const double*)prm.fgeo + (long long)(lf1 * 4 + c) * ne + fc.x);
#pragma unroll
        for (int k = 0; k < NEQ; ++k) s1[k] = sb.t[0][k][fl][t1];
        if (fc.y >= 0) {
          const int op = fc.z >> 6, t2 = op ? square_op(op, t1 % NQ1, t1 / NQ1, NQ1) : t1;
#pragma unroll
          for (int k = 0; k < NEQ; ++k) s2[k] = sb.t[1][k][fl][t2];
        } else {
          const BCSlot& bc = prm.bc[-2 - nb];
          right_state<3>(bc.type, bc.state, s1, s2, n, prm.gamma, prm.covolume, prm.rgas);
        }
        lmax = checked_speed(prm, riemann<3>(s1, s2, make_frame<3, double>(n), F, prm.gamma, prm.covolume,
                                             prm.rs, prm.avg), fc.x);
      }
    }
  }
  block_max_commit<double>(lmax, prm.mcs);
}

// Part of the mean of an element's float values (hi, and lo where given) with the
// weights wm of the nodes, to FP64: the limiter's switches read the mean.  Order 1
// takes all nodes at once, order 2 a plane of nine.  The values are summed in fixed
// point with 32 bits below the last place of the largest one (nothing is lost but
// what lies 2^-56 below it), those of one weight together (nodes of as many middle
// indices), so that a mean takes one or nine FP64 products instead of 8 or 27 on
// a pipe that issues two per clock and SM: those cost 31x29x23 Q2 limited 17 us a
// stage.
template <int P>
__device__ __forceinline__ double pair_mean(const float* hi, const float* lo, const double* __restrict__ wm) {
  constexpr int N = P == 2 ? 9 : 8, NC = P == 2 ? 3 : 1;
  unsigned top = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) top = max(top, __float_as_uint(hi[j]) & 0x7fffffffu);
  const int emax = (int)(top >> 23);
  double m = 0.0;
  if (emax < 64 || emax == 255) {  // tiny or not finite
    for (int j = 0; j < N; ++j) m += wm[j] * (widen(hi[j]) + (lo ? widen(lo[j]) : 0.0));
    return m;
  }
  auto fixed = [&](float x) {
    const unsigned b = __float_as_uint(x);
    const int e = (int)((b >> 23) & 0xff);
    const unsigned mant = e ? (b & 0x7fffffu) | 0x800000u : 0u;
    const long long v = (long long)(((unsigned long long)mant << 32) >> min(emax - e, 63));
    return (b >> 31) ? -v : v;
  };
  long long S[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) S[c] = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const int c = P == 2 ? (j % 3 == 1) + (j / 3 == 1) : 0;
    S[c] += fixed(hi[j]);
    if (lo) S[c] += fixed(lo[j]);
  }
  constexpr int AT[3] = {0, 1, 4};  // a node of each weight
#pragma unroll
  for (int c = 0; c < NC; ++c) m += wm[AT[c]] * (double)S[c];
  return m * __hiloint2double((emax - 182 + 1023) << 20, 0);
}

template <int P, typename R>
__global__ void __launch_bounds__(HexFaces<P>::NTN)
    k_node_hex(const __grid_constant__ RhsParams prm, const R* __restrict__ u,
               const __grid_constant__ EpiParams<R> ep) {
  using S = HexFaces<P>;
  constexpr int N1 = S::N1, NF2 = S::NF2, ND = S::ND, NEQ = S::NEQ, EPB = S::EPB, NT = S::NTN;
  constexpr int NP = ND | 1;
  __shared__ R sG[3][NEQ][EPB * NP];
  constexpr bool F32 = std::is_same<R, float>::value;  // float: the plain arithmetic (see riemann())
  __shared__ R sMD[N1 * N1], sGeo[EPB][11];  // sGeo: adj(J), 1/det J
  __shared__ R sW[N1], sMinv[N1];            // float: node weights, 1D inverse mass
  __shared__ R sA[F32 && P == 2 ? 3 : 1][F32 && P == 2 ? NEQ : 1][F32 && P == 2 ? EPB * NP : 1];
  const HexOps<R>& H = hex_ops<R>(prm.hops);
  const int tid = threadIdx.x, ne = prm.ne;
  const long long NDa = prm.ndofs;
  const int sl = tid / ND, i = tid - sl * ND;
  const int e = blockIdx.x * EPB + sl;
  const bool live = sl < EPB && e < ne;
  for (int t = tid; t < EPB * 10; t += NT) {
    const int c = t / EPB, s = t - c * EPB;
    if (blockIdx.x * EPB + s < ne)
      sGeo[s][c] = __ldg((const R*)prm.egeo + (long long)c * ne + blockIdx.x * EPB + s);
  }
  if (tid < N1 * N1) sMD[tid] = F32 ? H.d1[tid] : H.md[tid];
  if (F32 && tid < N1) {
    sW[tid] = H.w1[tid];
    sMinv[tid] = H.minv1[tid * N1 + tid];
  }
  const int jx = i % N1, jy = (i / N1) % N1, jz = i / NF2;
  const long long own = (long long)e * ND + i;
  R lmax = R(0), idet = R(0), acc[NEQ];
#pragma unroll
  for (int k = 0; k < NEQ; ++k) acc[k] = R(0);
  R st[NEQ];
  if (live) {
#pragma unroll
    for (int k = 0; k < NEQ; ++k) st[k] = u[k * NDa + own];
    // the faces' moments, in flight with the state
    const int4* rp = reinterpret_cast<const int4*>(prm.fref) + 2LL * e;
    const int4 ra = __ldg(rp), rb = __ldg(rp + 1);
    const int refs[6] = {ra.x, ra.y, ra.z, ra.w, rb.x, rb.y}, ops = rb.z;
    auto faces = [&](auto turned) {  // turned: some face is indexed another way by its Elem1
#pragma unroll
      for (int o = 0; o < 6; ++o) {
        constexpr int AX[6] = {2, 1, 0, 1, 0, 2}, SD[6] = {0, 0, 1, 1, 0, 1};
        // float: the order in which the team (Q1) and tile (Q2) kernels add them
        constexpr int ORD[6] = {4, 2, 1, 3, 0, 5};
        const int lf = F32 && P == 2 ? ORD[o] : o;
        const int ref = refs[lf];
        const int t0 = AX[lf] == 0 ? jy : jx, t1 = AX[lf] == 2 ? jy : jz;
        const int jn = AX[lf] == 0 ? jx : (AX[lf] == 1 ? jy : jz);
        const R* mb = (F32 ? H.lend : H.mb) + SD[lf] * N1;
        R b = mb[0];  // by selection: an indexed constant is read lane by lane
#pragma unroll
        for (int j = 1; j < N1; ++j) b = jn == j ? mb[j] : b;
        const R c = (ref & 1) ? b : -b;
        const int at = turned.value ? square_op((ops >> (3 * lf)) & 7, t0, t1, N1) : t0 + N1 * t1;
        const R* p = (const R*)prm.fslot + (long long)(ref >> 1) * (NEQ * NF2) + at;
#pragma unroll
        for (int k = 0; k < NEQ; ++k) acc[k] += c * __ldg(p + k * NF2);
      }
    };
    if (ops)
      faces(std::true_type{});
    else
      faces(std::false_type{});
  }
  __syncthreads();
  if (live) {
    idet = sGeo[sl][9];
    if constexpr (F32) {
      R F[NEQ][3];
      lmax = flux_and_speed<3>(st, F, (R)prm.gamma, (R)prm.covolume);
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const R a0 = sGeo[sl][3 * r], a1 = sGeo[sl][3 * r + 1], a2 = sGeo[sl][3 * r + 2];
#pragma unroll
        for (int k = 0; k < NEQ; ++k) sG[r][k][sl * NP + i] = a0 * F[k][0] + a1 * F[k][1] + a2 * F[k][2];
      }
    } else {
      const NodeFlux<3, R> N(st, (R)prm.gamma, (R)prm.covolume);
      lmax = N.speed;
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        R G[NEQ];
        N.contra(st, &sGeo[sl][3 * r], G);
#pragma unroll
        for (int k = 0; k < NEQ; ++k) sG[r][k][sl * NP + i] = G[k];
      }
    }
  }
  __syncthreads();
  if (live) {
    if constexpr (F32) {
      // one direction after the other, each with the other two node weights
      const int b = sl * NP;
      const R wx = sW[jx], wy = sW[jy], wz = sW[jz];
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const int j = r == 0 ? jx : (r == 1 ? jy : jz), st1 = r == 0 ? 1 : (r == 1 ? N1 : NF2);
        const int at = b + i - j * st1;
        const R w = r == 0 ? wy * wz : (r == 1 ? wx * wz : wx * wy);
        R d[N1];
#pragma unroll
        for (int m = 0; m < N1; ++m) d[m] = sMD[j * N1 + m];
#pragma unroll
        for (int k = 0; k < NEQ; ++k) {
          R s = R(0);
#pragma unroll
          for (int m = 0; m < N1; ++m) s += d[m] * sG[r][k][at + m * st1];
          acc[k] += w * s;
        }
      }
    } else {
#pragma unroll
      for (int m = 0; m < N1; ++m) {
        const R d0 = sMD[jx * N1 + m], d1 = sMD[jy * N1 + m], d2 = sMD[jz * N1 + m];
        const int b = sl * NP;
#pragma unroll
        for (int k = 0; k < NEQ; ++k)
          acc[k] += d0 * sG[0][k][b + m + N1 * jy + NF2 * jz] + d1 * sG[1][k][b + jx + N1 * m + NF2 * jz] +
                    d2 * sG[2][k][b + jx + N1 * jy + NF2 * m];
      }
    }
    if (prm.ncidx) {  // hanging faces of a nonconforming mesh
      const int ix = prm.ncidx[e];
      if (ix >= 0) {
        const R* xf = (const R*)prm.xface + (long long)ix * NEQ * ND + i;
        const R m = F32 ? R(1) : H.iw[jx] * H.iw[jy] * H.iw[jz];
#pragma unroll
        for (int k = 0; k < NEQ; ++k) acc[k] += m * xf[k * ND];
      }
    }
  }
  if constexpr (F32) {
    // the inverse mass, x, y, z.  Its 1D matrix is diagonal but for noise of
    // 1e-16, which decides one rounding in sixteen of the middle row of order
    // 2: 9/4 times a float is often half way between two floats
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int j = d == 0 ? jx : (d == 1 ? jy : jz), st1 = d == 0 ? 1 : (d == 1 ? N1 : NF2);
      const R m = sMinv[j];
      if constexpr (P == 2) {
        if (live && j == 0) {
#pragma unroll
          for (int k = 0; k < NEQ; ++k) sA[d][k][sl * NP + i] = acc[k];
        }
        __syncthreads();
        if (live && j == 1) {
          const R off = H.minv1[N1];
#pragma unroll
          for (int k = 0; k < NEQ; ++k) acc[k] = fmaf(m, acc[k], off * sA[d][k][sl * NP + i - st1]);
        } else {
#pragma unroll
          for (int k = 0; k < NEQ; ++k) acc[k] *= m;
        }
      } else {
#pragma unroll
        for (int k = 0; k < NEQ; ++k) acc[k] *= m;
      }
    }
  }
  const bool need_means = ep.mode == 1 && (ep.means || ep.means32);
  if (need_means) __syncthreads();  // every thread has read sG
  if (live) {
#pragma unroll
    for (int k = 0; k < NEQ; ++k) {
      R hi, lo;
      epi_node<R>(ep, k * NDa + own, acc[k] * idet, 1.0, make_float2(1.0f, 0.0f), hi, lo);
      if (need_means) {
        sG[0][k][sl * NP + i] = hi;
        sG[1][k][sl * NP + i] = lo;
      }
    }
  }
  if (need_means) {
    __syncthreads();
    // cell means, one (element, equation) per thread; float pairs of order 2: a
    // plane of nodes per thread, three neighbouring lanes
    const double* wm = prm.tab->wmean;
    constexpr int PL = F32 && P == 2 ? 3 : 1, W = 32 / PL;  // W means per warp
    static_assert(PL == 1 || EPB * NEQ <= NT / 32 * W, "one round of whole warps");
    const int lane = tid & 31, pl = lane % PL;
    for (int t = (tid >> 5) * W + lane / PL; PL > 1 || t < EPB * NEQ; t += NT) {
      const int k = t / EPB, s = t - k * EPB, em = blockIdx.x * EPB + s;
      const bool on = t < EPB * NEQ && lane < PL * W && em < ne;
      double m = 0.0;
      if (on) {
        const int j0 = s * NP + pl * NF2;
        if constexpr (F32) {
          m = pair_mean<P>(sG[0][k] + j0, ep.final_stage ? sG[1][k] + j0 : nullptr, wm + pl * NF2);
        } else {
#pragma unroll
          for (int j = 0; j < ND; ++j) m += wm[j] * sG[0][k][j0 + j];
        }
      }
      if constexpr (PL > 1) m += __shfl_down_sync(0xffffffffu, m, 1) + __shfl_down_sync(0xffffffffu, m, 2);
      if (on && pl == 0) {
        if constexpr (F32) {
          float h, l;
          split_value(m, h, l);
          if (ep.means32)
            ep.means32[(long long)k * ne + em] = make_float2(h, l);
          else
            ep.means[(long long)k * ne + em] = m;
        } else {
          store_mean(ep, (long long)k * ne + em, m);
        }
      }
      if (PL > 1) break;
    }
  }
  block_max_commit<R, std::is_same<R, double>::value>(lmax, prm.mcs);
}

}  // namespace rkdg
