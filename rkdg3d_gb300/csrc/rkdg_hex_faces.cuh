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
//      orientation.  SPEED: the wave speeds only (the initial time step).
//   2. k_node_hex, a thread per element node: the node's Euler flux
//      (FE_Evolution::GetFlux, fe_evolution.cpp:219-245) and its three
//      contravariant components through shared memory, then one line of each
//      direction's collocated derivative, one moment of each face, and the
//      Runge-Kutta epilogue.  The mass matrix of the Gauss-Legendre basis is
//      diagonal; its inverse sits in the 1D tables.
// Every trace, flux and moment is formed once; the state's traffic is coalesced.
// FP64, per RK step: 32^3 Q2 3.27 ms against 4.9 with the shared-face team
// kernel; 33x27x21 Q1 limited 0.83 ms against 1.5 with the team face and element
// passes, which wrote the fluxes once per side and applied a dense mass inverse.
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

template <int P, typename R, bool SPEED>
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
  __shared__ Frame<3, R> sFr[FB];
  __shared__ R sJ[FB];
  const HexOps<R>& H = hex_ops<R>(prm.hops);
  const int tid = threadIdx.x, f0 = blockIdx.x * FB, nface = prm.nface, ne = prm.ne;
  const long long NDa = prm.ndofs;
  if (tid < FB) {
    const int4 fc = f0 + tid < nface ? prm.flist[f0 + tid] : make_int4(-1, -1, 0, 0);
    sF[tid] = fc;
  }
  __syncthreads();
  if constexpr (STAGE) {
    // one row of ND values per warp and load (Q1: four), all in flight at once
    constexpr int RPW = 32 / ND, NG = 2 * FB / RPW, IT = (NG + S::NT / 32 - 1) / (S::NT / 32);
    const int warp = tid >> 5, lane = tid & 31, sub = lane / ND, i = lane - sub * ND;
    R tmp[IT][NEQ];
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int g = warp + it * (S::NT / 32), r = g * RPW + sub;
      const bool on = g < NG && sub < RPW;
      const int e = on ? (r >= FB ? sF[r - FB].y : sF[r].x) : -1;
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
    __syncthreads();
  }
  // the faces' frames, by the last threads (the first ones have traces to form)
  if (tid >= S::NT - FB) {
    const int fl = tid - (S::NT - FB);
    const int4 fc = sF[fl];
    if (fc.x >= 0) {
      const R* fg = (const R*)prm.fgeo + (long long)((fc.z & 7) * 4) * ne + fc.x;
      R n[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) n[c] = __ldg(fg + (long long)c * ne);
      sFr[fl] = make_frame<3, R>(n);
      sJ[fl] = __ldg(fg + 3LL * ne);
    }
  }
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
          right_state<3>(bc.type, bc.state, s1, s2, sFr[fl].n, gamma, cov, (R)prm.rgas);
        }
      }
      if (none) {
#pragma unroll
        for (int k = 0; k < NEQ; ++k) F[k] = R(0);
      } else {
        lmax = checked_speed(prm, riemann<3>(s1, s2, sFr[fl], F, gamma, cov, prm.rs, prm.avg), fc.x);
      }
      if constexpr (!SPEED) {
        // this thread alone reads the point it overwrites
#pragma unroll
        for (int k = 0; k < NEQ; ++k) sT[0][k][fl][t1] = F[k] * sJ[fl];
      }
    }
  }
  if constexpr (!SPEED) {
    __syncthreads();
    // moments with the tangential basis, M1^-1 of both directions included;
    // the second side's traces are done with
    R* sO = &sT[1][0][0][0];  // [NEQ][FB][NF2]
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
            for (int a = 0; a < NQ1; ++a) s += H.lw[a * N1 + i0] * fv[a];
            w[i0][b] = s;
          }
        }
        R* out = sO + (k * FB + fl) * NF2;
#pragma unroll
        for (int i1 = 0; i1 < N1; ++i1)
#pragma unroll
          for (int i0 = 0; i0 < N1; ++i0) {
            R s = R(0);
#pragma unroll
            for (int b = 0; b < NQ1; ++b) s += H.lw[b * N1 + i1] * w[i0][b];
            out[i0 + N1 * i1] = s;
          }
      }
    }
    __syncthreads();
    const int nval = min(FB, nface - f0) * NF2;
#pragma unroll
    for (int t0 = 0; t0 < NEQ * FB * NF2; t0 += S::NT) {
      const int t = t0 + tid, k = t / (FB * NF2), r = t - k * (FB * NF2);
      if (k < NEQ && r < nval) ((R*)prm.fslot)[((long long)k * nface + f0) * NF2 + r] = sO[t];
    }
  }
  block_max_commit<R>(lmax, prm.mcs);
}

template <int P, typename R>
__global__ void __launch_bounds__(HexFaces<P>::NTN)
    k_node_hex(const __grid_constant__ RhsParams prm, const R* __restrict__ u,
               const __grid_constant__ EpiParams<R> ep) {
  using S = HexFaces<P>;
  constexpr int N1 = S::N1, NF2 = S::NF2, ND = S::ND, NEQ = S::NEQ, EPB = S::EPB, NT = S::NTN;
  constexpr int NP = ND | 1;
  __shared__ R sG[3][NEQ][EPB * NP];
  __shared__ R sMD[N1 * N1], sGeo[EPB][11];  // sGeo: adj(J), 1/det J
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
  if (tid < N1 * N1) sMD[tid] = H.md[tid];
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
    const R* fx = (const R*)prm.fslot;
    const long long nf = (long long)prm.nface * NF2;
#pragma unroll
    for (int lf = 0; lf < 6; ++lf) {
      constexpr int AX[6] = {2, 1, 0, 1, 0, 2}, SD[6] = {0, 0, 1, 1, 0, 1};
      const int ref = prm.fref[lf * ne + e], op = prm.fop ? prm.fop[lf * ne + e] : 0;
      const int t0 = AX[lf] == 0 ? jy : jx, t1 = AX[lf] == 2 ? jy : jz;
      const int jn = AX[lf] == 0 ? jx : (AX[lf] == 1 ? jy : jz);
      R b = H.mb[SD[lf] * N1];  // by selection: an indexed constant is read lane by lane
#pragma unroll
      for (int j = 1; j < N1; ++j) b = jn == j ? H.mb[SD[lf] * N1 + j] : b;
      const R c = (ref & 1) ? b : -b;
      const R* p = fx + (long long)(ref >> 1) * NF2 + (op ? square_op(op, t0, t1, N1) : t0 + N1 * t1);
#pragma unroll
      for (int k = 0; k < NEQ; ++k) acc[k] += c * __ldg(p + k * nf);
    }
  }
  __syncthreads();
  if (live) {
    idet = sGeo[sl][9];
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
  __syncthreads();
  if (live) {
#pragma unroll
    for (int m = 0; m < N1; ++m) {
      const R d0 = sMD[jx * N1 + m], d1 = sMD[jy * N1 + m], d2 = sMD[jz * N1 + m];
      const int b = sl * NP;
#pragma unroll
      for (int k = 0; k < NEQ; ++k)
        acc[k] += d0 * sG[0][k][b + m + N1 * jy + NF2 * jz] + d1 * sG[1][k][b + jx + N1 * m + NF2 * jz] +
                  d2 * sG[2][k][b + jx + N1 * jy + NF2 * m];
    }
    if (prm.ncidx) {  // hanging faces of a nonconforming mesh
      const int ix = prm.ncidx[e];
      if (ix >= 0) {
        const R* xf = (const R*)prm.xface + (long long)ix * NEQ * ND + i;
        const R m = H.iw[jx] * H.iw[jy] * H.iw[jz];
#pragma unroll
        for (int k = 0; k < NEQ; ++k) acc[k] += m * xf[k * ND];
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
    // cell means, one (element, equation) per thread
    const double* wm = prm.tab->wmean;
    for (int t = tid; t < EPB * NEQ; t += NT) {
      const int k = t / EPB, s = t - k * EPB, em = blockIdx.x * EPB + s;
      if (em >= ne) continue;
      if constexpr (std::is_same<R, double>::value) {
        double m = 0.0;
#pragma unroll
        for (int j = 0; j < ND; ++j) m += wm[j] * sG[0][k][s * NP + j];
        store_mean(ep, (long long)k * ne + em, m);
      } else {
        float mh = 0.0f, ml = 0.0f, ph, pl;
#pragma unroll
        for (int j = 0; j < ND; ++j) {
          const float2 w = prm.tab->wmean32[j];
          ds_mul_f(w.x, w.y, sG[0][k][s * NP + j], ph, pl);
          ds_add(mh, ml, ph, pl);
          if (ep.final_stage) ds_add(mh, ml, w.x * sG[1][k][s * NP + j], 0.0f);
        }
        if (ep.means32)
          ep.means32[(long long)k * ne + em] = make_float2(mh, ml);
        else
          ep.means[(long long)k * ne + em] = (double)mh + (double)ml;
      }
    }
  }
  block_max_commit<R, std::is_same<R, double>::value>(lmax, prm.mcs);
}

}  // namespace rkdg
