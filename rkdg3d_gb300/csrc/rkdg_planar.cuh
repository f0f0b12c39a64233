// Right-hand side on triangles and quadrilaterals: a face pass and a node pass.
//
// FE_Evolution::Mult (fe_evolution.cpp:102-216) in two launches.
//   1. k_face_planar, one thread per face point: both traces, the numerical
//      flux with the arguments ordered (Elem1, Elem2, Elem1-outward normal) as
//      FaceIntegrator::AssembleFaceVector has them (face_integrator.cpp:11-276)
//      or the boundary condition's state, and |J_f| F into the face's slot.
//      Every face is evaluated once and both elements read the same flux, so
//      the scheme stays conservative without atomics.  SPEED: the wave speeds
//      only (the initial time step).
//   2. k_node_planar, one thread per element node: the node's Euler flux and
//      its contravariant components through shared memory, then
//        y_i = 1/det J (sum_r sum_m MD_r[i][m] G_r[m] -+ sum_faces MB[i][q] f_q)
//      with MD = M^-1 D and MB = M^-1 B^T w formed on the host, and the
//      Runge-Kutta epilogue.  Consecutive threads hold consecutive values of
//      every array, so all state traffic is coalesced and a thread keeps
//      neq values instead of neq * nd.
// FP32 elements of at most 16 values (Q1 quads, P1 triangles) run the second pass
// with a thread per element (k_elem_planar): there the instructions around a
// node's few values outnumber its arithmetic three to one.
//
// Quads add the volume before the faces, triangles and FP32 Q2 quads the faces
// first.  Neither order is the more accurate; a Sod run over its whole time (877
// steps, chaotic at one ulp) keeps the oracle's number of steps with this one, and
// about one rounding variant in seven gives 878.
//
// On quadrilaterals the mass, trace and derivative tables of the collocated
// Gauss-Legendre basis are sparse (the mass matrix is diagonal, a face point
// sees one line of nodes): N1 terms instead of ND.
//
// The FP64 kernels are bound by the FP64 pipe (two fused operations per clock
// and SM): evaluating each face once and the sparse tables is what counts.
// Against one thread per element with dense tables, which evaluated every face
// from both sides: 301x203 quad Q2 FP64 right-hand side 0.32 ms (0.77), 317x211
// quad Q3 FP32 stage 53 us (303), 302x101 P2 triangles FP64 stage 136 us (240),
// 200x4 quad Q1 FP64 stage 18 us (105; 9 us a launch is one FP64 flux's chain).
#pragma once

#include "rkdg_common.h"
#include "rkdg_generic.cuh"
#include "rkdg_physics.cuh"

namespace rkdg {

template <typename R>
__device__ __forceinline__ const PlanarOps<R>& planar_ops(const PlanarOpsPair* p) {
  if constexpr (std::is_same<R, float>::value)
    return p->f;
  else
    return p->d;
}

template <int G, int P>
struct Planar {
  using E = El<G, P>;
  static constexpr int N1 = P + 1;
  // elements per CTA of the node pass; SMALL: one or two warps, for meshes that
  // would leave SMs without a CTA
  static constexpr int EPB = G == 3 ? (P == 3 ? 12 : 32) : (P == 1 ? 64 : 32);
  static constexpr int SMALL = G == 3 ? (P == 1 ? 8 : (P == 2 ? 7 : 4)) : (P == 1 ? 10 : 5);
  // threads of n elements: whole warps (the wave-speed reductions)
  __host__ __device__ static constexpr int threads(int n) { return (n * E::ND + 31) / 32 * 32; }
  static constexpr int NT = threads(EPB);
};

// Node jn (from the face point inwards along the normal axis) behind point q
// of local face lf of a quadrilateral.
template <int N1>
__device__ __forceinline__ int quad_face_node(int lf, int q, int jn) {
  const int t = lf >= 2 ? N1 - 1 - q : q;  // faces 2 and 3 run backwards
  return (lf & 1) ? jn + N1 * t : t + N1 * jn;
}
__device__ __forceinline__ int quad_face_side(int lf) { return lf == 1 || lf == 2; }

// MAP: a batch with a map of the active work (prm.act_cum).
template <int G, int P, typename R, bool SPEED, bool MAP>
__global__ void __launch_bounds__(kGenericMaxBlock)
    k_face_planar(const __grid_constant__ RhsParams prm, const R* __restrict__ u) {
  using E = El<G, P>;
  constexpr int DIM = 2, ND = E::ND, NEQ = E::NEQ, NFPE = E::NFPE, NQF = E::NQF, N1 = P + 1;
  // FP32 Q1 and Q2 quads: the plain arithmetic (see riemann()), traces from the
  // dense table
  constexpr bool PLAIN = G == 3 && P <= 2 && std::is_same<R, float>::value;
  __shared__ R sB[G == 2 || PLAIN ? NFPE * NQF * ND : 1];
  const PlanarOps<R>& H = planar_ops<R>(prm.pops);
  if constexpr (G == 2 || PLAIN) {
    for (int t = threadIdx.x; t < NFPE * NQF * ND; t += blockDim.x) sB[t] = H.b[t];
    __syncthreads();
  }
  const int ne = prm.ne;
  const long long NDa = prm.ndofs;
  R lmax = R(0);
  // MAP: CTAs run over the points of the active problems' faces
  const int na = MAP ? *prm.act_n : 0, nfa = MAP ? prm.act_fcum[na] : prm.nface;
  // (face points: unsigned, up to four per face)
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x, next;; t = next) {
    next = t + gridDim.x * blockDim.x;
    int f = (int)(t / NQF);
    const int q = (int)(t - (unsigned)f * NQF);
    int pb = -1;
    bool live = f < nfa;
    if (MAP && live) f = active_face(prm, na, f);
    lmax = R(0);
    int4 face = make_int4(0, -1, 0, 0);
    int e1 = 0;
    R gamma = (R)prm.gamma, cov = (R)prm.covolume;
    if (live) {
      face = prm.flist[f];
      e1 = face.x;
      if (prm.prob) {
        pb = face.w;  // set with the batch
        live = prm.pactive[pb] != 0;
        if constexpr (std::is_same<R, float>::value) {
          gamma = prm.pgamma32 ? prm.pgamma32[pb] : (R)prm.pgamma[pb];
          cov = prm.pcov32 ? prm.pcov32[pb] : (R)prm.pcov[pb];
        } else {
          gamma = (R)prm.pgamma[pb];
          cov = (R)prm.pcov[pb];
        }
      }
    }
    if (live) {
      bool skip = false;
      const int lf1 = face.z & 7;
      const R* fg = (const R*)prm.fgeo;
      R n[DIM];
#pragma unroll
      for (int c = 0; c < DIM; ++c) n[c] = fg[(long long)(lf1 * (DIM + 1) + c) * ne + e1];
      const R jac = fg[(long long)(lf1 * (DIM + 1) + DIM) * ne + e1];
      // a side's trace at its own face point
      auto trace = [&](int e, int lf, int qq, R* s) {
        const R* ue = u + (long long)e * ND;
        if constexpr (G == 3) {
          R le[N1];
          const int sd = quad_face_side(lf);
#pragma unroll
          for (int j = 0; j < N1; ++j) le[j] = sd ? H.lend[N1 + j] : H.lend[j];
          const int i0 = quad_face_node<N1>(lf, qq, 0), st = (lf & 1) ? 1 : N1;
          if constexpr (PLAIN) {
#pragma unroll
            for (int j = 0; j < N1; ++j) le[j] = sB[(lf * NQF + qq) * ND + i0 + j * st];
          }
#pragma unroll
          for (int k = 0; k < NEQ; ++k) {
            R v = R(0);
#pragma unroll
            for (int j = 0; j < N1; ++j) v += le[j] * ue[k * NDa + i0 + j * st];
            s[k] = v;
          }
        } else {
          const R* B = sB + (lf * NQF + qq) * ND;
#pragma unroll
          for (int k = 0; k < NEQ; ++k) {
            R v = R(0);
#pragma unroll
            for (int j = 0; j < ND; ++j) v += B[j] * ue[k * NDa + j];
            s[k] = v;
          }
        }
      };
      R s1[NEQ], s2[NEQ], F[NEQ];
      if constexpr (SPEED) {
        // bounded in FP32, evaluated in FP64 only where the point could hold the
        // maximum
        if (face.y >= 0) {
          float a1[NEQ], a2[NEQ], nf[DIM], top[2][NEQ];
          auto est = [&](int e, int lf, int qq, float* s, float* tp) {
            const R* ue = u + (long long)e * ND;
            constexpr int NT = G == 3 ? N1 : ND;  // terms of the trace
            const int sd = quad_face_side(lf), i0 = G == 3 ? quad_face_node<N1>(lf, qq, 0) : 0;
            const int st = G == 3 && !(lf & 1) ? N1 : 1;
            const float* B = prm.pops->f.b + (lf * NQF + qq) * ND;
#pragma unroll
            for (int k = 0; k < NEQ; ++k) s[k] = tp[k] = 0.0f;
#pragma unroll
            for (int j = 0; j < NT; ++j) {
              const float w = G == 3 ? (sd ? prm.pops->f.lend[N1 + j] : prm.pops->f.lend[j]) : B[j];
#pragma unroll
              for (int k = 0; k < NEQ; ++k) {
                const float x = cut_f32((double)ue[k * NDa + i0 + j * st]);
                s[k] += w * x;
                tp[k] = fmaxf(tp[k], fabsf(x));
              }
            }
          };
          est(e1, lf1, q, a1, top[0]);
          est(face.y, (face.z >> 3) & 7, (face.z >> 6) ? NQF - 1 - q : q, a2, top[1]);
#pragma unroll
          for (int c = 0; c < DIM; ++c) nf[c] = (float)n[c];
          const float g = (float)gamma, b = (float)cov;
          SpeedSide A, B;
          if (speed_side<DIM>(a1, top[0], 1, nf, g, b, A) && speed_side<DIM>(a2, top[1], 1, nf, g, b, B) &&
              speed_below(speed_bound(A, B, g, prm.rs, prm.avg, prm.quirks & 1), prm.prob ? prm.pmcs + pb : prm.mcs))
            skip = true;
        }
      }
      if (!skip) trace(e1, lf1, q, s1);
      bool none = false;
      if (skip) {
        none = true;
      } else if (face.y >= 0) {
        trace(face.y, (face.z >> 3) & 7, (face.z >> 6) ? NQF - 1 - q : q, s2);
      } else {
        const int nb = prm.fnbr[lf1 * ne + e1];
        none = nb == -1;  // no integrator
        if (!none) {
          const BCSlot& bc = prm.bc[-2 - nb];
          right_state<DIM>(bc.type, bc.state, s1, s2, n, gamma, cov, (R)prm.rgas);
        }
      }
      // no integrator, or a non-physical state: no flux
#pragma unroll
      for (int k = 0; k < NEQ; ++k) F[k] = R(0);
      if (!none) {
        R sp;
        if constexpr (PLAIN)
          sp = riemann<DIM, R, true>(s1, s2, n, F, gamma, cov, prm.rs, prm.avg);
        else
          sp = riemann<DIM>(s1, s2, make_frame<DIM, R>(n), F, gamma, cov, prm.rs, prm.avg);
        lmax = checked_speed(prm, sp, e1, pb);
      }
      if constexpr (!SPEED) {
        R* out = (R*)prm.fslot + (long long)f * NQF + q;
        const long long nf = (long long)prm.nface * NQF;
#pragma unroll
        for (int k = 0; k < NEQ; ++k) out[k * nf] = PLAIN ? (F[k] * H.wf[q]) * jac : F[k] * jac;
      }
    }
    if (prm.prob) segmented_max_commit<R>(lmax, live ? pb : -1, prm.pmcs);
    if (!MAP || (long long)next - threadIdx.x >= (long long)nfa * NQF) break;
  }
  if (!prm.prob) block_max_commit<R>(lmax, prm.mcs);
}

// Runge-Kutta combination at one value; hi (and lo, for a float pair) receive
// the result.  dts scales the coefficients of batched problems.
template <typename R>
__device__ __forceinline__ void epi_node(const EpiParams<R>& ep, long long idx, R y, double dts,
                                         float2 dts2, R& hi, R& lo) {
  lo = R(0);
  hi = y;
  if (ep.mode == 0) {
    ep.out64[idx] = (double)y;
    return;
  }
  if constexpr (std::is_same<R, double>::value) {
    // the increment first: one rounding at the state's size
    double v = (ep.ccur * dts) * y;
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if (j < ep.nprev) v += (ep.cprev[j] * dts) * ep.kprev[j][idx];
    if (ep.base) v += ep.base[idx];
    if (ep.kout) ep.kout[idx] = y;
    if (ep.out64) ep.out64[idx] = v;
    if (ep.out32) ep.out32[idx] = (float)v;
    hi = v;
  } else {
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
      float inc = ep.baselo[idx];
#pragma unroll
      for (int j = 0; j < 3; ++j)
        if (j < ep.nprev) inc = fmaf(ch[j], ep.kprev[j][idx], inc);
      inc = fmaf(cch, y, inc);
      hi = ep.basehi[idx] + inc;
      if (ep.kout) ep.kout[idx] = y;
      ep.out32[idx] = hi;
    } else {
      float sh = 0.0f, sl = 0.0f, ph, pl;
#pragma unroll
      for (int j = 0; j < 3; ++j)
        if (j < ep.nprev) {
          ds_mul_f(ch[j], cl[j], ep.kprev[j][idx], ph, pl);
          ds_add(sh, sl, ph, pl);
        }
      ds_mul_f(cch, ccl, y, ph, pl);
      ds_add(sh, sl, ph, pl);
      hi = ep.basehi[idx];
      lo = ep.baselo[idx];
      ds_add(hi, lo, sh, sl);
      ep.out32[idx] = hi;
      ep.outlo[idx] = lo;
    }
  }
}

template <int G, int P, typename R, int EPB>
__global__ void __launch_bounds__(Planar<G, P>::threads(EPB))
    k_node_planar(const __grid_constant__ RhsParams prm, const R* __restrict__ u,
                  const __grid_constant__ EpiParams<R> ep) {
  using E = El<G, P>;
  using S = Planar<G, P>;
  constexpr int DIM = 2, ND = E::ND, NEQ = E::NEQ, NFPE = E::NFPE, NQF = E::NQF, N1 = P + 1;
  constexpr int NT = S::threads(EPB);
  constexpr int NP = ND | 1;  // odd element stride in shared memory
  // FP32 Q2 quads: the plain arithmetic (see riemann()), and the terms in the
  // order in which dense tables, their zeros left out, add them: the faces, then the
  // nodes of the row and the column in ascending order, then the inverse mass.  Many
  // limited steps part by 1e-4 to 1e-3 under any other rounding.  Batches and
  // problems alone take the same arithmetic.  9 x 1563 x 4 quads, 20 limited steps:
  // 4.74 ms against 6.24 with a thread per element; alone, 301x203 quads, 108 us a step
  // against 105 with the contravariant node fluxes (limited 207 against 186, with the
  // factor applied nd times).
  constexpr bool PLAIN = G == 3 && P == 2 && std::is_same<R, float>::value;
  constexpr int NTERM = 2 * N1;
  __shared__ R sG[DIM][NEQ][EPB * NP];
  // triangles: MD_r[i][m] and MB[i][lf][q], node i fastest; quadrilaterals:
  // d1[i][m] / w_i and lend[side][i] / w_i; PLAIN: each node's D_r[i][m] in order
  // (places in sG: sAt), 1 / w_i and traces [lf][i]
  __shared__ R sMD[G == 2 ? DIM * ND * ND : (PLAIN ? ND * NTERM + ND : N1 * N1)];
  __shared__ R sMB[G == 2 ? NFPE * NQF * ND : (PLAIN ? NFPE * ND : 2 * N1)];
  __shared__ int sAt[PLAIN ? ND * NTERM : 1];
  const PlanarOps<R>& H = planar_ops<R>(prm.pops);
  const int tid = threadIdx.x, ne = prm.ne;
  const long long NDa = prm.ndofs;
  const int sl = tid / ND, i = tid - sl * ND;
  int e = blockIdx.x * EPB + sl, pb = -1;
  // batched problems with a map of the active work: CTAs past it are idle
  if (prm.act_cum && (int)(blockIdx.x * EPB) >= prm.act_cum[*prm.act_n]) return;
  if constexpr (PLAIN) {
    for (int t = tid; t < ND * NTERM; t += NT) {
      const int at = prm.pops->at[t];
      sMD[t] = H.pd[t];
      sAt[t] = (at >> 4) * (NEQ * EPB * NP) + (at & 15);
    }
    for (int t = tid; t < ND; t += NT) sMD[ND * NTERM + t] = H.pm[t];
    for (int t = tid; t < NFPE * ND; t += NT) sMB[t] = H.pb[t];
  } else {
    for (int t = tid; t < (G == 2 ? DIM * ND * ND : N1 * N1); t += NT) sMD[t] = H.md[t];
    for (int t = tid; t < (G == 2 ? NFPE * NQF * ND : 2 * N1); t += NT) sMB[t] = H.mb[t];
  }
  R gamma = (R)prm.gamma, cov = (R)prm.covolume;
  bool live = sl < EPB && e < ne;
  double dts = 1.0;
  float2 dts2 = make_float2(1.0f, 0.0f);
  if (prm.act_cum) {
    const int na = *prm.act_n;
    live = sl < EPB && e < prm.act_cum[na];
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
  const long long own = (long long)e * ND + i;
  R lmax = R(0), idet = R(0), acc[NEQ];
#pragma unroll
  for (int k = 0; k < NEQ; ++k) acc[k] = R(0);
  if (live) {
    R st[NEQ];
#pragma unroll
    for (int k = 0; k < NEQ; ++k) st[k] = u[k * NDa + own];
    // contravariant flux at the node
    const R* ng = (const R*)prm.ngeo;  // per-node geometry (bilinear quads) or null
    R adj[DIM][DIM];
#pragma unroll
    for (int r = 0; r < DIM; ++r)
#pragma unroll
      for (int d = 0; d < DIM; ++d)
        adj[r][d] = ng ? ng[((long long)(r * DIM + d) * ND + i) * ne + e]
                       : ((const R*)prm.egeo)[(long long)(r * DIM + d) * ne + e];
    idet = ng ? ng[((long long)(DIM * DIM) * ND + i) * ne + e]
              : ((const R*)prm.egeo)[(long long)(DIM * DIM) * ne + e];
    if constexpr (PLAIN) {
      R F[NEQ][DIM];
      lmax = flux_and_speed<DIM>(st, F, gamma, cov);
#pragma unroll
      for (int r = 0; r < DIM; ++r)
#pragma unroll
        for (int k = 0; k < NEQ; ++k) sG[r][k][sl * NP + i] = fmaf(adj[r][1], F[k][1], adj[r][0] * F[k][0]);
    } else {
      const NodeFlux<DIM, R> N(st, gamma, cov);
      lmax = N.speed;
#pragma unroll
      for (int r = 0; r < DIM; ++r) {
        R G[NEQ];
        N.contra(st, adj[r], G);
#pragma unroll
        for (int k = 0; k < NEQ; ++k) sG[r][k][sl * NP + i] = G[k];
      }
    }
  }
  __syncthreads();
  if (live) {
    // faces: the slot of each, its side and direction
    const R* fx = (const R*)prm.fslot;
    const long long nf = (long long)prm.nface * NQF;
    if constexpr (G == 3) {
      const int jx = i % N1, jy = i / N1;
      // (the volume before the faces but in PLAIN's order)
#pragma unroll
      for (int m = 0; m < (PLAIN ? 0 : N1); ++m) {
        const R d0 = sMD[jx * N1 + m], d1 = sMD[jy * N1 + m];
#pragma unroll
        for (int k = 0; k < NEQ; ++k)
          acc[k] += d0 * sG[0][k][sl * NP + m + N1 * jy] + d1 * sG[1][k][sl * NP + jx + N1 * m];
      }
#pragma unroll
      for (int lf = 0; lf < NFPE; ++lf) {
        const int ref = prm.fref[lf * ne + e];
        const int t = (lf & 1) ? jy : jx;
        int q = lf >= 2 ? N1 - 1 - t : t;
        if (ref & 1) q = N1 - 1 - q;
        const R b = PLAIN ? sMB[lf * ND + i] : sMB[quad_face_side(lf) * N1 + ((lf & 1) ? jx : jy)];
        const R c = (ref & 2) ? b : -b;
        const R* p = fx + (long long)ref_face(ref) * NQF + q;
#pragma unroll
        for (int k = 0; k < NEQ; ++k) acc[k] += c * p[k * nf];
      }
      if constexpr (PLAIN) {
        const R* g = &sG[0][0][sl * NP];
#pragma unroll
        for (int o = 0; o < NTERM; ++o) {
          const R d = sMD[i * NTERM + o];
          const int at = sAt[i * NTERM + o];
#pragma unroll
          for (int k = 0; k < NEQ; ++k) acc[k] += d * g[k * EPB * NP + at];
        }
      }
    } else {
#pragma unroll
      for (int lf = 0; lf < NFPE; ++lf) {
        const int ref = prm.fref[lf * ne + e];
        const R* p = fx + (long long)ref_face(ref) * NQF;
#pragma unroll
        for (int q = 0; q < NQF; ++q) {
          const R b = sMB[(lf * NQF + q) * ND + i];
          const R c = (ref & 2) ? b : -b;
          const int qf = (ref & 1) ? NQF - 1 - q : q;
#pragma unroll
          for (int k = 0; k < NEQ; ++k) acc[k] += c * p[k * nf + qf];
        }
      }
#pragma unroll
      for (int m = 0; m < ND; ++m) {
        const R d0 = sMD[m * ND + i], d1 = sMD[(ND + m) * ND + i];
#pragma unroll
        for (int k = 0; k < NEQ; ++k)
          acc[k] += d0 * sG[0][k][sl * NP + m] + d1 * sG[1][k][sl * NP + m];
      }
    }
    if (prm.ncidx) {  // hanging faces of a nonconforming mesh
      const int ix = prm.ncidx[e];
      if (ix >= 0) {
        const R* xf = (const R*)prm.xface + (long long)ix * NEQ * ND;
        if constexpr (PLAIN) {
#pragma unroll
          for (int k = 0; k < NEQ; ++k) acc[k] += xf[k * ND + i];
        } else {
          for (int j = 0; j < ND; ++j) {
            const R m = (R)prm.tab->Minv[i][j];
#pragma unroll
            for (int k = 0; k < NEQ; ++k) acc[k] += m * xf[k * ND + j];
          }
        }
      }
    }
    if constexpr (PLAIN) {
#pragma unroll
      for (int k = 0; k < NEQ; ++k) acc[k] *= sMD[ND * NTERM + i];
    }
  }
  const bool need_means = ep.mode == 1 && (ep.means || ep.means32);
  if (need_means) __syncthreads();  // every thread has read sG
  if (live) {
#pragma unroll
    for (int k = 0; k < NEQ; ++k) {
      R hi, lo;
      epi_node<R>(ep, k * NDa + own, acc[k] * idet, dts, dts2, hi, lo);
      if (need_means) {
        sG[0][k][sl * NP + i] = hi;
        sG[1][k][sl * NP + i] = lo;
      }
    }
  }
  if (need_means) {
    // cell means, one (element, equation) per thread and round
    __shared__ int sE[EPB];
    if (i == 0 && sl < EPB) sE[sl] = live ? e : -1;
    __syncthreads();
    for (int t = tid; t < EPB * NEQ; t += NT) {
      const int k = t / EPB, s = t - k * EPB, em = sE[s];
      if (em < 0) continue;
      const double* we = prm.tab->wmn_e ? prm.tab->wmn_e + (long long)em * ND : nullptr;
      if constexpr (std::is_same<R, double>::value) {
        double m = 0.0;
#pragma unroll
        for (int j = 0; j < ND; ++j) m += (we ? we[j] : H.wm[j]) * sG[0][k][s * NP + j];
        store_mean(ep, (long long)k * ne + em, m);
      } else {
        float mh = 0.0f, ml = 0.0f, ph, pl;
#pragma unroll
        for (int j = 0; j < ND; ++j) {
          const float w = we ? (float)we[j] : H.wm[j];
          ds_mul_f(w, 0.0f, sG[0][k][s * NP + j], ph, pl);
          ds_add(mh, ml, ph, pl);
          if (ep.final_stage) ds_add(mh, ml, w * sG[1][k][s * NP + j], 0.0f);
        }
        if (ep.means32)
          ep.means32[(long long)k * ne + em] = make_float2(mh, ml);
        else
          ep.means[(long long)k * ne + em] = (double)mh + (double)ml;
      }
    }
  }
  constexpr bool SQ = std::is_same<R, double>::value;
  if (prm.prob)
    segmented_max_commit<R, SQ>(lmax, live ? pb : -1, prm.pmcs);
  else
    block_max_commit<R, SQ>(lmax, prm.mcs);
}

}  // namespace rkdg
