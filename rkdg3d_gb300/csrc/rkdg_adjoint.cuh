// Discrete adjoint (vector-Jacobian products) of the FP64 right-hand side and
// limiter.
//
// Right-hand side y = M^-1 z(u): given k_bar, r = M^-1 k_bar (M symmetric),
// then u_bar = (dz/du)^T r with
//   volume  z_j += sum_m sum_r D[r][j][m] G_r(u_m),  G_r = sum_d adj(J)[r][d] F_d
//           -> u_bar_m += (dF_d/du)^T (sum_r adj[r][d] sum_j D[r][j][m] r_j)
//   faces   z_e1 -= w|J| Fhat B1,  z_e2 += w|J| Fhat B2
//           -> Fhat_bar = w|J| (-B1 r_e1 + B2 r_e2),
//              u_bar_own += B_own (dFhat/du_own)^T Fhat_bar
// in two passes without atomics: a thread per face point takes Fhat_bar back
// through the numerical flux to both sides' traces in one reverse sweep
// (rkdg_flux_vjp.cuh; boundary faces with their ghost state in forward mode,
// Dual<NEQ>), and a thread per element node gathers the points of its faces
// and adds the nodal flux's share.  20^3 Q1 hexahedra, HLLC with TRRS speeds:
// 0.39 ms against 4.46 ms for one thread per element with Dual<5> through every
// flux, once per side, spilling 2 KB a thread.
//
// Limiter (Multi, BJ-family indicator): the limited values are
// v_i = mean + m^nd (u_i - mean) (the nd-fold application of
// limiter_multiplier.cpp:24-38), m = density indicator.  The indicator is
// recomputed and differentiated at its minimising point; the derivative with
// respect to a neighbour's mean is stored per element and gathered by the
// neighbour.
#pragma once

#include "rkdg_common.h"
#include "rkdg_dual.cuh"
#include "rkdg_flux_vjp.cuh"
#include "rkdg_generic.cuh"
#include "rkdg_hex_faces.cuh"
#include "rkdg_limit.cuh"
#include "rkdg_physics.cuh"

namespace rkdg {

// r = M^-1 k_bar (reference inverse mass / det J), one thread per value; the
// mass matrix is diagonal but on triangles.
template <int G, int P>
__global__ void k_minv_apply(int ne, long long ndofs, const RefTables* tab, const double* egeo,
                             const double* __restrict__ kb, double* __restrict__ r) {
  using E = El<G, P>;
  constexpr int ND = E::ND, DIM = E::DIM;
  const long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (v >= ndofs) return;
  const int e = (int)(v / ND), i = (int)(v - (long long)e * ND);
  const double* ng = tab->ngeo_e;  // bilinear quads: 1/det J per node
  const double idet = ng ? ng[((long long)(DIM * DIM) * ND + i) * ne + e] : egeo[(long long)(DIM * DIM) * ne + e];
#pragma unroll
  for (int k = 0; k < E::NEQ; ++k) {
    double s = 0.0;
    if constexpr (G == 2) {
#pragma unroll
      for (int j = 0; j < ND; ++j) s += tab->Minv[j][i] * kb[k * ndofs + (long long)e * ND + j];
    } else {
      s = tab->Minv[i][i] * kb[k * ndofs + v];
    }
    r[k * ndofs + v] = s * idet;
  }
}

// Threads and elements of a node-pass CTA.
template <int G, int P>
struct VjpSize {
  static constexpr int NT = Planar<G, P>::NT, EPB = Planar<G, P>::EPB;
};
template <int P>
struct VjpSize<5, P> {
  static constexpr int NT = HexFaces<P>::NTN, EPB = HexFaces<P>::EPB;
};

// Trace of a field at point q of local face lf of element e.
template <int G, int P>
__device__ __forceinline__ void vjp_trace(const double* __restrict__ f, long long NDa, int e, int lf,
                                          int q, const double* sB, double* v) {
  using E = El<G, P>;
  constexpr int ND = E::ND, NEQ = E::NEQ, NQF = E::NQF, N1 = P + 1;
  const double* fe = f + (long long)e * ND;
  const double* B = sB + (lf * NQF + q) * ND;
  if constexpr (G == 3) {  // the line of nodes behind the point
    const int i0 = quad_face_node<N1>(lf, q, 0), st = (lf & 1) ? 1 : N1;
#pragma unroll
    for (int k = 0; k < NEQ; ++k) {
      double s = 0.0;
#pragma unroll
      for (int j = 0; j < N1; ++j) s += B[i0 + j * st] * fe[k * NDa + i0 + j * st];
      v[k] = s;
    }
  } else {
#pragma unroll
    for (int k = 0; k < NEQ; ++k) v[k] = 0.0;
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      const double b = B[j];
#pragma unroll
      for (int k = 0; k < NEQ; ++k) v[k] += b * fe[k * NDa + j];
    }
  }
}

// Interior faces, one thread per point of Elem1's face rule: the cotangents of
// both sides' traces to gb[side][k][face * NQF + q].
template <int G, int P>
__global__ void __launch_bounds__(128)
    k_face_vjp(const __grid_constant__ RhsParams prm, const double* __restrict__ u,
               const double* __restrict__ r, double* __restrict__ gb) {
  using E = El<G, P>;
  constexpr int DIM = E::DIM, ND = E::ND, NEQ = E::NEQ, NFPE = E::NFPE, NQF = E::NQF;
  __shared__ double sB[NFPE * NQF * ND];
  const RefTables* T = prm.tab;
  for (int t = threadIdx.x; t < NFPE * NQF * ND; t += blockDim.x)
    sB[t] = T->B[t / (NQF * ND)][(t / ND) % NQF][t % ND];
  __syncthreads();
  const long long npt = (long long)prm.nface * NQF, t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= npt) return;
  const int f = (int)(t / NQF), q = (int)(t - (long long)f * NQF), ne = prm.ne;
  const int4 fc = prm.flist[f];
  if (fc.y < 0) return;  // k_bface_vjp
  const int lf1 = fc.z & 7, lf2 = (fc.z >> 3) & 7;
  const int q2 = T->perm[prm.fcode[lf1 * ne + fc.x] >> 4][q];
  const double* fg = (const double*)prm.fgeo + (long long)(lf1 * (DIM + 1)) * ne + fc.x;
  double n[DIM], s1[NEQ], s2[NEQ], fb[NEQ], g1[NEQ], g2[NEQ];
#pragma unroll
  for (int c = 0; c < DIM; ++c) n[c] = fg[(long long)c * ne];
  const double w = T->wf[q] * fg[(long long)DIM * ne];
  vjp_trace<G, P>(r, prm.ndofs, fc.x, lf1, q, sB, s1);
  vjp_trace<G, P>(r, prm.ndofs, fc.y, lf2, q2, sB, s2);
#pragma unroll
  for (int k = 0; k < NEQ; ++k) fb[k] = w * (s2[k] - s1[k]);
  vjp_trace<G, P>(u, prm.ndofs, fc.x, lf1, q, sB, s1);
  vjp_trace<G, P>(u, prm.ndofs, fc.y, lf2, q2, sB, s2);
  riemann_vjp<DIM>(s1, s2, n, fb, prm.gamma, prm.covolume, prm.rs, prm.avg, g1, g2);
#pragma unroll
  for (int k = 0; k < NEQ; ++k) {
    gb[k * npt + t] = g1[k];
    gb[(NEQ + k) * npt + t] = g2[k];
  }
}

// Boundary faces: forward mode through the ghost state and the flux; zero
// where the face carries no integrator.
template <int G, int P>
__global__ void __launch_bounds__(64)
    k_bface_vjp(const __grid_constant__ RhsParams prm, const double* __restrict__ u,
                const double* __restrict__ r, double* __restrict__ gb) {
  using E = El<G, P>;
  constexpr int DIM = E::DIM, ND = E::ND, NEQ = E::NEQ, NQF = E::NQF;
  using D = Dual<NEQ>;
  const RefTables* T = prm.tab;
  const long long npt = (long long)prm.nface * NQF, t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= npt) return;
  const int f = (int)(t / NQF), q = (int)(t - (long long)f * NQF), ne = prm.ne;
  const int4 fc = prm.flist[f];
  if (fc.y >= 0) return;
  const int e = fc.x, lf = fc.z & 7, nb = prm.fnbr[lf * ne + e];
  double g[NEQ];
  for (int k = 0; k < NEQ; ++k) g[k] = 0.0;
  if (nb != -1) {
    const double* fg = (const double*)prm.fgeo + (long long)(lf * (DIM + 1)) * ne + e;
    const double* B = T->B[lf][q];
    const D gamma = D(prm.gamma), cov = D(prm.covolume);
    D n[DIM], s1[NEQ], s2[NEQ], F[NEQ];
    double fb[NEQ];
    for (int c = 0; c < DIM; ++c) n[c] = D(fg[(long long)c * ne]);
    const double w = T->wf[q] * fg[(long long)DIM * ne];
    for (int k = 0; k < NEQ; ++k) {
      double v = 0.0, rv = 0.0;
      for (int s = 0; s < ND; ++s) {
        v += u[k * prm.ndofs + (long long)e * ND + s] * B[s];
        rv += r[k * prm.ndofs + (long long)e * ND + s] * B[s];
      }
      s1[k] = D::var(v, k);
      fb[k] = -w * rv;
    }
    const BCSlot& bc = prm.bc[-2 - nb];
    right_state<DIM>(bc.type, bc.state, s1, s2, n, gamma, cov, D(prm.rgas));
    riemann<DIM>(s1, s2, n, F, gamma, cov, prm.rs, prm.avg);
    for (int kk = 0; kk < NEQ; ++kk)
      for (int k = 0; k < NEQ; ++k) g[kk] += fb[k] * F[k].d[kk];
  }
  for (int k = 0; k < NEQ; ++k) gb[k * npt + t] = g[k];
}

// One thread per element node: the traces' cotangents of the element's faces
// and the nodal flux's.
template <int G, int P>
__global__ void __launch_bounds__(VjpSize<G, P>::NT)
    k_node_vjp(const __grid_constant__ RhsParams prm, const double* __restrict__ u,
               const double* __restrict__ r, const double* __restrict__ gb, double* __restrict__ ubar) {
  using E = El<G, P>;
  using S = VjpSize<G, P>;
  constexpr int DIM = E::DIM, ND = E::ND, NEQ = E::NEQ, NFPE = E::NFPE, NQF = E::NQF, N1 = P + 1;
  constexpr int NP = ND | 1, EPB = S::EPB;
  __shared__ double sR[NEQ][EPB * NP], sB[NFPE * NQF * ND], sD[G == 2 ? DIM * ND * ND : N1 * N1];
  const RefTables* T = prm.tab;
  const int tid = threadIdx.x, ne = prm.ne;
  const long long NDa = prm.ndofs, npt = (long long)prm.nface * NQF;
  for (int t = tid; t < NFPE * NQF * ND; t += S::NT) sB[t] = T->B[t / (NQF * ND)][(t / ND) % NQF][t % ND];
  if constexpr (G == 2) {
    for (int t = tid; t < DIM * ND * ND; t += S::NT) sD[t] = T->D[t / (ND * ND)][(t / ND) % ND][t % ND];
  } else {
    for (int t = tid; t < N1 * N1; t += S::NT) sD[t] = T->d1[t / N1][t % N1];
  }
  const int sl = tid / ND, i = tid - sl * ND, e = blockIdx.x * EPB + sl;
  const bool live = sl < EPB && e < ne;
  const long long own = (long long)e * ND + i;
  if (live) {
#pragma unroll
    for (int k = 0; k < NEQ; ++k) sR[k][sl * NP + i] = r[k * NDa + own];
  }
  __syncthreads();
  if (!live) return;
  double acc[NEQ];
#pragma unroll
  for (int k = 0; k < NEQ; ++k) acc[k] = 0.0;
  for (int lf = 0; lf < NFPE; ++lf) {
    const int ref = prm.fref[G == 5 ? (long long)e * 8 + lf : (long long)lf * ne + e], code = prm.fcode[lf * ne + e];
    const int f = G == 5 ? ref >> 1 : ref_face(ref), side = G == 5 ? ref & 1 : (ref >> 1) & 1;
    const double* g = gb + (long long)side * NEQ * npt + (long long)f * NQF;
    const int* pm = T->perm[code >> 4];
    if constexpr (G == 3) {  // one point of the face sees this node
      const int t = (lf & 1) ? i / N1 : i % N1;
      const int q = lf >= 2 ? N1 - 1 - t : t;
      const double b = sB[(lf * NQF + q) * ND + i];
      const int q1 = (ref & 1) ? NQF - 1 - q : q;
#pragma unroll
      for (int k = 0; k < NEQ; ++k) acc[k] += b * g[k * npt + q1];
    } else {
      for (int q1 = 0; q1 < NQF; ++q1) {
        const int q = side ? pm[q1] : q1;
        const double b = sB[(lf * NQF + q) * ND + i];
#pragma unroll
        for (int k = 0; k < NEQ; ++k) acc[k] += b * g[k * npt + q1];
      }
    }
  }
  // volume: the contravariant components' cotangents, then the flux's
  double gbar[NEQ][DIM];
  if constexpr (G == 2) {
#pragma unroll
    for (int k = 0; k < NEQ; ++k)
#pragma unroll
      for (int rr = 0; rr < DIM; ++rr) {
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < ND; ++j) s += sD[(rr * ND + j) * ND + i] * sR[k][sl * NP + j];
        gbar[k][rr] = s;
      }
  } else {
    const int m[3] = {i % N1, (i / N1) % N1, DIM == 3 ? i / (N1 * N1) : 0};
    const double w[3] = {T->w1[m[0]], T->w1[m[1]], DIM == 3 ? T->w1[m[2]] : 1.0};
    const int st[3] = {1, N1, N1 * N1};
#pragma unroll
    for (int rr = 0; rr < DIM; ++rr) {
      const double wo = rr == 0 ? w[1] * w[2] : (rr == 1 ? w[0] * w[2] : w[0] * w[1]);
      const int b = sl * NP + i - m[rr] * st[rr];
#pragma unroll
      for (int k = 0; k < NEQ; ++k) {
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < N1; ++j) s += sD[j * N1 + m[rr]] * sR[k][b + j * st[rr]];
        gbar[k][rr] = wo * s;
      }
    }
  }
  const double* ng = T->ngeo_e;  // bilinear quads: adj(J) at the node
  double fb[NEQ][DIM], st[NEQ], g[NEQ];
#pragma unroll
  for (int d = 0; d < DIM; ++d)
#pragma unroll
    for (int k = 0; k < NEQ; ++k) fb[k][d] = 0.0;
#pragma unroll
  for (int rr = 0; rr < DIM; ++rr)
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const double a = ng ? ng[((long long)(rr * DIM + d) * ND + i) * ne + e]
                          : ((const double*)prm.egeo)[(long long)(rr * DIM + d) * ne + e];
#pragma unroll
      for (int k = 0; k < NEQ; ++k) fb[k][d] += a * gbar[k][rr];
    }
#pragma unroll
  for (int k = 0; k < NEQ; ++k) st[k] = u[k * NDa + own];
  flux_vjp<DIM>(st, fb, prm.gamma, prm.covolume, g);
#pragma unroll
  for (int k = 0; k < NEQ; ++k) ubar[k * NDa + own] = acc[k] + g[k];
}

// Hanging faces of a nonconforming mesh (see rkdg_nc.cu).  The element VJP
// above skips them (they carry no integrator of their own); here, per slave
// point q, Fhat_bar = w_q |J_f| (-B1 r_fine + Bc r_coarse) and, in one reverse
// sweep through the flux, g_side = (dFhat/du_side)^T Fhat_bar
// (k_nc_vjp_point, stored [face][q][side][k]); k_nc_vjp_gather then adds
// phi_j(q) g_side over each touched element's slave faces to u_bar.
template <int G, int P>
__global__ void __launch_bounds__(64)
    k_nc_vjp_point(const RhsParams prm, const NcParams nc, const double* __restrict__ u,
                   const double* __restrict__ r) {
  using E = El<G, P>;
  constexpr int DIM = E::DIM, ND = E::ND, NEQ = E::NEQ, NQF = E::NQF;
  const RefTables* T = prm.tab;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nc.nnc * NQF) return;
  const int f = t / NQF, q = t - f * NQF;
  const int e1 = nc.face[f * 4], lf1 = nc.face[f * 4 + 1], e2 = nc.face[f * 4 + 2];
  const int ne = prm.ne;
  const long long NDa = prm.ndofs;
  const double* fg = (const double*)prm.fgeo;
  double n[DIM];
  for (int c = 0; c < DIM; ++c) n[c] = fg[(long long)(lf1 * (DIM + 1) + c) * ne + e1];
  const double jac = fg[(long long)(lf1 * (DIM + 1) + DIM) * ne + e1];
  const double* B1 = T->B[lf1][q];
  const double* B2 = nc.bnc + ((long long)f * NQF + q) * ND;
  double v1[NEQ], v2[NEQ], fbar[NEQ];
  for (int k = 0; k < NEQ; ++k) {
    double a = 0.0, b = 0.0, ra = 0.0, rb = 0.0;
    for (int s = 0; s < ND; ++s) {
      a += u[k * NDa + (long long)e1 * ND + s] * B1[s];
      ra += r[k * NDa + (long long)e1 * ND + s] * B1[s];
      b += u[k * NDa + (long long)e2 * ND + s] * B2[s];
      rb += r[k * NDa + (long long)e2 * ND + s] * B2[s];
    }
    v1[k] = a;
    v2[k] = b;
    fbar[k] = T->wf[q] * jac * (-ra + rb);
  }
  double* g = (double*)nc.flux + ((long long)f * NQF + q) * 2 * NEQ;
  double g1[NEQ], g2[NEQ];
  riemann_vjp<DIM>(v1, v2, n, fbar, prm.gamma, prm.covolume, prm.rs, prm.avg, g1, g2);
  for (int kk = 0; kk < NEQ; ++kk) {
    g[kk] = g1[kk];
    g[NEQ + kk] = g2[kk];
  }
}

template <int G, int P>
__global__ void __launch_bounds__(128)
    k_nc_vjp_gather(const NcParams nc, const RefTables* __restrict__ T, long long NDa,
                    double* __restrict__ ubar) {
  using E = El<G, P>;
  constexpr int ND = E::ND, NEQ = E::NEQ, NQF = E::NQF;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nc.nel * ND) return;
  const int i = t / ND, j = t - i * ND;
  double s[NEQ];
  for (int k = 0; k < NEQ; ++k) s[k] = 0.0;
  const double* gb = (const double*)nc.flux;
  for (int c = nc.ptr[i]; c < nc.ptr[i + 1]; ++c) {
    const int f = nc.ent[c] >> 1, side = nc.ent[c] & 1;
    const int lf1 = nc.face[f * 4 + 1];
    for (int q = 0; q < NQF; ++q) {
      const double phi = side ? nc.bnc[((long long)f * NQF + q) * ND + j] : T->B[lf1][q][j];
      const double* g = gb + (((long long)f * NQF + q) * 2 + side) * NEQ;
      for (int k = 0; k < NEQ; ++k) s[k] += phi * g[k];
    }
  }
  const int e = nc.elem[i];
  for (int k = 0; k < NEQ; ++k) ubar[k * NDa + (long long)e * ND + j] += s[k];
}

// The limiter's stencil of element e (limiter.cpp:95-123): its face
// neighbours, then the elements across its hanging faces (nonconforming
// meshes).  stencil_size / stencil_at enumerate it; an entry is -1 where a
// face has no neighbour.
__device__ __forceinline__ int lim_ncrow(const LimParams& prm, int e) {
  return prm.ncidx ? prm.ncidx[e] : -1;
}
__device__ __forceinline__ int stencil_size(const LimParams& prm, int row, int nfpe) {
  return nfpe + (row >= 0 ? prm.nc_ptr[row + 1] - prm.nc_ptr[row] : 0);
}
__device__ __forceinline__ int stencil_at(const LimParams& prm, int e, int row, int nfpe, int i) {
  if (i < nfpe) return prm.fnbr[i * prm.ne + e];
  const int ent = prm.nc_ent[prm.nc_ptr[row] + i - nfpe];
  return prm.nc_face[(ent >> 1) * 4 + ((ent & 1) ? 0 : 2)];
}
// Local faces of e that are slave or master faces: they carry indicator
// points although no conforming neighbour lies across them.
__device__ __forceinline__ unsigned hanging_faces(const LimParams& prm, int row) {
  unsigned m = 0;
  if (row >= 0)
    for (int c = prm.nc_ptr[row]; c < prm.nc_ptr[row + 1]; ++c) {
      const int f = prm.nc_ent[c] >> 1, side = prm.nc_ent[c] & 1;
      m |= 1u << prm.nc_face[f * 4 + (side ? 3 : 1)];
    }
  return m;
}

// Limiter VJP, own part, with the forward limiter's threads per element
// (LimTeam).  The indicator is a minimum over face points, so its gradient is
// that of one point: the group finds the point (the first in order on ties, as
// the forward minimum keeps it) and differentiates the limiter function there in
// reverse, (d y_c/d y) (d y/d diff) times the point's row of basis values.
// Likewise the stencil's minimum and maximum are each one element's mean; the
// derivative with respect to them goes to cross[0..3][e] = (argmin element or -1
// for e itself, d/dmin, argmax element or -1, d/dmax), which k_limit_vjp_gather
// hands to those elements.  A thread per element that carried Dual<ND + 3>
// through every point took 205 us on 20^3 Q1 hexahedra, spilling; this one about
// 60.
template <int G, int P>
struct LimVjp {
  using E = El<G, P>;
  static constexpr int L = LimTeam<G, P>::L, NDP = LimTeam<G, P>::NDP;
  // threads per CTA: the values and their cotangents within 30 KB
  static constexpr int NT = 2 * 8 * E::NEQ * NDP * (128 / L) > 30000 ? 64 : 128;
  static constexpr int EPB = NT / L;
};

template <int G, int P>
__global__ void __launch_bounds__(LimVjp<G, P>::NT)
    k_limit_vjp(const LimParams prm, const double* __restrict__ z, const double* __restrict__ ybar,
                double* __restrict__ zbar, double* __restrict__ cross) {
  using E = El<G, P>;
  using S = LimVjp<G, P>;
  constexpr int DIM = E::DIM, ND = E::ND, NEQ = E::NEQ, NFPE = E::NFPE, NQL = E::NQL, NV = E::NV;
  constexpr int L = S::L, NDP = S::NDP, NT = S::NT, EPB = S::EPB, NPT = NFPE * NQL;
  __shared__ double sU[NEQ][EPB][NDP], sY[NEQ][EPB][NDP];  // values, cotangents
  __shared__ double sBl[ND][NPT], sBv[ND][NV];
  __shared__ double sM[NEQ][EPB], sSy[NEQ][EPB];  // means, sums of cotangents
  // factor m^nd, d/d(values) = sGu * basis row sPt, d/d(own mean)
  __shared__ double sMnd[EPB], sGu[EPB], sGm[EPB];
  __shared__ int sPt[EPB];
  const RefTables* T = prm.tab;
  const int ne = prm.ne, tid = threadIdx.x, e0 = blockIdx.x * EPB;
  const int nel = min(EPB, ne - e0);
  const long long NDa = prm.ndofs;
  for (int t = tid; t < ND * NPT; t += NT) {
    const int j = t / NPT, pt = t - j * NPT;
    sBl[j][pt] = T->Bl[pt / NQL][pt % NQL][j];
  }
  for (int t = tid; t < ND * NV; t += NT) sBv[t / NV][t % NV] = T->Bv[t % NV][t / NV];
  for (int t = tid; t < NEQ * EPB; t += NT) {
    const int k = t / EPB, s = t - k * EPB;
    if (s < nel) sM[k][s] = prm.means[(long long)k * ne + e0 + s];
  }
  for (int t = tid; t < nel * ND; t += NT) {
    const int s = t / ND, j = t - s * ND;
#pragma unroll
    for (int k = 0; k < NEQ; ++k) {
      sU[k][s][j] = z[k * NDa + (long long)e0 * ND + t];
      sY[k][s][j] = ybar[k * NDa + (long long)e0 * ND + t];
    }
  }
  __syncthreads();
  const int slot = tid / L, lane = tid - slot * L;
  const bool on = slot < nel;
  const int e = e0 + slot;
  const bool multi = prm.limiter == 1;
  const int kind = multi ? 0 : NEQ - 1;  // the equation whose indicator counts
  double m = prm.indicator == 1 ? 0.0 : 1.0;
  double gu = 0.0, gm = 0.0, gmin = 0.0, gmax = 0.0;  // d m / d(values), own mean, min, max
  int ptmin = -1, amin = -1, amax = -1;
  if (prm.indicator >= 2) {
    const double own = on ? sM[kind][slot] : 0.0;
    double mI = own < 1e9 ? own : 1e9, MI = own > -1e9 ? own : -1e9;
    int imin = -1, imax = -1;  // places in the stencil, -1 the element itself
    unsigned inner = 0;
    if (on) {
      const int row = lim_ncrow(prm, e), nst = stencil_size(prm, row, NFPE);
      if (row >= 0) inner = hanging_faces(prm, row);
      for (int i = lane; i < nst; i += L) {
        const int nb = stencil_at(prm, e, row, NFPE, i);
        if (nb < 0) continue;
        if (i < NFPE) inner |= 1u << i;
        const double v = prm.means[(long long)kind * ne + nb];
        if (v < mI) mI = v, imin = i, amin = nb;
        if (v > MI) MI = v, imax = i, amax = nb;
      }
    }
    __syncwarp();
#pragma unroll
    for (int o = 1; o < L; o <<= 1) {  // the smaller (mean, place)
      const double a = __shfl_xor_sync(0xffffffffu, mI, o), b = __shfl_xor_sync(0xffffffffu, MI, o);
      const int ia = __shfl_xor_sync(0xffffffffu, imin, o), ib = __shfl_xor_sync(0xffffffffu, imax, o);
      const int na = __shfl_xor_sync(0xffffffffu, amin, o), nb = __shfl_xor_sync(0xffffffffu, amax, o);
      if (a < mI || (a == mI && ia < imin)) mI = a, imin = ia, amin = na;
      if (b > MI || (b == MI && ib < imax)) MI = b, imax = ib, amax = nb;
      inner |= __shfl_xor_sync(0xffffffffu, inner, o);
    }
    double yMin = 1e9;
    if (on)
      for (int pt = lane; pt < NPT; pt += L) {
        if (!((inner >> (pt / NQL)) & 1u)) continue;  // only interior faces carry indicator points
        double v = 0.0;
#pragma unroll
        for (int j = 0; j < ND; ++j) v += sU[kind][slot][j] * sBl[j][pt];
        const double diff = v - own;
        const bool up = diff > 1e-3, dn = diff < -1e-3;
        const double idiff = 1.0 / diff;
        const double y = up ? (MI - own) / diff : (dn ? (mI - own) / diff : 1.0);
        double yc, dy;  // limiter function and its derivative
        if (prm.function == 0) {
          yc = y <= 1.0 ? y : 1.0;
          dy = y <= 1.0 ? 1.0 : 0.0;
        } else if (prm.function == 1) {
          const double den = y * y + y + 2.0;
          yc = (y * y + 2.0 * y) / den;
          dy = (2.0 * y + 2.0 - yc * (2.0 * y + 1.0)) / den;
        } else {
          const double ys = 1.5;
          const double yr = y / ys;
          yc = y < 1.0 ? y + (3.0 - 2.0 * ys) * yr * yr + (ys - 2.0) * yr * yr * yr : 1.0;
          dy = y < 1.0 ? 1.0 + (2.0 * (3.0 - 2.0 * ys) * yr + 3.0 * (ys - 2.0) * yr * yr) / ys : 0.0;
        }
        if (yc < yMin) {
          yMin = yc;
          ptmin = pt;
          const double g = up || dn ? dy * idiff : 0.0;
          gu = -y * g;
          gm = (y - 1.0) * g;
          gmin = dn ? g : 0.0;
          gmax = up ? g : 0.0;
        }
      }
    // the smaller (value, point) of the group
    double yb = yMin;
    int pb = ptmin;
#pragma unroll
    for (int o = 1; o < L; o <<= 1) {
      const double a = __shfl_xor_sync(0xffffffffu, yb, o);
      const int p = __shfl_xor_sync(0xffffffffu, pb, o);
      if (a < yb || (a == yb && (unsigned)p < (unsigned)pb)) yb = a, pb = p;
    }
    m = yb;
    // point pt belongs to lane pt % L
    const int src = (tid & 31) - lane + (pb >= 0 ? pb % L : 0);
    gu = __shfl_sync(0xffffffffu, gu, src);
    gm = __shfl_sync(0xffffffffu, gm, src);
    gmin = __shfl_sync(0xffffffffu, gmin, src);
    gmax = __shfl_sync(0xffffffffu, gmax, src);
    ptmin = pb;
    // a minimum or maximum that is the element's own mean moves with it
    if (amin < 0 && own < 1e9) gm += gmin;
    if (amax < 0 && own > -1e9) gm += gmax;
  }
  for (int k = lane; k < NEQ; k += L) {
    double sy = 0.0;
    if (on)
      for (int i = 0; i < ND; ++i) sy += sY[k][slot][i];
    sSy[k][slot] = sy;
  }
  __syncwarp();
  double mnd = 1.0;  // FinDiff: as it is, or the mean
  double mbar = 0.0;
  if (multi) {
    const int reps = (prm.quirks & 1) ? 1 : ND;
    double pm1 = 1.0;  // m^(reps-1)
    for (int i = 1; i < reps; ++i) pm1 *= m;
    mnd = pm1 * m;
    int bad = 0;
    if (on && prm.last_hope)  // forward values at the vertices: the last-hope reset
      for (int v = lane; v < NV; v += L) {
        double fv[NEQ];
#pragma unroll
        for (int k = 0; k < NEQ; ++k) {
          const double um = sM[k][slot];
          double s = 0.0;
          for (int j = 0; j < ND; ++j) s += (um + mnd * (sU[k][slot][j] - um)) * sBv[j][v];
          fv[k] = s;
        }
        if (!state_is_physical<DIM>(fv, prm.gamma, prm.covolume)) bad = 1;
      }
    __syncwarp();
#pragma unroll
    for (int o = 1; o < L; o <<= 1) bad |= __shfl_xor_sync(0xffffffffu, bad, o);
    if (on && !bad && prm.indicator == 2)
      for (int k = lane; k < NEQ; k += L) {
        const double um = sM[k][slot];
        double s = 0.0;
        for (int i = 0; i < ND; ++i) s += sY[k][slot][i] * (sU[k][slot][i] - um);
        mbar += s;
      }
    __syncwarp();
#pragma unroll
    for (int o = 1; o < L; o <<= 1) mbar += __shfl_xor_sync(0xffffffffu, mbar, o);
    mbar *= reps * pm1;
    if (bad) mnd = 0.0, mbar = 0.0, amin = amax = -1;
  } else if (m < 0.999) {
    mnd = 0.0;
  }
  if (lane == 0) {
    const bool x = on && multi && prm.indicator == 2;
    sMnd[slot] = mnd;
    sGu[slot] = x && ptmin >= 0 ? mbar * gu : 0.0;
    sGm[slot] = x ? mbar * gm : 0.0;
    sPt[slot] = ptmin >= 0 ? ptmin : 0;
    if (on) {
      cross[e] = x ? amin : -1;
      cross[(long long)ne + e] = x ? mbar * gmin : 0.0;
      cross[2LL * ne + e] = x ? amax : -1;
      cross[3LL * ne + e] = x ? mbar * gmax : 0.0;
    }
  }
  __syncthreads();
  for (int t = tid; t < nel * ND; t += NT) {
    const int s = t / ND, j = t - s * ND;
    const double w = T->wmn_e ? T->wmn_e[(long long)e0 * ND + t] : T->wmean[j];
    const double mn = sMnd[s], own = w * (1.0 - mn);
#pragma unroll
    for (int k = 0; k < NEQ; ++k) {
      double r = own * sSy[k][s] + mn * sY[k][s][j];
      if (k == 0) r += sGu[s] * sBl[j][sPt[s]] + sGm[s] * w;
      zbar[k * NDa + (long long)e0 * ND + t] = r;
    }
  }
}

// Gather, for element c, the derivatives that the elements of its stencil
// (which hold c in theirs) took with respect to c's density mean (mean =
// sum_j w_j rho_j), each stencil element once.
template <int G, int P>
__global__ void k_limit_vjp_gather(const LimParams prm, const double* __restrict__ cross,
                                   double* __restrict__ zbar) {
  using E = El<G, P>;
  constexpr int ND = E::ND, NFPE = E::NFPE;
  const int ne = prm.ne;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ne) return;
  const int row = lim_ncrow(prm, c);
  const int nst = stencil_size(prm, row, NFPE);
  double s = 0.0;
  for (int i = 0; i < nst; ++i) {
    const int e = stencil_at(prm, c, row, NFPE, i);
    if (e < 0 || e == c) continue;
    bool seen = false;
    for (int i2 = 0; i2 < i && !seen; ++i2) seen = stencil_at(prm, c, row, NFPE, i2) == e;
    if (seen) continue;
    if (cross[e] == (double)c) s += cross[(long long)ne + e];
    if (cross[(long long)2 * ne + e] == (double)c) s += cross[(long long)3 * ne + e];
  }
  if (s != 0.0)
    for (int j = 0; j < ND; ++j)
      zbar[(long long)c * ND + j] +=
          (prm.tab->wmn_e ? prm.tab->wmn_e[(long long)c * ND + j] : prm.tab->wmean[j]) * s;
}

}  // namespace rkdg
