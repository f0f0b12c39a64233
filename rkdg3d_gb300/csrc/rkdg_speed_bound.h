// Upper bound of a face point's wave speed in FP32.
//
// The initial time step needs the largest wave speed of an FP64 state over all
// face points.  k_face_planar<SPEED> and k_speed_hex form both traces of a point
// in FP32 first and leave the point there if the speed that the FP64 evaluation
// can give at most lies below the largest FP64 speed found so far.  So the bound
// has to hold for whatever rounding did to the traces:
//   - a trace summed in FP32 from nodal values cut to FP32 errs by less than
//     kTraceErr times the largest nodal value: a cut of 1.2e-7, and 6e-8 for each
//     table entry, product and sum (7 in one sum of up to six terms, 12 in the
//     three sums of a hexahedron) times the Lebesgue sum of the row, at most
//     5.1 (order 2 hexahedra): 4.3e-6;
//   - every quantity carries the error that follows from it, to first order with
//     a tenth on top, and no error above a tenth is accepted;
//   - the normal velocity is n . u, not taken through a rotation: 1 - n_z^2
//     cancels in FP32 for normals close to the z axis.  The FP64 rotation itself
//     departs from n . u by at most 1e-6 |u| (its degenerate branch);
//   - a TRRS star pressure is bounded through its power 2 gamma/(gamma - 1),
//     whatever that is.
// The results are intervals of SL and SR; HLLC's signed max(SL, SR) must not be
// negative (an error that only the FP64 evaluation reports).
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define RKDG_HD __host__ __device__ __forceinline__
#else
#define RKDG_HD inline
#endif

namespace rkdg {

constexpr float kTraceErr = 6e-6f;
constexpr float kNoBound = 1e30f;

// division and square root to 2 ulp
RKDG_HD float bdiv(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fdividef(a, b);
#else
  return a / b;
#endif
}

RKDG_HD float bsqrt(float x) {
#ifdef __CUDA_ARCH__
  return x > 0.0f ? x * rsqrtf(x) : 0.0f;
#else
  return sqrtf(x);
#endif
}

// A side of the face in FP32: normal velocity, |u| and sound speed with their
// errors, and the relative errors of density and pressure.
struct SpeedSide {
  float r, u, v, du, c, dc, p, er, ep;
};

// s: the trace, top[k * stride]: the largest nodal |value| of variable k.
// False where nothing can be said.
template <int DIM>
RKDG_HD bool speed_side(const float* s, const float* top, int stride, const float* n, float gamma, float b,
                        SpeedSide& S) {
  const float r = s[0], E = s[1 + DIM];
  if (!(r > 1e-15f && r < 1e15f && E > 1e-15f && E < 1e15f && gamma - 1.0f > 0.01f)) return false;
  float m2 = 0.0f, mn = 0.0f, mt = 0.0f;
  for (int d = 0; d < DIM; ++d) {
    m2 += s[1 + d] * s[1 + d];
    mn += n[d] * s[1 + d];
    mt = fmaxf(mt, top[(1 + d) * stride]);
  }
  const float ir = bdiv(1.0f, r), m = bsqrt(m2), dm = (DIM == 3 ? 1.7321f : 1.4143f) * kTraceErr * mt;
  const float er = kTraceErr * top[0] * ir, ee = bdiv(kTraceErr * top[(1 + DIM) * stride], E);
  const float re = r * E, ie = re - 0.5f * m2, f = 1.0f - r * b;  // ie: rho times the internal energy
  if (!(ie >= 0.02f * re && f >= 0.5f)) return false;
  const float ei = bdiv(re * (er + ee + 1e-6f) + (m + dm) * dm, ie);
  const float ef = bdiv(r * fabsf(b) * er, f) + 1e-6f;  // of 1 - rho b
  const float e2 = ei + 2.0f * (er + ef);               // of c^2 = gamma (gamma - 1) ie / (rho (1 - rho b))^2
  if (!(e2 < 0.1f)) return false;
  const float g = bdiv(ir, f);
  S.r = r;
  S.u = mn * ir;
  S.v = m * ir;
  S.du = 1.2f * (dm * ir + S.v * er) + 3e-6f * S.v;
  S.c = bsqrt(gamma * (gamma - 1.0f) * ie) * g;
  S.dc = S.c * (0.6f * e2 + 1e-5f);
  S.p = ie * g;  // pressure / (gamma - 1)
  S.er = er;
  S.ep = 1.1f * (ei + er + ef) + 1e-6f;
  return true;
}

// The largest wave speed that riemann() (rs: 0 Rusanov, 1 LLF, 2 HLL, 3 HLLC;
// avg: 1 Einfeldt, else TRRS) can return for the two sides, or kNoBound.
RKDG_HD float speed_bound(const SpeedSide& L, const SpeedSide& R, float gamma, int rs, int avg, bool negative_ok) {
  if (rs == 0) return fmaxf(L.v + L.du + L.c + L.dc, R.v + R.du + R.c + R.dc) * 1.000001f;
  const float D = R.u - L.u;
  float SLlo, SLhi, SRlo, SRhi;
  if (avg == 1) {
    const float t = bsqrt(bdiv(R.r, L.r)), wL = bdiv(1.0f, 1.0f + t), wR = t * wL;
    const float et = 0.6f * (L.er + R.er) + 1e-6f;
    const float uav = wL * L.u + wR * R.u;
    const float cav = bsqrt(wL * L.c * L.c + wR * R.c * R.c + 0.5f * wL * wR * D * D);
    const float err = fmaxf(L.du, R.du) + fmaxf(L.dc, R.dc) + 0.36f * (L.du + R.du) +
                      (0.6f * et + 1e-6f) * (fabsf(D) + cav) + 1e-6f * (fabsf(L.u) + fabsf(R.u));
    SLlo = uav - cav - err;
    SLhi = uav - cav + err;
    SRlo = uav + cav - err;
    SRhi = uav + cav + err;
  } else {
    const float gm1 = gamma - 1.0f, z = bdiv(0.5f * gm1, gamma), iz = bdiv(1.0f, z);
    const float x = bdiv(L.p, R.p), ex = L.ep + R.ep;
    const float xz = exp2f(z * log2f(x));
    const float A = L.c + R.c - 0.5f * gm1 * D;
    const float dA = L.dc + R.dc + 0.5f * gm1 * (L.du + R.du) + 1e-5f * (L.c + R.c + 0.5f * gm1 * fabsf(D));
    const float B = L.c + R.c * xz, dB = L.dc + xz * R.dc + R.c * xz * (1.2f * z * ex + 1e-5f) + 1e-6f * B;
    // a base that may be negative: the FP64 evaluation decides on its power
    if (!(A - dA > 0.0f && ex < 0.2f && B - dB > 0.0f)) return kNoBound;
    const float t = bdiv(A + dA, B - dB);
    const float pl = exp2f(iz * log2f(t)) * (1.00001f + 1e-6f * iz), pr = pl * x * (1.00001f + 1.1f * ex);
    const float hg = bdiv(0.5f * (gamma + 1.0f), gamma);
    const float qL = pl > 1.0f ? bsqrt(1.0f + hg * (pl - 1.0f)) * 1.000001f : 1.0f;
    const float qR = pr > 1.0f ? bsqrt(1.0f + hg * (pr - 1.0f)) * 1.000001f : 1.0f;
    SLlo = L.u - L.du - qL * (L.c + L.dc);
    SLhi = L.u + L.du - (L.c - L.dc);
    SRlo = R.u - R.du + (R.c - R.dc);
    SRhi = R.u + R.du + qR * (R.c + R.dc);
  }
  float hi = fmaxf(SLhi, SRhi);
  if (rs == 3) {
    if (!(negative_ok || fmaxf(SLlo, SRlo) >= 0.0f)) return kNoBound;
  } else {
    hi = fmaxf(hi, fmaxf(-SLlo, -SRlo));
  }
  return hi >= 0.0f ? hi * 1.000001f : (hi < 0.0f ? 0.0f : kNoBound);
}

}  // namespace rkdg
