// Vector-Jacobian products of the pointwise physics in reverse mode: given the
// cotangent of a flux, the cotangents of the states it was formed from.
//
// One reverse sweep costs about three evaluations of the flux and yields both
// sides' gradients; forward mode (Dual<NEQ>) costs NEQ + 1 evaluations per
// side and spills.  Branches (min/max, HLL/HLLC cases, TRRS switches) follow
// the primal values, the derivative of the active branch.
#pragma once

#include "rkdg_physics.cuh"

namespace rkdg {

// One side's state in the frame its flux is taken in, what is formed from it,
// and the cotangents of those quantities.
template <int DIM>
struct FluxSide {
  static constexpr int NEQ = DIM + 2;
  double s[NEQ], r, q, p, u2;  // state, 1/rho, 1/(1 - rho b), pressure, |u|^2
  double sb[NEQ], rb, pb, cb;  // cotangents; cb: of c^2 = gamma p q / rho
  __device__ __forceinline__ bool load(const double* x, double gamma, double b) {
#pragma unroll
    for (int i = 0; i < NEQ; ++i) {
      s[i] = x[i];
      sb[i] = 0.0;
    }
    rb = pb = cb = 0.0;
    return eos_state<DIM>(s, gamma, b, r, q, p, u2);
  }
  __device__ __forceinline__ double c2(double gamma) const { return gamma * p * r * q; }
  // pressure, sound speed and 1/rho back to the state
  __device__ __forceinline__ void finish(double gamma, double b) {
    double qb = cb * (gamma * p * r);
    pb += cb * (gamma * r * q);
    rb += cb * (gamma * p * q);
    const double g = pb * (gamma - 1.0) * q;
    sb[NEQ - 1] += g;
    double m2 = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      m2 += s[1 + d] * s[1 + d];
      sb[1 + d] -= g * r * s[1 + d];
    }
    rb -= 0.5 * g * m2;
    sb[0] -= rb * r * r;
    if (b != 0.0) {
      qb += pb * (gamma - 1.0) * (s[NEQ - 1] - 0.5 * m2 * r);
      sb[0] += qb * b * q * q;
    }
  }
};

// Rusanov (rs_rusanov.cpp:6-40) on unrotated states.
template <int DIM>
__device__ __forceinline__ void rusanov_vjp(FluxSide<DIM>& A, FluxSide<DIM>& B, const Frame<DIM, double>& fr,
                                            const double* fb, double gamma) {
  constexpr int NEQ = DIM + 2;
  const double h = fr.h, *n = fr.n;
  const double cA = root(A.c2(gamma)), cB = root(B.c2(gamma)), vA = root(A.u2), vB = root(B.u2);
  const bool left = vA + cA > vB + cB;
  const double a = 0.5 * (left ? vA + cA : vB + cB);
  double ab = 0.0;  // cotangent of max(|u| + c)
#pragma unroll
  for (int i = 0; i < NEQ; ++i) {
    ab -= 0.5 * fb[i] * (B.s[i] - A.s[i]);
    A.sb[i] += a * fb[i];
    B.sb[i] -= a * fb[i];
  }
  auto side = [&](FluxSide<DIM>& S) {
    double dn = 0.0, tb = 0.0, pn = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      dn += S.s[1 + d] * n[d];
      tb += fb[1 + d] * S.s[1 + d];
      pn += fb[1 + d] * n[d];
    }
    const double H = S.s[NEQ - 1] + S.p, un = dn * S.r, eb = fb[NEQ - 1];
    const double dnb = h * (fb[0] + S.r * (tb + eb * H));  // of m.n
    S.rb += h * dn * (tb + eb * H);
    S.pb += h * (pn + eb * un);
    S.sb[NEQ - 1] += h * eb * un;
#pragma unroll
    for (int d = 0; d < DIM; ++d) S.sb[1 + d] += dnb * n[d] + h * un * fb[1 + d];
  };
  side(A);
  side(B);
  const double c = left ? cA : cB, v = left ? vA : vB;
  // one side holds the maximum: no indexed copies
  auto speed = [&](FluxSide<DIM>& S, bool on) {
    const double e = on ? ab : 0.0;
    S.cb += on ? 0.5 * e * rcp(c) : 0.0;
    const double vb = v > 0.0 ? e * rcp(v) : 0.0;  // 2 d|u| / d|u|^2
    double m2 = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      m2 += S.s[1 + d] * S.s[1 + d];
      S.sb[1 + d] += vb * S.r * S.r * S.s[1 + d];
    }
    S.rb += vb * S.r * m2;
  };
  speed(A, left);
  speed(B, !left);
}

// LLF, HLL, HLLC (rs_llf.cpp:6-37, rs_hll.cpp:6-50, rs_hllc.cpp:71-161) on
// states rotated into the face frame (s[1] along the normal).
template <int DIM>
__device__ __forceinline__ void hll_vjp(FluxSide<DIM>& A, FluxSide<DIM>& B, const double* fb,
                                        double gamma, int rs, int avg) {
  constexpr int NEQ = DIM + 2;
  const double u1 = A.s[1] * A.r, u2 = B.s[1] * B.r;
  double u1b = 0.0, u2b = 0.0, SLb = 0.0, SRb = 0.0;
  const double cA2 = A.c2(gamma), cB2 = B.c2(gamma);
  double SL, SR;
  // intermediates of the wave speeds that the sweep needs again
  double t, wL = 0.0, wR = 0.0, cav = 1.0, cL = 0.0, cR = 0.0, xz = 0.0, den = 1.0, pl = 0.0, x = 0.0,
            qL = 1.0, qR = 1.0;
  const double gm1 = gamma - 1.0, iz = 2.0 * gamma / gm1, hg = 0.5 * (gamma + 1.0) / gamma;
  if (avg == 1) {
    t = root(B.s[0] * A.r);
    wL = rcp(1.0 + t);
    wR = t * wL;
    const double du = u2 - u1, uav = wL * u1 + wR * u2;
    cav = root(wL * cA2 + wR * cB2 + 0.5 * wL * wR * du * du);
    SL = uav - cav;
    SR = uav + cav;
  } else {
    cL = root(cA2);
    cR = root(cB2);
    x = A.p * rcp(B.p);
    const int n = (int)rint(iz);
    const bool whole = n >= 2 && n <= 16 && fabs(iz - n) <= n * 1e-14;
    xz = whole ? root_n(x, n, 0.5 * gm1 / gamma) : exp2(log2(x) / iz);
    den = cL + cR * xz;
    t = (cL + cR - 0.5 * gm1 * (u2 - u1)) * rcp(den);
    if (t < 0.0) {
      pl = trrs_negative_base(t, gamma);
    } else if (whole) {
      pl = t;
      for (int i = 1; i < n; ++i) pl *= t;
    } else {
      pl = powr(t, iz);
    }
    const double pr = pl * x;
    if (pl > 1.0) qL = root(1.0 + hg * (pl - 1.0));
    if (pr > 1.0) qR = root(1.0 + hg * (pr - 1.0));
    SL = u1 - qL * cL;
    SR = u2 + qR * cR;
  }
  // cotangents f of a side's x-flux
  auto flux_back = [&](FluxSide<DIM>& S, double u, double& ub, const double* f) {
    S.sb[1] += f[0] + f[1] * u;
    S.pb += f[1] + f[NEQ - 1] * u;
    double v = f[1] * S.s[1] + f[NEQ - 1] * (S.s[NEQ - 1] + S.p);
#pragma unroll
    for (int d = 1; d < DIM; ++d) {
      S.sb[1 + d] += f[1 + d] * u;
      v += f[1 + d] * S.s[1 + d];
    }
    S.sb[NEQ - 1] += f[NEQ - 1] * u;
    ub += v;
  };
  auto side_flux = [&](const FluxSide<DIM>& S, double u, double* f) {
    f[0] = S.s[1];
    f[1] = S.s[1] * u + S.p;
#pragma unroll
    for (int d = 1; d < DIM; ++d) f[1 + d] = S.s[1 + d] * u;
    f[NEQ - 1] = (S.s[NEQ - 1] + S.p) * u;
  };
  if (rs == 1) {
    const bool useL = fabs(SL) >= fabs(SR);
    const double m = useL ? fabs(SL) : fabs(SR);
    double hb[NEQ], mb = 0.0;
#pragma unroll
    for (int i = 0; i < NEQ; ++i) {
      hb[i] = 0.5 * fb[i];
      mb -= hb[i] * (B.s[i] - A.s[i]);
      A.sb[i] += m * hb[i];
      B.sb[i] -= m * hb[i];
    }
    flux_back(A, u1, u1b, hb);
    flux_back(B, u2, u2b, hb);
    if (useL)
      SLb = SL < 0.0 ? -mb : mb;
    else
      SRb = SR < 0.0 ? -mb : mb;
  } else if (SL >= 0.0) {
    flux_back(A, u1, u1b, fb);
  } else if (SR <= 0.0) {
    flux_back(B, u2, u2b, fb);
  } else if (rs == 2) {
    double f1[NEQ], f2[NEQ];
    side_flux(A, u1, f1);
    side_flux(B, u2, f2);
    const double inv = rcp(SR - SL);
    double tot = 0.0;
#pragma unroll
    for (int i = 0; i < NEQ; ++i) {
      const double d = B.s[i] - A.s[i], v = fb[i] * inv;
      tot += v * ((SR * f1[i] - SL * f2[i] + SL * SR * d) * inv);
      SRb += v * (f1[i] + SL * d);
      SLb += v * (SR * d - f2[i]);
      B.sb[i] += v * SL * SR;
      A.sb[i] -= v * SL * SR;
      f1[i] = v * SR;
      f2[i] = -v * SL;
    }
    SRb -= tot;
    SLb += tot;
    flux_back(A, u1, u1b, f1);
    flux_back(B, u2, u2b, f2);
  } else {
    const double k1 = SL - u1, k2 = SR - u2;
    const double dn = A.s[0] * k1 - B.s[0] * k2, idn = rcp(dn);
    const double ss = (B.p - A.p + A.s[1] * k1 - B.s[1] * k2) * idn;
    const bool left = ss > 0.0;
    double ssb = 0.0, k1b = 0.0, k2b = 0.0;
    auto star = [&](FluxSide<DIM>& S, double SK, double u, double k, double& SKb, double& ub, double& kb) {
      double f[NEQ];
      side_flux(S, u, f);
      const double G = S.p + S.s[0] * k * (ss - u), extra = SK * G, inv = rcp(SK - ss);
      double tot = 0.0, skb = 0.0;
      const double eb = (fb[1] + fb[NEQ - 1] * ss) * inv;
#pragma unroll
      for (int i = 0; i < NEQ; ++i) {
        const double v = fb[i] * inv, w = S.s[i] * SK - f[i];
        const double D = i == 1 ? extra : (i == NEQ - 1 ? ss * extra : 0.0);
        tot += v * ((ss * w + D) * inv);
        ssb += v * w;
        S.sb[i] += v * ss * SK;
        skb += v * ss * S.s[i];
        f[i] = -v * ss;
      }
      ssb += fb[NEQ - 1] * inv * extra + tot;
      const double Gb = eb * SK;
      SKb += skb - tot + eb * G;
      S.pb += Gb;
      S.sb[0] += Gb * k * (ss - u);
      kb += Gb * S.s[0] * (ss - u);
      ssb += Gb * S.s[0] * k;
      ub -= Gb * S.s[0] * k;
      flux_back(S, u, ub, f);
    };
    if (left)
      star(A, SL, u1, k1, SLb, u1b, k1b);
    else
      star(B, SR, u2, k2, SRb, u2b, k2b);
    const double nb = ssb * idn, db = -nb * ss;
    B.pb += nb;
    A.pb -= nb;
    A.sb[1] += nb * k1;
    B.sb[1] -= nb * k2;
    k1b += nb * A.s[1] + db * A.s[0];
    k2b -= nb * B.s[1] + db * B.s[0];
    A.sb[0] += db * k1;
    B.sb[0] -= db * k2;
    SLb += k1b;
    u1b -= k1b;
    SRb += k2b;
    u2b -= k2b;
  }
  // wave speeds
  if (avg == 1) {
    const double du = u2 - u1, ub = SLb + SRb, xb = 0.5 * (SRb - SLb) * rcp(cav);
    double wLb = ub * u1 + xb * (cA2 + 0.5 * wR * du * du);
    const double wRb = ub * u2 + xb * (cB2 + 0.5 * wL * du * du);
    const double dub = xb * wL * wR * du;
    u1b += ub * wL - dub;
    u2b += ub * wR + dub;
    A.cb += xb * wL;
    B.cb += xb * wR;
    wLb += wRb * t;
    const double tb = wRb * wL - wLb * wL * wL;
    // t^2 = rhoR / rhoL
    A.sb[0] -= 0.5 * tb * t * A.r;
    B.sb[0] += 0.5 * tb * t * B.r;
  } else {
    double cLb = -SLb * qL, cRb = SRb * qR;
    double plb = pl > 1.0 ? -0.5 * SLb * cL * hg * rcp(qL) : 0.0;
    const double prb = pl * x > 1.0 ? 0.5 * SRb * cR * hg * rcp(qR) : 0.0;
    plb += prb * x;
    double xb = prb * pl;
    const double tb = plb * iz * pl * rcp(t), ab = tb * rcp(den), db = -ab * t;
    cLb += ab + db;
    cRb += ab + db * xz;
    xb += db * cR * xz * rcp(iz * x);
    const double dub = -0.5 * gm1 * ab;
    u1b += SLb - dub;
    u2b += SRb + dub;
    const double ip = rcp(B.p);
    A.pb += xb * ip;
    B.pb -= xb * x * ip;
    A.cb += 0.5 * cLb * rcp(cL);
    B.cb += 0.5 * cRb * rcp(cR);
  }
  A.sb[1] += u1b * A.r;
  A.rb += u1b * A.s[1];
  B.sb[1] += u2b * B.r;
  B.rb += u2b * B.s[1];
}

// g1 = (dF/ds1)^T fb, g2 = (dF/ds2)^T fb of the numerical flux riemann(s1, s2,
// n); zero where a state is non-physical.  rotate() and inverse_rotate() are
// each other's transposes.
template <int DIM>
__device__ __forceinline__ void riemann_vjp(const double* s1, const double* s2, const double* n,
                                            const double* fb, double gamma, double b, int rs, int avg,
                                            double* g1, double* g2) {
  constexpr int NEQ = DIM + 2;
  FluxSide<DIM> A, B;
  double x1[NEQ], x2[NEQ], f[NEQ];
#pragma unroll
  for (int i = 0; i < NEQ; ++i) {
    x1[i] = s1[i];
    x2[i] = s2[i];
    f[i] = fb[i];
    g1[i] = g2[i] = 0.0;
  }
  const Frame<DIM, double> fr = make_frame<DIM, double>(n);
  if (rs != 0) {
    rotate<DIM>(x1, fr);
    rotate<DIM>(x2, fr);
    rotate<DIM>(f, fr);
  }
  const bool ok1 = A.load(x1, gamma, b), ok2 = B.load(x2, gamma, b);
  if (!ok1 || !ok2) return;
  if (rs == 0)
    rusanov_vjp<DIM>(A, B, fr, f, gamma);
  else
    hll_vjp<DIM>(A, B, f, gamma, rs, avg);
  A.finish(gamma, b);
  B.finish(gamma, b);
  if (rs != 0) {
    inverse_rotate<DIM>(A.sb, fr);
    inverse_rotate<DIM>(B.sb, fr);
  }
#pragma unroll
  for (int i = 0; i < NEQ; ++i) {
    g1[i] = A.sb[i];
    g2[i] = B.sb[i];
  }
}

// g = (dF/ds)^T : fb for the nodal Euler flux F[k][d] (flux_and_speed).
template <int DIM>
__device__ __forceinline__ void flux_vjp(const double* s, const double (*fb)[DIM], double gamma,
                                         double b, double* g) {
  constexpr int NEQ = DIM + 2;
  const double r = rcp(s[0]), p = pressure<DIM>(s, gamma, b), H = s[NEQ - 1] + p;
  const double q = b == 0.0 ? 1.0 : rcp(1.0 - s[0] * b);
  double rb = 0.0, pb = 0.0, eb = 0.0, m2 = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    double v = fb[0][d] + fb[NEQ - 1][d] * H * r, w = fb[NEQ - 1][d] * H;
#pragma unroll
    for (int i = 0; i < DIM; ++i) {
      v += (fb[1 + i][d] + fb[1 + d][i]) * s[1 + i] * r;
      w += fb[1 + i][d] * s[1 + i];
    }
    g[1 + d] = v;
    rb += w * s[1 + d];
    eb += fb[NEQ - 1][d] * s[1 + d] * r;
    pb += fb[1 + d][d];
    m2 += s[1 + d] * s[1 + d];
  }
  pb += eb;
  const double gp = pb * (gamma - 1.0) * q;
  g[NEQ - 1] = eb + gp;
#pragma unroll
  for (int d = 0; d < DIM; ++d) g[1 + d] -= gp * r * s[1 + d];
  rb -= 0.5 * gp * m2;
  g[0] = -rb * r * r;
  if (b != 0.0) g[0] += pb * p * b * q;
}

}  // namespace rkdg
