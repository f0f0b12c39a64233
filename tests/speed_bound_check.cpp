// CPU check of rkdg_speed_bound.h: for random nodal values, face rows of the
// reference elements and normals, the FP32 bound against the FP64 wave speed
// (the reference's formulas, physics.cpp:252-350, from the FP64 traces).
// Prints: Lebesgue sum, points, bounded points, bounds below the speed, HLLC
// points taken though the speed is negative, smooth points bounded within 1e-3.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>

#include "rkdg_refelem.h"
#include "rkdg_speed_bound.h"

using namespace rkdg;

static float cut(double x) {  // towards zero
  float f = (float)x;
  if (std::fabs((double)f) > std::fabs(x)) f = std::nextafterf(f, 0.0f);
  return f;
}

template <int DIM>
struct Exact {
  double g, b;
  double p(const double* s) const {
    double m2 = 0;
    for (int d = 0; d < DIM; ++d) m2 += s[1 + d] * s[1 + d];
    return (g - 1) * (s[1 + DIM] - 0.5 * m2 / s[0]) / (1 - s[0] * b);
  }
  double c(const double* s) const { return std::sqrt(g * p(s) / (s[0] * (1 - s[0] * b))); }
  // momentum along the first axis of RiemannSolver::Rotate's frame
  double mn(const double* s, const double* n) const {
    if (DIM == 2) return n[0] * s[1] + n[1] * s[2];
    const double cp = std::sqrt(1 - n[2] * n[2]);
    const bool ok = std::fabs(cp) > 1e-6;
    const double st = ok ? n[1] / cp : 1, ct = ok ? n[0] / cp : 0;
    return cp * ct * s[1] + cp * st * s[2] + n[2] * s[3];
  }
  double speed(const double* L, const double* R, const double* n, int rs, int avg) const {
    if (rs == 0) {
      double e[2];
      for (int i = 0; i < 2; ++i) {
        const double* s = i ? R : L;
        double m2 = 0;
        for (int d = 0; d < DIM; ++d) m2 += s[1 + d] * s[1 + d];
        e[i] = std::sqrt(m2) / s[0] + c(s);
      }
      return std::max(e[0], e[1]);
    }
    const double cL = c(L), cR = c(R), uL = mn(L, n) / L[0], uR = mn(R, n) / R[0];
    double SL, SR;
    if (avg == 1) {
      const double sL = std::sqrt(L[0]), sR = std::sqrt(R[0]), sum = sL + sR;
      const double ua = (uL * sL + uR * sR) / sum;
      const double ca = std::sqrt((sL * cL * cL + sR * cR * cR) / sum +
                                  0.5 * sL * sR / (sum * sum) * (uR - uL) * (uR - uL));
      SL = ua - ca;
      SR = ua + ca;
    } else {
      const double pL = p(L), pR = p(R), z = 0.5 * (g - 1) / g;
      const double ps = std::pow((cL + cR - 0.5 * (g - 1) * (uR - uL)) / (cL / std::pow(pL, z) + cR / std::pow(pR, z)),
                                 1 / z);
      SL = uL - cL * (ps > pL ? std::sqrt(1 + 0.5 * (g + 1) * (ps / pL - 1) / g) : 1);
      SR = uR + cR * (ps > pR ? std::sqrt(1 + 0.5 * (g + 1) * (ps / pR - 1) / g) : 1);
    }
    return rs == 3 ? std::max(SL, SR) : std::max(std::fabs(SL), std::fabs(SR));
  }
};

template <int DIM>
void run(int geom, int p, int n, unsigned seed) {
  static RefTables T;
  build_ref_tables(geom, p, T, nullptr);
  const int nd = T.nd, nfpe = T.nfpe, nqf = T.nqf;
  double leb = 0;
  for (int lf = 0; lf < nfpe; ++lf)
    for (int q = 0; q < nqf; ++q) {
      double a = 0;
      for (int j = 0; j < nd; ++j) a += std::fabs(T.B[lf][q][j]);
      leb = std::max(leb, a);
    }
  std::mt19937_64 gen(seed);
  std::uniform_real_distribution<double> U(-1, 1);
  long bounded = 0, below = 0, neg = 0, points = 0, smooth = 0, tight = 0;
  const double gammas[] = {1.02, 1.05, 1.1, 1.2, 4.0 / 3, 1.4, 5.0 / 3, 2.0, 3.0};
  for (int it = 0; it < n; ++it) {
    Exact<DIM> X{gammas[gen() % 9], gen() % 2 ? 0.0 : 0.01};
    double nn[3] = {U(gen), U(gen), U(gen)};
    if (DIM == 3 && gen() % 2) {  // close to the z axis
      const double t = std::pow(10.0, -1.0 - 6.5 * std::fabs(U(gen)));
      nn[0] *= t;
      nn[1] *= t;
      nn[2] = nn[2] < 0 ? -1 : 1;
    }
    double len = 0;
    for (int d = 0; d < DIM; ++d) len += nn[d] * nn[d];
    for (int d = 0; d < DIM; ++d) nn[d] /= std::sqrt(len);
    const double amp = std::pow(10.0, -4 * std::fabs(U(gen))) * 0.3, mach = std::pow(10.0, 1.5 * U(gen));
    const double scale = std::pow(10.0, 3 * U(gen));
    double dir[3] = {U(gen), U(gen), U(gen)};
    const bool jump = gen() % 2;
    float sf[2][5], top[2][5], nf[3];
    double s[2][5];
    double rho0 = scale, p0 = scale * std::pow(10.0, U(gen));
    for (int d = 0; d < DIM; ++d) nf[d] = (float)nn[d];
    for (int side = 0; side < 2; ++side) {
      if (side && jump) {
        rho0 *= std::pow(10.0, U(gen));
        p0 *= std::pow(10.0, U(gen));
        for (int d = 0; d < DIM; ++d) dir[d] += U(gen);
      }
      const double c0 = std::sqrt(X.g * p0 / rho0);
      const int row = (int)(gen() % (nfpe * nqf));
      const double* B = T.B[row / nqf][row % nqf];
      for (int k = 0; k < 5; ++k) s[side][k] = sf[side][k] = top[side][k] = 0;
      for (int j = 0; j < nd; ++j) {
        const double r = rho0 * (1 + amp * U(gen)), pr = p0 * (1 + amp * U(gen));
        double v[5] = {r}, e = pr * (1 - r * X.b) / (X.g - 1);
        for (int d = 0; d < DIM; ++d) {
          const double u = mach * c0 * (dir[d] + amp * U(gen));
          v[1 + d] = r * u;
          e += 0.5 * r * u * u;
        }
        v[1 + DIM] = e;
        for (int k = 0; k < DIM + 2; ++k) {
          s[side][k] += B[j] * v[k];
          sf[side][k] += (float)B[j] * cut(v[k]);
          top[side][k] = std::max(top[side][k], std::fabs(cut(v[k])));
        }
      }
    }
    bool ok = true;
    for (int side = 0; side < 2; ++side)
      ok = ok && s[side][0] > 0 && s[side][1 + DIM] > 0 && X.p(s[side]) > 0 && s[side][0] * X.b < 1;
    if (!ok) continue;
    for (int rs = 0; rs < 4; ++rs)
      for (int avg = 0; avg < 2; ++avg) {
        ++points;
        SpeedSide A, C;
        float hi = kNoBound;
        if (speed_side<DIM>(sf[0], top[0], 1, nf, (float)X.g, (float)X.b, A) &&
            speed_side<DIM>(sf[1], top[1], 1, nf, (float)X.g, (float)X.b, C))
          hi = speed_bound(A, C, (float)X.g, rs, avg, false);
        const double sp = X.speed(s[0], s[1], nn, rs, avg);
        if (!jump && amp < 0.01 && mach < 1 && X.g > 1.15 && rs < 3) {
          ++smooth;
          tight += hi < sp * 1.001;
        }
        if (!(hi < kNoBound)) continue;
        ++bounded;
        below += !(hi >= sp);
        neg += sp < 0;
      }
  }
  printf("%.4f %ld %ld %ld %ld %ld %ld\n", leb, points, bounded, below, neg, smooth, tight);
}

int main(int argc, char** argv) {
  const int geom = atoi(argv[1]), p = atoi(argv[2]), n = atoi(argv[3]);
  geom == 5 ? run<3>(geom, p, n, 11) : run<2>(geom, p, n, 12);
}
