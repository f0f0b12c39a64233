// Limiter::update (limiter.cpp:22-94) with the BJ-family, Everywhere and
// Nowhere indicators: a few threads per element.
#pragma once

#include "rkdg_common.h"
#include "rkdg_generic.cuh"
#include "rkdg_physics.cuh"

namespace rkdg {

// Threads per element: quads one per face (two indicator points and one
// vertex each), hexahedra eight (three points, one vertex), triangles two.
template <int G, int P>
struct LimTeam {
  using E = El<G, P>;
  static constexpr int L = G == 2 ? 2 : (G == 3 ? 4 : 8);
  static constexpr int NPT = E::NFPE * E::NQL;
  static constexpr int NDP = E::ND | 1;  // odd row stride: the slots of a warp fall into distinct banks
  static constexpr int MAX_BLOCK = 256;
  template <typename R, bool DS>
  static constexpr size_t smem_bytes(int block) {
    const size_t epb = block / L;
    // means, values (and low words), operators, factors, gas constants, ids
    return 8 * epb * E::NEQ + (sizeof(R) + (DS ? 4 : 0)) * epb * E::NEQ * NDP +
           8 * (size_t)E::ND * NPT + sizeof(R) * (size_t)E::ND * E::NV + 16 * epb + 2 * sizeof(R) * epb +
           2 * sizeof(int) * epb + (sizeof(R) == 8 ? 8 * epb * E::NEQ : 0) + 16;
  }
};

__device__ __forceinline__ double shfl_xor_mean(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ float2 shfl_xor_mean(float2 v, int o) {
  return make_float2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}

// StateIsPhysical (physics.cpp:6-50) without its quotients: the covolume
// pressure has the sign of (gamma - 1) (rho E - |m|^2 / 2) (1 - rho b).  Float
// states that cancel, or so small that the products leave the normal numbers
// (FP32 flushes below 1.2e-38), are judged in FP64; FP64 states as small with the
// quotients.
template <int DIM, typename R>
__device__ __forceinline__ bool vertex_is_physical(const R* s, R gamma, R b) {
  if (!(s[0] >= R(0)) || !(s[1 + DIM] > R(0))) return false;
  R m2 = R(0);
#pragma unroll
  for (int d = 0; d < DIM; d++) m2 += s[1 + d] * s[1 + d];
  const R re = s[0] * s[1 + DIM];
  R x = re - R(0.5) * m2;
  if constexpr (std::is_same<R, float>::value) {
    if (!(fabsf(x) > fmaxf(1e-3f * re, 1e-30f))) {
      double m2d = 0.0;
#pragma unroll
      for (int d = 0; d < DIM; d++) m2d += (double)s[1 + d] * (double)s[1 + d];
      x = (double)s[0] * (double)s[1 + DIM] - 0.5 * m2d > 0.0 ? 1.0f : -1.0f;
    }
  } else {
    if (!(re > 1e-290)) return state_is_physical<DIM>(s, gamma, b);
  }
  return (gamma - R(1)) * x * (R(1) - s[0] * b) > R(0);
}

// Stencil = the element and its face neighbours (ElementToElementTable,
// limiter.cpp:115-123), the BJ-family indicator at the order-2 points of its
// interior faces (indicator_bj.cpp:88-200, updateYMin 15-86), then
// LimiterMultiplier::limit (limiter_multiplier.cpp:12-99, including the
// nd-fold application of the density factor, quirks Q4/Q5, and the last-hope
// vertex check) or LimiterFinDiff::limit (limiter_findiff.cpp:3-33, last
// equation only, Q6).  The update reads only the element's own values and the
// cell means, so it is done in place.  DS = true: the values are a float pair
// (u = hi, ulo = lo).
//
// The indicator takes its branch decisions (face-point value minus mean
// against the +-1e-3 switches, stencil min/max) on the values the state holds:
// in FP64 for a double state; for a float state in double-single arithmetic
// (face-point values from the float state and its low word with the
// float-pair basis table, about 44 significant bits, so a switch differs from
// FP64 only within ~1e-13 relative of its threshold), and the ratio and
// limiter function, which only scale the float multiplier, in FP32.
//
// Only one equation's indicator is used (Multi: density, FinDiff: the last),
// so only that one is evaluated; the factor applied nd times is its nd-th
// power, formed once per element.  A group of L threads shares an element:
// the values come in coalesced through shared memory, each thread takes NPT/L
// indicator points and NV/L vertices, and elements that stay as they are are
// not written back.  Per launch against the thread-per-element form, which
// evaluated every equation's indicator, applied the factor nd times per value
// and spilled on Q2 hexahedra: 31x29x23 hex Q2 FP32 24 us (99) and float pair
// 32 us (287), 48x45x51 hex Q1 float pair 54 us (134), 33x27x21 hex Q1 FP64
// 40 us (191), 524,288 P1 triangles FP64 187 us (459; 254 with a division for
// every point), FP32 43 us (45) and float pair 66 us (76): there the arithmetic
// of the few values is what is left.
// MAP: a batch with a map of the active work (prm.act_cum).
template <int G, int P, typename R, bool DS, bool MAP>
__global__ void __launch_bounds__(LimTeam<G, P>::MAX_BLOCK)
    k_limit_team(const LimParams prm, R* __restrict__ u, float* __restrict__ ulo) {
  using E = El<G, P>;
  using T = LimTeam<G, P>;
  constexpr int DIM = E::DIM, ND = E::ND, NEQ = E::NEQ, NFPE = E::NFPE, NQL = E::NQL, NV = E::NV;
  constexpr int L = T::L, NPT = T::NPT, NDP = T::NDP;
  constexpr bool F32 = std::is_same<R, float>::value;
  // float states of hexahedra, small planar elements and Q2 quads: the factor is
  // applied nd times as the reference does (their limited runs amplify another
  // rounding, see riemann()); a float pair's power rounds far below that
  constexpr bool REPEAT = F32 && (ND <= 4 || (G == 5 && !DS) || (G == 3 && P == 2));
  // the means' low parts: FP64 hexahedra (on 200x4 quads the extra pass over
  // the values is 6% of a step, and a planar mesh's means change more per step)
  constexpr bool LOW = !F32 && G == 5;
  using MeanT = typename std::conditional<F32, float2, double>::type;
  using IndT = typename std::conditional<F32, float, double>::type;
  const RefTables* tab = prm.tab;
  const int tid = threadIdx.x, NT = blockDim.x, EPB = NT / L;
  if (MAP && (int)(blockIdx.x * EPB) >= prm.act_cum[*prm.act_n]) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  MeanT* sM = reinterpret_cast<MeanT*>(smraw);                     // [NEQ][EPB]
  MeanT* sBl = sM + NEQ * EPB;                                     // [ND][NPT]
  double* sMr = reinterpret_cast<double*>(sBl + ND * NPT);         // [EPB] factor (float: a float pair)
  R* sU = reinterpret_cast<R*>(sMr + EPB);                         // [NEQ][EPB][NDP]
  R* sBv = sU + NEQ * EPB * NDP;                                   // [ND][NV]
  R* sG = sBv + ND * NV;                                           // [EPB] gamma, [EPB] covolume
  float* sLo = reinterpret_cast<float*>(sG + 2 * EPB);             // [NEQ][EPB][NDP]
  double* sL = reinterpret_cast<double*>(sLo);                     // FP64: [NEQ][EPB] means' low parts
  int* sE = reinterpret_cast<int*>(sLo + (DS ? NEQ * EPB * NDP : (F32 ? 0 : 2 * NEQ * EPB)));  // [EPB]
  int* sF = sE + EPB;                                              // [EPB] 1 changed, 2 mean
  const int ne = prm.ne;
  const long long NDa = prm.ndofs;
  for (int t = tid; t < ND * NPT; t += NT) {
    const int j = t / NPT, pt = t - j * NPT;
    if constexpr (F32)
      sBl[t] = tab->Bl32[j][pt];
    else
      sBl[t] = tab->Bl[pt / NQL][pt % NQL][j];
  }
  for (int t = tid; t < ND * NV; t += NT) {
    const int j = t / NV, v = t - j * NV;
    if constexpr (F32)
      sBv[t] = tab->Bv32[j][v];
    else
      sBv[t] = tab->Bv[v][j];
  }
  // MAP: CTAs run over the elements of the active problems
  for (int blk = blockIdx.x;; blk += gridDim.x) {
    for (int s = tid; s < EPB; s += NT) {
      int e = blk * EPB + s, pb = -1;
      R gamma = (R)prm.gamma, cov = (R)prm.covolume;
      if (MAP) {  // the i-th element of the active problems
        const int na = *prm.act_n;
        e = e < prm.act_cum[na] ? active_element(prm.act_cum, prm.act_pid, prm.poff, na, e, prm.ne, prm.prob, pb) : -1;
      } else if (e >= ne) {
        e = -1;
      } else if (prm.prob) {
        pb = prm.prob[e];
      }
      if (e >= 0 && prm.prob) {
        if (!prm.pactive[pb]) e = -1;
        if constexpr (F32) {
          gamma = prm.pgamma32 ? prm.pgamma32[pb] : (R)prm.pgamma[pb];
          cov = prm.pcov32 ? prm.pcov32[pb] : (R)prm.pcov[pb];
        } else {
          gamma = (R)prm.pgamma[pb];
          cov = (R)prm.pcov[pb];
        }
      }
      sE[s] = e;
      sG[s] = gamma;
      sG[EPB + s] = cov;
    }
    __syncthreads();
    const bool multi = prm.limiter == 1;
    const int kind = multi ? 0 : NEQ - 1;  // the equation whose indicator counts
    for (int t = tid; t < EPB * NEQ; t += NT) {
      const int k = t / EPB, s = t - k * EPB, e = sE[s];
      if (e < 0) continue;
      if constexpr (F32)
        sM[t] = prm.means32[(long long)k * ne + e];
      else
        sM[t] = prm.means[(long long)k * ne + e];
    }
    for (int t = tid; t < EPB * ND; t += NT) {
      const int s = t / ND, j = t - s * ND, e = sE[s];
      if (e < 0) continue;
      const long long i0 = (long long)e * ND + j;
      if (multi) {
#pragma unroll
        for (int k = 0; k < NEQ; ++k) {
          sU[(k * EPB + s) * NDP + j] = u[k * NDa + i0];
          if constexpr (DS) sLo[(k * EPB + s) * NDP + j] = ulo[k * NDa + i0];
        }
      } else {
        sU[(kind * EPB + s) * NDP + j] = u[kind * NDa + i0];
        if constexpr (DS) sLo[(kind * EPB + s) * NDP + j] = ulo[kind * NDa + i0];
      }
    }
    __syncthreads();
    const int slot = tid / L, lane = tid - slot * L;
    const int e = sE[slot];
    IndT ind = IndT(1);
    if (prm.indicator == 1) {
      ind = IndT(0);
    } else if (prm.indicator == 2) {
      // stencil min / max of the means, started from the element's own mean
      // clamped to +-1e9: FP64, or for the float path float pairs compared
      // lexicographically (a normalised pair orders as its value)
      const MeanT own = sM[kind * EPB + slot];
      MeanT mI = own, MI = own;
      unsigned ncfaces = 0;
      int nbr[(NFPE + L - 1) / L];
#pragma unroll
      for (int i = 0; i < (NFPE + L - 1) / L; ++i) {
        const int lf = lane + i * L;
        nbr[i] = e >= 0 && lf < NFPE ? prm.fnbr[lf * ne + e] : -1;
        if (nbr[i] < 0) continue;
        const MeanT v = load_mean<F32>(prm, (long long)kind * ne + nbr[i]);
        if (mean_lt(v, mI)) mI = v;
        if (mean_lt(MI, v)) MI = v;
      }
      // hanging faces: the elements across them are stencil cells
      // (ElementToElementTable, limiter.cpp:118-123) and the element's own
      // slave or master faces carry indicator points (limiter.cpp:125-161)
      if (prm.ncidx && e >= 0 && prm.ncidx[e] >= 0) {
        const int row = prm.ncidx[e];
        for (int c = prm.nc_ptr[row] + lane; c < prm.nc_ptr[row + 1]; c += L) {
          const int f = prm.nc_ent[c] >> 1, side = prm.nc_ent[c] & 1;
          const int nb = prm.nc_face[f * 4 + (side ? 0 : 2)];
          ncfaces |= 1u << prm.nc_face[f * 4 + (side ? 3 : 1)];
          const MeanT v = load_mean<F32>(prm, (long long)kind * ne + nb);
          if (mean_lt(v, mI)) mI = v;
          if (mean_lt(MI, v)) MI = v;
        }
      }
      unsigned inner = ncfaces;
#pragma unroll
      for (int i = 0; i < (NFPE + L - 1) / L; ++i)
        if (nbr[i] >= 0) inner |= 1u << (lane + i * L);
      __syncwarp();
#pragma unroll
      for (int o = 1; o < L; o <<= 1) {
        const MeanT a = shfl_xor_mean(mI, o), b = shfl_xor_mean(MI, o);
        if (mean_lt(a, mI)) mI = a;
        if (mean_lt(MI, b)) MI = b;
        inner |= __shfl_xor_sync(0xffffffffu, inner, o);
      }
      const R* un = sU + (kind * EPB + slot) * NDP;
      IndT yMin = IndT(1e9);
      if constexpr (F32) {
        const float2 big = make_float2(1e9f, 0.0f), small = make_float2(-1e9f, 0.0f);
        if (mean_lt(big, mI)) mI = big;
        if (mean_lt(MI, small)) MI = small;
        // double-single: the +-1e-3 switches as float pairs, the numerators of
        // the ratio (stencil max / min minus the mean) rounded to FP32
        const float* ul = DS ? sLo + (kind * EPB + slot) * NDP : nullptr;
        const float th = 1e-3f, tl = (float)(1e-3 - (double)1e-3f);
        const float nMax = (MI.x - own.x) + (MI.y - own.y);
        const float nMin = (mI.x - own.x) + (mI.y - own.y);
        for (int pt = lane; pt < NPT; pt += L) {
          if (!((inner >> (pt / NQL)) & 1u)) continue;  // only interior faces carry indicator points
          // value at the point minus the mean, as a float pair
          float sh = -own.x, sl = -own.y;
#pragma unroll
          for (int j = 0; j < ND; ++j) {
            const float2 bq = sBl[j * NPT + pt];
            const float x = un[j];
            const float ph = x * bq.x;
            float pl = fmaf(x, bq.x, -ph);
            pl = fmaf(x, bq.y, pl);
            if constexpr (DS) pl = fmaf(ul[j], bq.x, pl);
            float t, er;
            two_sum(sh, ph, t, er);
            er += sl + pl;
            sh = t + er;
            sl = er - (sh - t);
          }
          const bool above = sh > th || (sh == th && sl > tl);
          const bool below = sh < -th || (sh == -th && sl < -tl);
          const float y = above ? nMax / sh : (below ? nMin / sh : 1.0f);
          if (prm.function == 0) {
            yMin = fminf(fminf(y, yMin), 1.0f);
          } else if (prm.function == 1) {
            const float yc = (y * y + 2.0f * y) / (y * y + y + 2.0f);
            yMin = fminf(yc, yMin);
          } else {
            const float ys = 1.5f;
            const float yr = y / ys;
            const float yc = y < 1.0f ? y + (3.0f - 2.0f * ys) * yr * yr + (ys - 2.0f) * yr * yr * yr : 1.0f;
            yMin = fminf(yc, yMin);
          }
        }
#pragma unroll
        for (int o = 1; o < L; o <<= 1) yMin = fminf(yMin, __shfl_xor_sync(0xffffffffu, yMin, o));
      } else {
        if (mI > 1e9) mI = 1e9;
        if (MI < -1e9) MI = -1e9;
        // y = (stencil max or min - mean) / diff falls with |diff|, and every
        // limiter function is smallest at the smallest y (Venkatakrishnan's,
        // where that lies below 2): only the points of largest |diff| above and
        // below the mean are divided for, one by the even and one by the odd
        // lanes.  |diff| is compared as integers, off the FP64 pipe.
        const long long dead = __double_as_longlong(1e-3), inf = 0x7ff0000000000000ll;
        const long long sign = (long long)0x8000000000000000ull;
        long long far[2] = {0, 0}, near[2] = {inf, inf};  // |diff| above, below
        bool level = false;                               // some point within the +-1e-3 switch
        for (int pt = lane; pt < NPT; pt += L) {
          if (!((inner >> (pt / NQL)) & 1u)) continue;  // only interior faces carry indicator points
          double v = 0.0;
#pragma unroll
          for (int j = 0; j < ND; ++j) v += un[j] * sBl[j * NPT + pt];
          const long long d = __double_as_longlong(v - own), ad = d & ~sign;
          const bool in = ad <= dead || ad > inf;  // (NaN compares as neither)
          level |= in;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const bool on = !in && (d < 0) == (h == 1);
            far[h] = on && ad > far[h] ? ad : far[h];
            near[h] = on && ad < near[h] ? ad : near[h];
          }
        }
        __syncwarp();
#pragma unroll
        for (int o = 1; o < L; o <<= 1) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const long long x = __shfl_xor_sync(0xffffffffu, far[h], o);
            far[h] = x > far[h] ? x : far[h];
          }
          level |= __shfl_xor_sync(0xffffffffu, (int)level, o) != 0;
        }
        const int h = lane & 1;
        const double num = h ? own - mI : MI - own;
        auto function = [&](double y) {
          if (prm.function == 0) return y > 1.0 ? 1.0 : y;
          if (prm.function == 1) return (y * y + 2.0 * y) / (y * y + y + 2.0);
          const double ys = 1.5;
          const double yr = y / ys;
          return y < 1.0 ? y + (3.0 - 2.0 * ys) * yr * yr + (ys - 2.0) * yr * yr * yr : 1.0;
        };
        if (level) yMin = prm.function == 1 ? 0.75 : 1.0;
        const long long fh = h ? far[1] : far[0];
        const double y = fh ? num / __longlong_as_double(fh) : 1e9;
        if (fh) {
          const double yc = function(y);
          yMin = yc < yMin ? yc : yMin;
        }
        // Venkatakrishnan's function rises to y = 2 + sqrt(8), then falls to 1: with
        // every y above 2 the largest may be the minimum
        if (prm.function == 1 && __any_sync(0xffffffffu, y > 2.0 && fh)) {
#pragma unroll
          for (int o = 1; o < L; o <<= 1)
#pragma unroll
            for (int g = 0; g < 2; ++g) {
              const long long x = __shfl_xor_sync(0xffffffffu, near[g], o);
              near[g] = x < near[g] ? x : near[g];
            }
          if (fh) {
            const double yc = function(num / __longlong_as_double(h ? near[1] : near[0]));
            yMin = yc < yMin ? yc : yMin;
          }
        }
        const double other = __shfl_xor_sync(0xffffffffu, yMin, 1);
        yMin = other < yMin ? other : yMin;
      }
      ind = yMin;
    }
    if (!multi) {
      // no float lies between 0.999 and its FP32 rounding
      if (lane == 0) sF[slot] = e >= 0 && ind < IndT(0.999) ? 3 : 0;
      __syncthreads();
    } else {
      const int reps = (prm.quirks & 1) ? 1 : ND;
      const bool lin = G != 2 && (prm.quirks & 2);
      if (lane == 0) {
        if constexpr (F32) {
          float h = (float)ind, l = 0.0f;
          if (!REPEAT)
            for (int r = 1; r < reps; ++r) ds_mul(h, l, (float)ind, 0.0f, h, l);
          // an element without indicator points: a factor of 1e9 per pass
          if (!(h <= 3e38f)) h = 3e38f, l = 0.0f;
          reinterpret_cast<float2*>(sMr)[slot] = make_float2(h, l);
          sF[slot] = e >= 0 && (REPEAT || lin || h != 1.0f || l != 0.0f);
        } else {
          double m = ind;
          for (int r = 1; r < reps; ++r) m *= ind;
          if (!(m <= 1e308)) m = 1e308;
          sMr[slot] = m;
          sF[slot] = e >= 0 && (lin || m != 1.0);
        }
      }
      __syncthreads();
      if (lin) {
        // linearize (limiter_multiplier.cpp:101-178): mean + centre gradient
        // . (x_j - c); a linear state is its own linearisation, so once here
        // equals the reference's application before every multiplier pass
        for (int t = tid; t < EPB * NEQ; t += NT) {
          const int k = t / EPB, s = t - k * EPB;
          if (sE[s] < 0) continue;
          R* v = sU + t * NDP;
          float* vl = DS ? sLo + t * NDP : nullptr;
          double g[3] = {0.0, 0.0, 0.0};
#pragma unroll
          for (int d = 0; d < DIM; ++d)
#pragma unroll
            for (int j = 0; j < ND; ++j) {
              double x = (double)v[j];
              if constexpr (DS) x += (double)vl[j];
              g[d] += x * tab->dcen[j][d];
            }
          const double m = mean_value(prm, (long long)k * ne + sE[s]);
#pragma unroll
          for (int j = 0; j < ND; ++j) {
            double x = m;
#pragma unroll
            for (int d = 0; d < DIM; ++d) x -= g[d] * (0.5 - tab->xlin[j][d]);
            v[j] = (R)x;
            if constexpr (DS) vl[j] = (float)(x - (double)(float)x);
          }
        }
        __syncthreads();
      }
      if constexpr (LOW) {
        // what rounding the mean to FP64 left out: with it the limited values
        // average to the unrounded mean, and a limited run's rounding does not
        // accumulate one bit of every mean per stage
        for (int t = tid; t < EPB * NEQ; t += NT) {
          const int s = t % EPB;
          if (!sF[s]) continue;
          const double* w = tab->wmn_e ? tab->wmn_e + (long long)sE[s] * ND : tab->wmean;
          double l = 0.0;
#pragma unroll
          for (int j = 0; j < ND; ++j) l += w[j] * (sU[t * NDP + j] - sM[t]);
          sL[t] = l;
        }
        __syncthreads();
      }
      for (int t = tid; t < EPB * ND; t += NT) {
        const int s = t / ND, j = t - s * ND;
        if (!sF[s]) continue;
#pragma unroll
        for (int k = 0; k < NEQ; ++k) {
          R& v = sU[(k * EPB + s) * NDP + j];
          const MeanT um = sM[k * EPB + s];
          if constexpr (!F32) {
            const double l = LOW ? sL[k * EPB + s] : 0.0, d = v - um;
            v = um + (l + sMr[s] * (d - l));
          } else {
            const float2 m = reinterpret_cast<float2*>(sMr)[s];
            float h = v;
            if constexpr (DS) {
              float l = sLo[(k * EPB + s) * NDP + j];
              for (int r = 0; r < (REPEAT ? reps : 1); ++r) {
                ds_add(h, l, -um.x, -um.y);
                float ph, pl;
                if constexpr (REPEAT)
                  ds_mul_f(h, l, m.x, ph, pl);
                else
                  ds_mul(h, l, m.x, m.y, ph, pl);
                ds_add(ph, pl, um.x, um.y);
                h = ph;
                l = pl;
              }
              sLo[(k * EPB + s) * NDP + j] = l;
            } else {
              for (int r = 0; r < (REPEAT ? reps : 1); ++r) h = um.x + m.x * (h - um.x);
            }
            v = h;
          }
        }
      }
      if (prm.last_hope) {
        __syncthreads();
        bool bad = false;
        if (e >= 0) {
          for (int v = lane; v < NV; v += L) {
            R fv[NEQ];
#pragma unroll
            for (int k = 0; k < NEQ; ++k) {
              R s = R(0);
#pragma unroll
              for (int j = 0; j < ND; ++j) {
                s += sU[(k * EPB + slot) * NDP + j] * sBv[j * NV + v];
                if constexpr (DS) s += sLo[(k * EPB + slot) * NDP + j] * sBv[j * NV + v];
              }
              fv[k] = s;
            }
            bad |= !vertex_is_physical<DIM>(fv, sG[slot], sG[EPB + slot]);
          }
        }
        const unsigned all = __ballot_sync(0xffffffffu, bad);
        const int g0 = (tid & 31) / L * L;
        if (lane == 0 && ((all >> g0) & ((1u << L) - 1u))) sF[slot] = 3;
      }
      __syncthreads();
    }
    for (int t = tid; t < EPB * ND; t += NT) {
      const int s = t / ND, j = t - s * ND, f = sF[s];
      if (!f) continue;
      const long long i0 = (long long)sE[s] * ND + j;
#pragma unroll
      for (int k = 0; k < NEQ; ++k) {
        const MeanT um = sM[k * EPB + s];
        if constexpr (F32) {
          u[k * NDa + i0] = (f & 2) ? um.x : sU[(k * EPB + s) * NDP + j];
          if constexpr (DS) ulo[k * NDa + i0] = (f & 2) ? um.y : sLo[(k * EPB + s) * NDP + j];
        } else {
          u[k * NDa + i0] = (f & 2) ? um : sU[(k * EPB + s) * NDP + j];
        }
      }
    }
    if (!MAP || (long long)(blk + gridDim.x) * EPB >= prm.act_cum[*prm.act_n]) break;
    __syncthreads();
  }
}

}  // namespace rkdg
