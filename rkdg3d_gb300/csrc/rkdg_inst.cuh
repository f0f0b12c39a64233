// Explicit instantiation helpers for the generic kernels (one translation
// unit per geometry keeps the build parallel).
#pragma once

#include <algorithm>

#include "rkdg_generic.cuh"
#include "rkdg_launch.h"
#include "rkdg_limit.cuh"
#include "rkdg_planar.cuh"

namespace rkdg {

constexpr int kGenericBlock = 128;

// Threads per CTA: the tuned value (a multiple of 32 up to kGenericMaxBlock)
// or the default.
inline int generic_block(int b) {
  return (b >= 32 && b <= kGenericMaxBlock && b % 32 == 0) ? b : kGenericBlock;
}

// Threads per CTA of a pass over n work items: at most `most`, halved while a
// small mesh would leave SMs without a CTA.
inline int spread_block(long long n, int most) {
  int b = most;
  while (b > 32 && n < 152LL * b) b >>= 1;
  return b;
}

// CTAs of a batch's face pass and limiter, which loop over the active work: a
// CTA past it costs its launch and two loads, so at most 64 per SM (256 strips of
// 4,400 quads need 35,000 with every problem active, and run two thirds of their
// steps with less than half of them).
inline unsigned batch_grid(unsigned grid) { return std::min(grid, 152u * 64u); }

template <int G, int P, typename R>
cudaError_t launch_planar(const RhsParams& prm, const R* u, const EpiParams<R>& ep, cudaStream_t st) {
  if (!prm.flist || !prm.fslot) return cudaErrorInvalidValue;
  const long long npt = (long long)prm.nface * El<G, P>::NQF;
  const int blk = prm.block ? generic_block(prm.block) : spread_block(npt, 128);
  const unsigned grid = (unsigned)((npt + blk - 1) / blk);
  if (prm.faces_only) {
    if (prm.act_cum)
      k_face_planar<G, P, R, true, true><<<batch_grid(grid), blk, 0, st>>>(prm, u);
    else
      k_face_planar<G, P, R, true, false><<<grid, blk, 0, st>>>(prm, u);
    return cudaGetLastError();
  }
  if (prm.act_cum)
    k_face_planar<G, P, R, false, true><<<batch_grid(grid), blk, 0, st>>>(prm, u);
  else
    k_face_planar<G, P, R, false, false><<<grid, blk, 0, st>>>(prm, u);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  using S = Planar<G, P>;
  constexpr bool F32 = std::is_same<R, float>::value;
  if constexpr (F32 && El<G, P>::NEQ * El<G, P>::ND <= 16) {
    const int eb = prm.block ? std::min(generic_block(prm.block), 128) : spread_block(prm.ne, 128);
    k_elem_planar<G, P, R><<<(prm.ne + eb - 1) / eb, eb, 0, st>>>(prm, u, ep);
  } else if (prm.ne < 152 * S::EPB) {
    k_node_planar<G, P, R, S::SMALL><<<(prm.ne + S::SMALL - 1) / S::SMALL, S::threads(S::SMALL), 0, st>>>(prm, u, ep);
  } else {
    k_node_planar<G, P, R, S::EPB><<<(prm.ne + S::EPB - 1) / S::EPB, S::NT, 0, st>>>(prm, u, ep);
  }
  return cudaGetLastError();
}

template <int G, int P>
cudaError_t launch_rhs_t(int prec, const RhsParams& prm, const void* u, const void* ep,
                         cudaStream_t st) {
  return prec == 0 ? launch_planar<G, P, double>(prm, (const double*)u, *(const EpiParams<double>*)ep, st)
                   : launch_planar<G, P, float>(prm, (const float*)u, *(const EpiParams<float>*)ep, st);
}

// Threads per CTA of the limiter: the tuned value, or by the mesh's size.
inline int limit_block(int tuned, int ne, int lanes) {
  if (tuned >= 32 && tuned <= kGenericMaxBlock && tuned % 32 == 0) return tuned;
  return spread_block((long long)ne * lanes, 128);
}

template <int G, int P, typename R, bool DS>
cudaError_t launch_limit_mode(const LimParams& prm, R* u, float* ulo, cudaStream_t st) {
  using T = LimTeam<G, P>;
  if (prm.indicator == 3) {
    const int blk = std::min(generic_block(prm.block), generic_max_block<R, El<G, P>::NEQ * El<G, P>::ND>());
    k_limit_shu<G, P, R, DS><<<(prm.ne + blk - 1) / blk, blk, 0, st>>>(prm, u, ulo);
    return cudaGetLastError();
  }
  static_assert(T::template smem_bytes<R, DS>(T::MAX_BLOCK) <= 48 * 1024, "shared memory of the largest CTA");
  const int blk = limit_block(prm.block, prm.ne, T::L), epb = blk / T::L;
  const unsigned grid = (unsigned)((prm.ne + epb - 1) / epb);
  const size_t smem = T::template smem_bytes<R, DS>(blk);
  if constexpr (G != 5) {  // batches are planar
    if (prm.act_cum) {
      k_limit_team<G, P, R, DS, true><<<batch_grid(grid), blk, smem, st>>>(prm, u, ulo);
      return cudaGetLastError();
    }
  }
  k_limit_team<G, P, R, DS, false><<<grid, blk, smem, st>>>(prm, u, ulo);
  return cudaGetLastError();
}

template <int G, int P>
cudaError_t launch_limit_t(int mode, const LimParams& prm, void* u, float* ulo, cudaStream_t st) {
  if (mode == 0) return launch_limit_mode<G, P, double, false>(prm, (double*)u, nullptr, st);
  if (mode == 1) return launch_limit_mode<G, P, float, false>(prm, (float*)u, nullptr, st);
  return launch_limit_mode<G, P, float, true>(prm, (float*)u, ulo, st);
}

template <int G, int P>
cudaError_t launch_means_t(int mode, int ne, long long ndofs, const RefTables* tab, const void* u,
                           const float* ulo, double* means, cudaStream_t st) {
  const int grid = (ne + kGenericBlock - 1) / kGenericBlock;
  if (mode == 0)
    k_means_generic<G, P, double><<<grid, kGenericBlock, 0, st>>>(ne, ndofs, tab, (const double*)u,
                                                                  nullptr, means);
  else
    k_means_generic<G, P, float><<<grid, kGenericBlock, 0, st>>>(
        ne, ndofs, tab, (const float*)u, mode == 2 ? ulo : nullptr, means);
  return cudaGetLastError();
}

#define RKDG_INSTANTIATE(G, P)                                                                 \
  template cudaError_t launch_rhs_t<G, P>(int, const RhsParams&, const void*, const void*,     \
                                          cudaStream_t);                                       \
  template cudaError_t launch_limit_t<G, P>(int, const LimParams&, void*, float*, cudaStream_t); \
  template cudaError_t launch_means_t<G, P>(int, int, long long, const RefTables*, const void*, \
                                            const float*, double*, cudaStream_t);

}  // namespace rkdg
