// Explicit instantiation helpers for the generic kernels (one translation
// unit per geometry keeps the build parallel).
#pragma once

#include <algorithm>

#include "rkdg_generic.cuh"
#include "rkdg_launch.h"
#include "rkdg_limit.cuh"

namespace rkdg {

constexpr int kGenericBlock = 128;

// Threads per CTA: the tuned value (a multiple of 32 up to kGenericMaxBlock)
// or the default.
inline int generic_block(int b) {
  return (b >= 32 && b <= kGenericMaxBlock && b % 32 == 0) ? b : kGenericBlock;
}

template <int G, int P>
cudaError_t launch_rhs_t(int prec, const RhsParams& prm, const void* u, const void* ep,
                         cudaStream_t st) {
  constexpr int NVAL = El<G, P>::NEQ * El<G, P>::ND;
  const int blk = prec == 0 ? generic_block(prm.block)
                            : std::min(generic_block(prm.block), generic_max_block<float, NVAL>());
  const int grid = (prm.ne + blk - 1) / blk;
  if (prec == 0)
    k_rhs_generic<G, P, double><<<grid, blk, 0, st>>>(prm, (const double*)u,
                                                      *(const EpiParams<double>*)ep);
  else
    k_rhs_generic<G, P, float><<<grid, blk, 0, st>>>(prm, (const float*)u,
                                                     *(const EpiParams<float>*)ep);
  return cudaGetLastError();
}

// Threads per CTA of the limiter: the tuned value, or 128, halved while a
// small mesh would leave SMs without a CTA.
inline int limit_block(int tuned, int ne, int lanes) {
  if (tuned >= 32 && tuned <= kGenericMaxBlock && tuned % 32 == 0) return tuned;
  int b = 128;
  while (b > 32 && (long long)ne * lanes < 152LL * b) b >>= 1;
  return b;
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
  k_limit_team<G, P, R, DS><<<(prm.ne + epb - 1) / epb, blk, T::template smem_bytes<R, DS>(blk), st>>>(prm, u, ulo);
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
