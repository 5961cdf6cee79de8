// Explicit instantiation of the Dslash kernel family for one precision; each
// precision lives in its own translation unit so they compile in parallel.
#pragma once

#include <type_traits>

#include "qpx_finalize.cuh"
#include "qpx_host.h"

namespace qpx {

inline void check_pdl(cudaError_t e)
{
  if (e != cudaSuccess) throw Error(QPHIX_GPU_ECUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
}

// Four blocks of the 16-bit one-site kernels fit on a multiprocessor, two or
// three of the others: half their number counts for programmatic dependent
// launch, so that it starts where the launch fills the device once.  With it
// from 296 blocks on, InvRichardsonMultiPrec with FP16 inside took 2 to 3 %
// longer than the two-site form of fewer than 296 blocks (18x8x14x16 x 3 rhs,
// us per operator application: 39.5, two sites 38.6, this 36.4; 16^3x20 x 1
// 41.3, 41.2, 38.2).
template <typename P, int RECON, int R, int S, int SP, int GEN, bool RL = false>
void launch_dslash_k(int epi, int achi, const DslashArgs &a, dim3 grid, cudaStream_t st)
{
  const long long size = (long long)grid.x * grid.y / (P::has_norm && SP == 1 && R == 1 ? 2 : 1);
  auto go = [&](auto kernel) { check_pdl(launch_pdl(kernel, grid, dim3(QPX_BLOCK), st, size, a)); };
  if (achi == ACHI_NONE) {
    switch (epi) {
    case EPI_NONE: return go(dslash_kernel<P, RECON, EPI_NONE, ACHI_NONE, R, S, SP, GEN, RL>);
    case EPI_CLOV: return go(dslash_kernel<P, RECON, EPI_CLOV, ACHI_NONE, R, S, SP, GEN, RL>);
    case EPI_TMINV: return go(dslash_kernel<P, RECON, EPI_TMINV, ACHI_NONE, R, S, SP, GEN, RL>);
    case EPI_FCLOV: return go(dslash_kernel<P, RECON, EPI_FCLOV, ACHI_NONE, R, S, SP, GEN, RL>);
    }
  } else if (epi == EPI_NONE) {
    switch (achi) {
    case ACHI_ALPHA: return go(dslash_kernel<P, RECON, EPI_NONE, ACHI_ALPHA, R, S, SP, GEN, RL>);
    case ACHI_CLOV: return go(dslash_kernel<P, RECON, EPI_NONE, ACHI_CLOV, R, S, SP, GEN, RL>);
    case ACHI_TM: return go(dslash_kernel<P, RECON, EPI_NONE, ACHI_TM, R, S, SP, GEN, RL>);
    }
  }
  throw Error(QPHIX_GPU_EINVAL, "unsupported dslash epilogue combination");
}

// the two-flavour twisted-mass kernels (two right-hand sides per thread)
template <typename P, int RECON, int S>
void launch_dslash_nd(int epi, int achi, const DslashArgs &a, dim3 grid, cudaStream_t st)
{
  dim3 block(QPX_BLOCK);
  if (achi == ACHI_NONE && epi == EPI_NDTM)
    check_pdl(launch_pdl(dslash_kernel<P, RECON, EPI_NDTM, ACHI_NONE, 2, S, 1, GEN_NONE>, grid, block, st, (long long)grid.x * grid.y, a));
  else if (epi == EPI_NONE && achi == ACHI_NDTM)
    check_pdl(launch_pdl(dslash_kernel<P, RECON, EPI_NONE, ACHI_NDTM, 2, S, 1, GEN_NONE>, grid, block, st, (long long)grid.x * grid.y, a));
  else if (achi == ACHI_NONE && epi == EPI_NDFCLOV)
    check_pdl(launch_pdl(dslash_kernel<P, RECON, EPI_NDFCLOV, ACHI_NONE, 2, S, 1, GEN_NONE>, grid, block, st, (long long)grid.x * grid.y, a));
  else if (epi == EPI_NONE && achi == ACHI_NDCLOV)
    check_pdl(launch_pdl(dslash_kernel<P, RECON, EPI_NONE, ACHI_NDCLOV, 2, S, 1, GEN_NONE>, grid, block, st, (long long)grid.x * grid.y, a));
  else
    throw Error(QPHIX_GPU_EINVAL, "unsupported two-flavour dslash combination");
}

// isign is a template parameter: the projector signs become adds / subtracts
template <typename P, int RECON, int R, int SP, int GEN, bool RL = false>
void launch_dslash_s(int epi, int achi, const DslashArgs *a, dim3 grid, cudaStream_t st)
{
  if (!a) return;  // shape query
  if (a->isign == 1)
    launch_dslash_k<P, RECON, R, 1, SP, GEN, RL>(epi, achi, *a, grid, st);
  else
    launch_dslash_k<P, RECON, R, -1, SP, GEN, RL>(epi, achi, *a, grid, st);
}

// The shapes built for storage P.  a == nullptr: only report whether the
// shape exists.  Returns false for a shape that is not built.
//   general path (dir mask, halo, twisted phases) and phases alone: R = 1, SP = 1
//   fast path: R = 1 SP = 1 for every precision; for FP32 arithmetic also
//   SP = 2 (both link kinds), R = 2 (12-real links) and two right-hand sides
//   in the float2 lanes (rl, 12-real links, even nrhs)
template <typename P>
bool launch_dslash_p(int recon, int epi, int achi, const DslashShape &sh, const DslashArgs *a, dim3 grid,
                     cudaStream_t st)
{
  constexpr bool fp32 = std::is_same<typename P::real, float>::value;
  if (recon != 12 && recon != 18) return false;
  if (is_two_flavour(epi, achi)) {  // two-flavour twisted mass (clover): R = 2 only
    if (sh.R != 2 || sh.SP != 1 || sh.gen) return false;
    if (!a) return true;
    const bool plus = a->isign == 1;
    if (recon == 12)
      plus ? launch_dslash_nd<P, 12, 1>(epi, achi, *a, grid, st) : launch_dslash_nd<P, 12, -1>(epi, achi, *a, grid, st);
    else
      plus ? launch_dslash_nd<P, 18, 1>(epi, achi, *a, grid, st) : launch_dslash_nd<P, 18, -1>(epi, achi, *a, grid, st);
    return true;
  }
  if (sh.rl) {
    if constexpr (fp32) {
      if (sh.R != 1 || sh.SP != 2 || sh.gen || recon != 12) return false;
      if (a && a->nrhs % 2) return false;
      launch_dslash_s<P, 12, 1, 2, GEN_NONE, true>(epi, achi, a, grid, st);
      return true;
    }
    return false;
  }
  if (sh.gen) {
    if (sh.R != 1 || sh.SP != 1) return false;
    if (sh.phases) {
      recon == 12 ? launch_dslash_s<P, 12, 1, 1, GEN_PHASES>(epi, achi, a, grid, st)
                  : launch_dslash_s<P, 18, 1, 1, GEN_PHASES>(epi, achi, a, grid, st);
      return true;
    }
    if (recon == 12)
      launch_dslash_s<P, 12, 1, 1, GEN_ALL>(epi, achi, a, grid, st);
    else
      launch_dslash_s<P, 18, 1, 1, GEN_ALL>(epi, achi, a, grid, st);
    return true;
  }
  if (sh.R == 1 && sh.SP == 1) {
    if (recon == 12)
      launch_dslash_s<P, 12, 1, 1, GEN_NONE>(epi, achi, a, grid, st);
    else
      launch_dslash_s<P, 18, 1, 1, GEN_NONE>(epi, achi, a, grid, st);
    return true;
  }
  if constexpr (fp32) {
    if (sh.R == 1 && sh.SP == 2) {
      if (recon == 12)
        launch_dslash_s<P, 12, 1, 2, GEN_NONE>(epi, achi, a, grid, st);
      else
        launch_dslash_s<P, 18, 1, 2, GEN_NONE>(epi, achi, a, grid, st);
      return true;
    }
    if (sh.R == 2 && sh.SP == 1 && recon == 12) {
      launch_dslash_s<P, 12, 2, 1, GEN_NONE>(epi, achi, a, grid, st);
      return true;
    }
  }
  return false;
}

}  // namespace qpx
