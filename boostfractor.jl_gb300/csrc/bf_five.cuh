// Variants and launches of the transform lengths 40, 80 and 160: the lengths
// 5 2^a between the powers of two, for boxes just above a quarter of one
// (2 * 38 - 1 <= 80 for the 0.15 m disk on the 128-point grid).
#pragma once

#include <initializer_list>

#include "bf_stage.cuh"

namespace bf {

// One fused variant: with `a` null whether it fits (0 or 1), else its launch
// (rc the CUDA status).
template <typename R, int N, bool JOINT, int THREADS, int MINB, int MODE>
static int five_one(const FusedArgs<cplx_t<R>>* a, int nby, int nsteps, cudaStream_t st, int* rc) {
  const size_t smem = fused_smem_for<N, MODE>(nby, sizeof(cplx_t<R>), JOINT ? 2 : 1, THREADS);
  if (smem > kMaxSmem || MINB * (smem + kSmemReservedPerCta) > kSmemPerSM) return 0;
  if (a) {
    note_launch();
    *rc = launch_fused_v<R, N, JOINT, Team<N>::RR / 2, THREADS, MINB, MODE>(*a, dim3(nsteps, a->nfreq), smem, st);
  }
  return 1;
}

// Threads and CTAs per SM.  40 teams (160 threads at length 80) take the 76 box
// rows of a joint step in two rounds and its 160 columns in four; 48 teams (96
// threads at length 40) the 36 rows in one, the 80 columns in two.  A thread
// holds 20 points (40 registers) and its 19 twiddles (38): 128 registers, 15
// warps per SM.  A full stage of 21 steps x 256 frequencies (38 x 38 box, length
// 80) took 235 us joint, 242 us joint with staged phasor rows, 282 us with
// separate slots; 263 us with 320 threads, and 295 us with separate slots, both
// at 96 registers and the twiddles in shared memory; the 128-point team kernels
// 574 us.  Two other shapes of the same stage were slower: two threads a line
// (the even and the odd bins of a half-filled line are independent transforms)
// 328 us, and one thread a line (255 registers, 8 warps per SM) 437 us; both
// halve the shared-memory traffic but leave too few warps to cover the loads
// at the ends of a step.
// Length 160 (40 points a thread) and complex128 read the twiddles from the
// shared table.  26 steps x 64 frequencies at length 160 (76 x 76 box): 453 us
// separate, 486 us joint, 597 us separate with 128 threads at 2 CTAs per SM.
template <typename R, int N>
static int five_case(int variant, const FusedArgs<cplx_t<R>>* a, int nby, int nsteps, cudaStream_t st, int* rc) {
  if constexpr (sizeof(R) == 8) {
    if (variant == kFusedSeparate) return five_one<R, N, false, 160, 1, kModeTwShared>(a, nby, nsteps, st, rc);
    if (variant == kFusedJoint) return five_one<R, N, true, 160, 1, kModeTwShared>(a, nby, nsteps, st, rc);
  } else if constexpr (N == 160) {
    if (variant == kFusedSeparate) return five_one<R, N, false, 320, 1, kModeTwShared>(a, nby, nsteps, st, rc);
    if (variant == kFusedJoint) return five_one<R, N, true, 256, 1, kModeTwShared>(a, nby, nsteps, st, rc);
  } else {
    constexpr int T = N == 40 ? 96 : 160, B = N == 40 ? 5 : 3;
    if (variant == kFusedSeparate) return five_one<R, N, false, T, B, 0>(a, nby, nsteps, st, rc);
    if (variant == kFusedJoint) return five_one<R, N, true, T, B, 0>(a, nby, nsteps, st, rc);
    if (variant == kFusedJointStaged) return five_one<R, N, true, T, B, kModeStage>(a, nby, nsteps, st, rc);
  }
  return 0;
}

template <typename R, int N>
static std::vector<int> five_variants_t(int nby) {
  std::vector<int> v = {kFusedRule};
  for (int k : std::initializer_list<int>{kFusedSeparate, kFusedJoint, kFusedJointStaged})
    if (five_case<R, N>(k, nullptr, nby, 0, 0, nullptr)) v.push_back(k);
  return v;
}

template <typename R, int N>
static int launch_five_t(const FusedArgs<cplx_t<R>>& a, int nsteps, cudaStream_t st) {
  constexpr int NZ = Team<N>::RR / 2;
  if ((std::max(a.nbx, a.nby) + Team<N>::G - 1) / Team<N>::G > NZ) return (int)cudaErrorInvalidValue;
  if (a.mg && split_stage(nsteps, a.nfreq)) return launch_split<R, N, NZ>(a, nsteps, st);
  int rc = (int)cudaErrorInvalidValue;
  // the variant asked for, else the rule: joint where its tiles fit
  for (int v : std::initializer_list<int>{a.variant, kFusedJoint, kFusedSeparate})
    if (five_case<R, N>(v, &a, a.nby, nsteps, st, &rc)) return rc;
  return a.mg ? launch_split<R, N, NZ>(a, nsteps, st) : rc;   // tiles above shared memory
}

}  // namespace bf
