// Device kernels of the GB300 boost-factor library.
//
// * k_fused_stage   -- the hot path: one launch runs one bounce stage of the
//   recursive Fourier propagation for every frequency of a batch.  Each CTA
//   propagates one or two region fields through the angular-spectrum
//   propagator (src/boost_fractor.jl:137-179) and applies the boundary's
//   reflection/transmission (src/boost_fractor_recurprop.jl:90-120, 310-345)
//   in its epilogue.  Fields are stored only on the pruned box of pixels the
//   disk mask can reach; the 2D FFT is separable, so the forward row pass,
//   the fused column pass (FFT, phasor, inverse FFT) and the inverse row pass
//   each touch only the lines that can be non-zero or are needed.
// * phasor / tilt table kernels -- FP64 phase arguments, stored in the field
//   precision.
// * general full-grid path -- any grid size (also odd sizes like 101), used
//   for the per-op propagator, the exit fields and the exact (unpruned) mode.
// * 1D-propagator solvers -- every pixel is independent.
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "bf_common.cuh"
#include "bf_device.cuh"
#include "bf_stage.cuh"

namespace bf {

// Kernel launches made by the calling host thread (one handle's call runs on
// one thread, so per-call differences are exact even with several handles
// working concurrently).
static thread_local unsigned long long g_launches = 0;
unsigned long long launch_count() { return g_launches; }
void note_launch() { ++g_launches; }
void note_launches(unsigned long long n) { g_launches += n; }
void unnote_launches(unsigned long long n) { g_launches -= n; }
#define COUNT_LAUNCH() (++g_launches)

void fill_roots(int n, double2* hd, float2* hf) {
  for (int k = 0; k < n; ++k) {
    // cos/sin evaluated on the first octant and mapped by symmetry so that
    // the table is exactly symmetric
    int q = k / (n / 4), r = k % (n / 4);
    double c, s;
    int rr = r <= n / 8 ? r : n / 4 - r;
    double a = 2.0 * M_PI * rr / n;
    double cr = cos(a), sr = sin(a);
    if (r > n / 8) { double t = cr; cr = sr; sr = t; }
    // float copy of the first-octant pair, rounded for the smallest modulus error,
    // then mapped by the same exact symmetry as the FP64 pair
    const float2 o = round_c64_host_device(cr, sr);
    float cf, sf;
    // angle theta = 2 pi k / n = q*pi/2 + 2 pi r/n; (cos, sin) of theta
    switch (q) {
      case 0: c = cr; s = sr; cf = o.x; sf = o.y; break;
      case 1: c = -sr; s = cr; cf = -o.y; sf = o.x; break;
      case 2: c = -cr; s = -sr; cf = -o.x; sf = -o.y; break;
      default: c = sr; s = -cr; cf = o.y; sf = -o.x; break;
    }
    hd[k] = make_double2(c, -s);
    hf[k] = make_float2(cf, -sf);
  }
}

void init_constant_roots() {
  upload_roots();
  init_roots_five_f();
  init_roots_five_d();
}

// ---------------------------------------------------------------------------
// small FP64 complex helpers (phase arguments are always FP64)
// ---------------------------------------------------------------------------
__device__ __forceinline__ double2 dcsqrt(double x, double y) {
  // principal square root honouring the sign of a zero imaginary part, so that
  // sqrt(a - 0.0im) = 0 - sqrt(|a|)im for a < 0 (evanescent bins decay)
  if (x == 0.0 && y == 0.0) return make_double2(0.0, y);
  // a zero imaginary part (real permittivities): with hypot(x, 0) = |x| the
  // general formula below reduces to these values in exact arithmetic; they
  // skip hypot and the division (FP64 runs at 1/64 of the FP32 rate)
  if (y == 0.0) return x > 0.0 ? make_double2(sqrt(x), y) : make_double2(0.0, copysign(sqrt(-x), y));
  double t = sqrt((fabs(x) + hypot(x, y)) * 0.5);
  if (x >= 0.0) return make_double2(t, y / (2.0 * t));
  return make_double2(fabs(y) / (2.0 * t), copysign(t, y));
}
__device__ __forceinline__ double2 dcexp(double re, double im) {
  double s, c;
  sincos(im, &s, &c);
  if (re == 0.0) return make_double2(c, s);   // exp(0) = 1 exactly (propagating bins)
  double m = exp(re);
  return make_double2(m * c, m * s);
}
// k0 = 2 pi / lambda * sqrt(eps), eps real -> re - 0.0im (src/boost_fractor.jl:140,:161)
__device__ __forceinline__ double2 k0_of(double lambda, double eps_re, double eps_im) {
  if (eps_im == 0.0) eps_im = -0.0;
  double2 s = dcsqrt(eps_re, eps_im);
  double c = 2.0 * M_PI / lambda;
  return make_double2(c * s.x, c * s.y);
}
// exp(-1im * sqrt(k0^2 - kx^2 - ky^2) * dz)
__device__ __forceinline__ double2 phasor_value(double2 k0, double kx, double ky, double dz) {
  double2 k0sq = make_double2(k0.x * k0.x - k0.y * k0.y, k0.x * k0.y + k0.y * k0.x);
  double re = (k0sq.x - kx * kx) - ky * ky;
  double2 kz = dcsqrt(re, k0sq.y);
  // -1im * kz * dz = (kz.y * dz, -kz.x * dz)
  return dcexp(kz.y * dz, -kz.x * dz);
}
// exp(-1im * k0 * t) for complex k0 and real t
__device__ __forceinline__ double2 phase_k0(double2 k0, double t) {
  return dcexp(k0.y * t, -k0.x * t);
}
// exp(-1im * k0 * s) for complex k0 and complex s
__device__ __forceinline__ double2 phase_k0c(double2 k0, double2 s) {
  double re = k0.x * s.x - k0.y * s.y, im = k0.x * s.y + k0.y * s.x;
  return dcexp(im, -re);
}

#define SPEED_OF_LIGHT 299792458.0

static int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 1;
  }
  return n;
}

// Whether stages of this transform length may take the split-phase path.
bool split_length(int N) { return N >= 40; }

// Bytes of the split-phase row tiles for a stage of `nsteps` steps.
size_t split_tile_bytes(int N, int nby, int nfreq, int nsteps, bool fp64) {
  return (size_t)nsteps * nfreq * 2 * nby * pitch_of(N) * (fp64 ? 16 : 8);
}

// Whether a stage of `nsteps` steps x `nfreq` frequencies takes the split path.
bool split_stage(int nsteps, int nfreq) { return (long long)nsteps * nfreq < sm_count(); }

// One launch for a run of split stages while a phase has at most 4 warps an SM: above, the phases are bound by the FP64
// pipe, and larger CTAs in separate launches are as fast (dancer at 64^2, 31 stages: 1 frequency 1.20 -> 1.13 ms, 4
// 2.13 -> 1.20 ms; 5 and more take the launches).  complex64, which has no such pipe, stays with the launches (0.65
// against 0.75 ms).
bool split_run_fits(int N, int nsteps, int nfreq) {
  const int lanes = N == 40 || N == 80 || N == 160 ? 4 : N >= 256 ? 16 : 8;   // a line's threads, at least
  return (long long)nsteps * nfreq * 2 * N * lanes / 32 <= 4LL * sm_count();
}

static size_t smem_for(int N, int nby, size_t csz) {
  switch (N) {
    case 8: return fused_smem_for<8>(nby, csz);
    case 16: return fused_smem_for<16>(nby, csz);
    case 32: return fused_smem_for<32>(nby, csz);
    case 40: return fused_smem_for<40>(nby, csz, 1, 96);
    case 80: return fused_smem_for<80, kModeTwShared>(nby, csz, 1, 160);
    case 160: return fused_smem_for<160, kModeTwShared>(nby, csz, 1, 320);
    case 64: return fused_smem_for<64>(nby, csz);
    case 128: return fused_smem_for<128>(nby, csz);
    case 256: return fused_smem_for<256>(nby, csz);
    default: return (size_t)-1;
  }
}

size_t fused_smem_bytes(int N, int nbx, int nby, bool fp64) {
  (void)nbx;
  return smem_for(N, nby, fp64 ? 16 : 8);
}

bool fused_split_only(int N, int nbx, int nby, bool fp64) {
  return split_length(N) && fused_smem_bytes(N, nbx, nby, fp64) > kMaxSmem;
}

bool fused_supported(int N, int nbx, int nby, bool fp64) {
  const bool five = N == 80 || (!fp64 && (N == 40 || N == 160));
  if (N < 8 || N > 256 || ((N & (N - 1)) && !five)) return false;
  if (nbx < 1 || nby < 1 || nbx > N || nby > N) return false;
  // row tiles too large for shared memory (complex128 at 256^2): every stage
  // takes the split-phase path, whose tiles live in global memory
  return fused_smem_bytes(N, nbx, nby, fp64) <= kMaxSmem || fused_split_only(N, nbx, nby, fp64);
}

// Register slots a box line may occupy in the pruned variants (complex64 for
// N >= 64, complex128 for N = 64, 128): half of them, since a transform of the
// truncated kernel (compact_length) is at least twice as long as the box.
template <int N> constexpr int pruned_slots() { return Team<N>::RR / 2; }

// Shape of one fused-stage launch: shared memory of the single and doubled
// (joint) row tiles and whether the rule takes the joint path.
struct FusedShape {
  size_t smem, smem_j, smem512, smem_jl, smem_sl, smem_js, smem_ss, smem_s5;
  bool joint_rule, joint_fits, wide_fits;
  // complex64, N = 128: joint steps with 320 threads at 2 CTAs per SM and
  // shared twiddles (lean), separate slots at 3 CTAs per SM and shared
  // twiddles (lean), joint steps with staged phasor rows, separate slots at 3
  // CTAs per SM with shared twiddles and staged phasor rows, separate slots
  // with 20 teams (160 threads: 38 box rows in two rounds) at 3 CTAs per SM
  // with staged phasor rows
  bool joint_lean_fits, sep_lean_fits, joint_staged_fits, sep_staged_fits, sep5_staged_fits;
};
constexpr int kLeanJointThreads = 320, kSep5Threads = 160;
constexpr int kModeLean = kModeTwShared | kModeHalf;
constexpr int kModeHalfStaged = kModeHalf | kModeStage;
constexpr int kModeLeanStaged = kModeTwShared | kModeHalf | kModeStage;
template <int N>
static FusedShape fused_shape(int nby, size_t csz) {
  FusedShape f;
  f.smem = fused_smem_for<N>(nby, csz, 1);
  f.smem_j = fused_smem_for<N>(nby, csz, 2);
  f.smem512 = fused_smem_for<N>(nby, csz, 1, 512);
  // the joint path when the doubled row tile keeps as many CTAs per SM
  const int ctas = (csz == 8 && N <= 128) ? 2 : 1;
  f.joint_fits = f.smem_j <= kMaxSmem;
  f.joint_rule = f.joint_fits && (size_t)ctas * (f.smem_j + kSmemReservedPerCta) <= kSmemPerSM &&
                 (size_t)ctas * (f.smem + kSmemReservedPerCta) <= kSmemPerSM;
  f.wide_fits = csz == 8 && N == 256 && f.smem512 <= kMaxSmem;
  f.smem_jl = fused_smem_for<N, kModeLean>(nby, csz, 2, kLeanJointThreads);
  f.smem_sl = fused_smem_for<N, kModeLean>(nby, csz, 1, kFusedThreads);
  f.smem_js = fused_smem_for<N, kModeHalfStaged>(nby, csz, 2, kFusedThreads);
  f.smem_ss = fused_smem_for<N, kModeLeanStaged>(nby, csz, 1, kFusedThreads);
  f.smem_s5 = fused_smem_for<N, kModeHalfStaged>(nby, csz, 1, kSep5Threads);
  const bool c128 = csz == 8 && N == 128;
  f.joint_lean_fits = c128 && 2 * (f.smem_jl + kSmemReservedPerCta) <= kSmemPerSM;
  f.sep_lean_fits = c128 && 3 * (f.smem_sl + kSmemReservedPerCta) <= kSmemPerSM;
  f.joint_staged_fits = c128 && 2 * (f.smem_js + kSmemReservedPerCta) <= kSmemPerSM;
  f.sep_staged_fits = c128 && 3 * (f.smem_ss + kSmemReservedPerCta) <= kSmemPerSM;
  f.sep5_staged_fits = c128 && 3 * (f.smem_s5 + kSmemReservedPerCta) <= kSmemPerSM;
  return f;
}

template <int N>
static std::vector<int> fused_variants_t(int nbx, int nby, bool fp64) {
  const FusedShape f = fused_shape<N>(nby, fp64 ? 16 : 8);
  // the lean variants exist for boxes within the pruned register slots only
  const bool pruned = (std::max(nbx, nby) + Team<N>::G - 1) / Team<N>::G <= pruned_slots<N>();
  std::vector<int> v = {kFusedRule};
  if (f.smem > kMaxSmem) return v;
  v.push_back(kFusedSeparate);
  if (f.joint_fits) v.push_back(kFusedJoint);
  if (f.wide_fits) v.push_back(kFusedWide);
  if (f.joint_lean_fits && pruned) v.push_back(kFusedJointLean);
  if (f.sep_lean_fits && pruned) v.push_back(kFusedSeparateLean);
  if (f.joint_staged_fits && pruned) v.push_back(kFusedJointStaged);
  if (f.sep_staged_fits && pruned) v.push_back(kFusedSeparateStaged);
  if (f.sep5_staged_fits && pruned) v.push_back(kFusedSeparate160Staged);
  return v;
}

std::vector<int> fused_variants(int N, int nbx, int nby, bool fp64) {
  switch (N) {
    case 8: return fused_variants_t<8>(nbx, nby, fp64);
    case 16: return fused_variants_t<16>(nbx, nby, fp64);
    case 32: return fused_variants_t<32>(nbx, nby, fp64);
    case 40:
    case 80:
    case 160: return fp64 ? five_variants_d(N, nby) : five_variants_f(N, nby);
    case 64: return fused_variants_t<64>(nbx, nby, fp64);
    case 128: return fused_variants_t<128>(nbx, nby, fp64);
    case 256: return fused_variants_t<256>(nbx, nby, fp64);
    default: return {kFusedRule};
  }
}

template <typename R, int N>
static int launch_fused_t(const FusedArgs<cplx_t<R>>& a, int nsteps, cudaStream_t st) {
  const size_t csz = sizeof(cplx_t<R>);
  const FusedShape sh = fused_shape<N>(a.nby, csz);
  const size_t smem = sh.smem, smem_j = sh.smem_j;
  const bool split_only = smem > kMaxSmem;   // every stage in global-memory row tiles
  if (split_only && !(a.mg && N >= 64)) return (int)cudaErrorInvalidValue;
  constexpr int G = Team<N>::G, RR = Team<N>::RR;
  const int rv = (std::max(a.nbx, a.nby) + G - 1) / G;
  if (a.mg && N >= 64 && (split_only || split_stage(nsteps, a.nfreq))) {
    if constexpr ((sizeof(R) == 4 && N >= 64) || (sizeof(R) == 8 && (N == 64 || N == 128)))
      if (rv <= pruned_slots<N>()) return launch_split<R, N, pruned_slots<N>()>(a, nsteps, st);
    return launch_split<R, N, RR>(a, nsteps, st);
  }
  // the variant: the rule's choice, or one picked by the autotuner (an
  // invalid choice falls back to the rule)
  bool joint = sh.joint_rule, wide = sh.wide_fits && !sh.joint_rule;
  if (a.variant == kFusedSeparate) {
    joint = false;
    wide = false;
  } else if (a.variant == kFusedJoint && sh.joint_fits) {
    joint = true;
    wide = false;
  } else if (a.variant == kFusedWide && sh.wide_fits) {
    joint = false;
    wide = true;
  }
  dim3 grid(nsteps, a.nfreq);
  COUNT_LAUNCH();
  if constexpr (sizeof(R) == 4 && N == 128) {
    if (rv <= pruned_slots<N>()) {
      constexpr int NZ = pruned_slots<N>();
      if (a.variant == kFusedJointLean && sh.joint_lean_fits)
        return launch_fused_v<R, N, true, NZ, kLeanJointThreads, 2, kModeLean>(a, grid, sh.smem_jl, st);
      if (a.variant == kFusedSeparateLean && sh.sep_lean_fits)
        return launch_fused_v<R, N, false, NZ, kFusedThreads, 3, kModeLean>(a, grid, sh.smem_sl, st);
      if (a.variant == kFusedJointStaged && sh.joint_staged_fits)
        return launch_fused_v<R, N, true, NZ, kFusedThreads, 2, kModeHalfStaged>(a, grid, sh.smem_js, st);
      if (a.variant == kFusedSeparateStaged && sh.sep_staged_fits)
        return launch_fused_v<R, N, false, NZ, kFusedThreads, 3, kModeLeanStaged>(a, grid, sh.smem_ss, st);
      if (a.variant == kFusedSeparate160Staged && sh.sep5_staged_fits)
        return launch_fused_v<R, N, false, NZ, kSep5Threads, 3, kModeHalfStaged>(a, grid, sh.smem_s5, st);
    }
  }
  if constexpr (sizeof(R) == 4 && N == 256) {
    // one CTA per SM (the 256-point row tile): 512 threads (32 teams, at most
    // 128 registers each) when the team scratch still fits beside the tile
    if (wide)
      return rv <= pruned_slots<N>() ? launch_fused_v<R, N, false, pruned_slots<N>(), 512>(a, grid, sh.smem512, st)
                                     : launch_fused_v<R, N, false, Team<N>::RR, 512>(a, grid, sh.smem512, st);
  }
  if constexpr ((sizeof(R) == 4 && N >= 64) || (sizeof(R) == 8 && (N == 64 || N == 128))) {
    if (rv <= pruned_slots<N>())
      return joint ? launch_fused_v<R, N, true, pruned_slots<N>()>(a, grid, smem_j, st)
                   : launch_fused_v<R, N, false, pruned_slots<N>()>(a, grid, smem, st);
  }
  return joint ? launch_fused_v<R, N, true, RR>(a, grid, smem_j, st) : launch_fused_v<R, N, false, RR>(a, grid, smem, st);
}

template <typename R>
static int launch_fused_dispatch(int N, const FusedArgs<cplx_t<R>>& a, int nsteps, cudaStream_t st) {
  if (nsteps <= 0 || a.nfreq <= 0) return 0;
  switch (N) {
    case 8: return launch_fused_t<R, 8>(a, nsteps, st);
    case 16: return launch_fused_t<R, 16>(a, nsteps, st);
    case 32: return launch_fused_t<R, 32>(a, nsteps, st);
    case 40:
    case 80:
    case 160:
      if constexpr (sizeof(R) == 4) return launch_five_f(N, a, nsteps, st);
      else return launch_five_d(N, a, nsteps, st);
    case 64: return launch_fused_t<R, 64>(a, nsteps, st);
    case 128: return launch_fused_t<R, 128>(a, nsteps, st);
    case 256: return launch_fused_t<R, 256>(a, nsteps, st);
    default: return (int)cudaErrorInvalidValue;
  }
}

int launch_fused_stage_f(int N, const FusedArgs<float2>& a, int nsteps, cudaStream_t st) {
  return launch_fused_dispatch<float>(N, a, nsteps, st);
}
int launch_fused_stage_d(int N, const FusedArgs<double2>& a, int nsteps, cudaStream_t st) {
  return launch_fused_dispatch<double>(N, a, nsteps, st);
}

// ---------------------------------------------------------------------------
// Phasor and tilt tables
// ---------------------------------------------------------------------------
template <typename C>
__global__ void k_phasor_table(C* out, const double* freqs, int stride, const int* regions,
                               const RegionGeo* geo, int N, const double* kX, const double* kY,
                               int fold) {
  const int W = fold ? N / 2 : N;
  const int per = W * W;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  const int t = blockIdx.y, f = blockIdx.z;
  if (idx >= per) return;
  const int kxb = idx / W, kyb = idx % W;
  const int sx = (kxb + N / 2) % N, sy = (kyb + N / 2) % N;
  const RegionGeo gg = geo[regions[t]];
  const double lambda = SPEED_OF_LIGHT / freqs[f];
  const double2 k0 = k0_of(lambda, gg.eps_re, gg.eps_im);
  double2 v = phasor_value(k0, kX[sx], kY[sy], gg.dz);
  const double sc = 1.0 / ((double)N * (double)N);   // a power of two: exact
  out[((size_t)f * stride + t) * per + idx] = from_d_phase<C>(make_double2(v.x * sc, v.y * sc));
}

int launch_phasor_table(bool fp64, void* out, int nfreq, const double* d_freqs, int ntab, int stride,
                        const int* d_regions, const RegionGeo* d_geo, int N, const double* d_kX,
                        const double* d_kY, int fold, cudaStream_t st) {
  if (ntab <= 0 || nfreq <= 0) return 0;
  const int W = fold ? N / 2 : N;
  dim3 grid((W * W + 255) / 256, ntab, nfreq);
  if (fp64) { COUNT_LAUNCH(); k_phasor_table<double2><<<grid, 256, 0, st>>>((double2*)out, d_freqs, stride, d_regions, d_geo, N, d_kX, d_kY, fold); }
  else { COUNT_LAUNCH(); k_phasor_table<float2><<<grid, 256, 0, st>>>((float2*)out, d_freqs, stride, d_regions, d_geo, N, d_kX, d_kY, fold); }
  return (int)cudaGetLastError();
}

// Spectrum of the truncated kernel (see compact_length) of one (frequency,
// region) per CTA: S = Ax^T D Ay over one quadrant, D the N x N grid's phasors
// at the non-negative wavenumbers and A the real matrix of compact_matrix
// (weights, both cosine sums and all scales included).  blockIdx.z takes a
// slice of BS columns of S.  Rows of D are evaluated kChunk at a time, reduced
// to BS columns, and added to the CTA's S in registers (E per thread).
// Bound by the FP64 pipe (2 FMA per clock and SM): for N = 128 to length 80 a
// table takes 4096 phasors and 532k real FMAs, about equal shares; operands
// come from L1 and shared memory far faster than that.
constexpr int kChunk = 16;
template <typename C, int E>
__global__ void __launch_bounds__(256) k_compact_table(C* out, const double* freqs, int stride, const int* regions,
                                                       const RegionGeo* geo, int Q, int first, const double* kX,
                                                       const double* kY, const double* A, int H, int BS) {
  extern __shared__ __align__(16) unsigned char sm[];
  double2* D = reinterpret_cast<double2*>(sm);   // [kChunk][Q]
  double2* T = D + kChunk * Q;                   // [kChunk][BS]
  const int tid = threadIdx.x, b0 = blockIdx.z * BS;
  const RegionGeo gg = geo[regions[blockIdx.x]];
  const double2 k0 = k0_of(SPEED_OF_LIGHT / freqs[blockIdx.y], gg.eps_re, gg.eps_im);
  double2 s[E];
#pragma unroll
  for (int i = 0; i < E; ++i) s[i] = make_double2(0.0, 0.0);
  for (int x0 = 0; x0 < Q; x0 += kChunk) {
    const int nx = min(kChunk, Q - x0);
    for (int i = tid; i < nx * Q; i += 256)
      D[i] = phasor_value(k0, kX[first + x0 + i / Q], kY[first + i % Q], gg.dz);
    __syncthreads();
    for (int i = tid; i < nx * BS; i += 256) {
      const int r = i / BS, b = i % BS;
      double2 t = make_double2(0.0, 0.0);
      for (int q = 0; q < Q; ++q) {
        const double w = A[q * H + b0 + b];
        const double2 d = D[r * Q + q];
        t.x = fma(d.x, w, t.x);
        t.y = fma(d.y, w, t.y);
      }
      T[i] = t;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < E; ++i) {
      const int e = tid + 256 * i;
      if (e < H * BS) {
        const int a = e / BS, b = e % BS;
        for (int r = 0; r < nx; ++r) {
          const double w = A[(x0 + r) * H + a];
          const double2 t = T[r * BS + b];
          s[i].x = fma(t.x, w, s[i].x);
          s[i].y = fma(t.y, w, s[i].y);
        }
      }
    }
  }
  C* o = out + ((size_t)blockIdx.y * stride + blockIdx.x) * (size_t)(H * H);
#pragma unroll
  for (int i = 0; i < E; ++i) {
    const int e = tid + 256 * i;
    const int x = e / BS, y = b0 + e % BS;
    if (e < H * BS) o[x * H + folded_at(2 * H, y)] = from_d<C>(s[i]);
  }
}

// The same in two launches for fewer tables than SMs (a call of one or few
// frequencies): a CTA takes kSplitRows rows of D to T in global memory, then a
// thread an entry of S, its sums in the order that k_compact_table has them.
// One SM's FP64 pipe took 0.75 ms for a table of 256 points to length 160.
constexpr int kSplitRows = 4;
__global__ void __launch_bounds__(256) k_compact_rows(double2* T, const double* freqs, const int* regions,
                                                      const RegionGeo* geo, int Q, int first, const double* kX,
                                                      const double* kY, const double* A, int H) {
  extern __shared__ __align__(16) unsigned char sm[];
  double2* D = reinterpret_cast<double2*>(sm);   // [kSplitRows][Q]
  const RegionGeo gg = geo[regions[blockIdx.x]];
  const double2 k0 = k0_of(SPEED_OF_LIGHT / freqs[blockIdx.y], gg.eps_re, gg.eps_im);
  const int x0 = blockIdx.z * kSplitRows, nx = min(kSplitRows, Q - x0);
  for (int i = threadIdx.x; i < nx * Q; i += blockDim.x)
    D[i] = phasor_value(k0, kX[first + x0 + i / Q], kY[first + i % Q], gg.dz);
  __syncthreads();
  double2* t0 = T + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * (size_t)(Q * H) + (size_t)x0 * H;
  for (int i = threadIdx.x; i < nx * H; i += blockDim.x) {
    const int r = i / H, b = i % H;
    double2 t = make_double2(0.0, 0.0);
    for (int q = 0; q < Q; ++q) {
      const double w = A[q * H + b];
      const double2 d = D[r * Q + q];
      t.x = fma(d.x, w, t.x);
      t.y = fma(d.y, w, t.y);
    }
    t0[i] = t;
  }
}
template <typename C>
__global__ void __launch_bounds__(128) k_compact_sums(C* out, const double2* T, int stride, const double* A, int Q, int H) {
  const int e = blockIdx.z * blockDim.x + threadIdx.x;
  if (e >= H * H) return;
  const int a = e / H, b = e % H;
  const double2* t0 = T + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * (size_t)(Q * H) + b;
  double2 s = make_double2(0.0, 0.0);
#pragma unroll 8
  for (int r = 0; r < Q; ++r) {
    const double w = A[r * H + a];
    const double2 t = t0[(size_t)r * H];
    s.x = fma(t.x, w, s.x);
    s.y = fma(t.y, w, s.y);
  }
  out[((size_t)blockIdx.y * stride + blockIdx.x) * (size_t)(H * H) + a * H + folded_at(2 * H, b)] = from_d<C>(s);
}

// Smallest transform length of the kernels that is at least 2 box - 1.  Both the
// input and the needed output of a propagation lie in the box, so only the
// offsets |d| < box of the propagator's N x N convolution kernel are ever used:
// a circular convolution with that kernel truncated to them, of any length >=
// 2 box - 1, gives the same field (in FP64 to 2e-14 after 100 bounces).  In
// complex64 the field is closer to it than by the grid's own transform: 3.7e-6
// against 1.2e-5 after 100 bounces of 10 disks at 128^2 (length 80), since
// fewer rounded roots act on a mode in each bounce; the spectrum's entries are
// rounded to nearest (keeping more of their bits changes nothing).
int compact_length(int box, bool fp64) {
  // complex128 takes neither 160 (40 points a thread) nor 40 (20 points for 2
  // threads a line: the one-frequency dancer at 64^2, whose few lines leave an
  // FP64 instruction's 16 cycles a warp exposed, took 12.0 ms against 7.5 ms at
  // length 64 with 8 points a thread)
  for (int M : {8, 16, 32, 40, 64, 80, 128, 160, 256})
    if (M >= 2 * box - 1 && !(fp64 && (M == 40 || M == 160))) return M;
  return 0;
}

// A[q][a] (q over the non-negative wavenumbers of the n-point grid: q + 1/2 for
// even n, q for odd n, in units of 2 pi / (n dx); a < M/2: the wavenumber
// (a + 1/2) of the M-point transform): weight (2, or 1 at wavenumber 0) / (n M)
// times sum_{|d| < box} cos(2 pi q' d / n) cos(2 pi a' d / M).  On the device,
// since a plan of a call of its own emission, or of a one-shot call, makes it
// anew: on the host it took 0.15 ms at 128 and 1.2 ms at 256 points.
__global__ void k_compact_matrix(double* A, int n, int M, int box) {
  const int Q = (n + 1) / 2, H = M / 2, i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= Q * H) return;
  const int q = i / H, a = i % H;
  const bool even = n % 2 == 0;
  // sum_{|d| < box} cos(theta d), theta / 2 = pi num / (2 n M)
  auto dirichlet = [&](long long num) {
    const double den = 2.0 * n * M;
    if (num % (2LL * n * M) == 0) return 2.0 * box - 1.0;
    return sinpi((double)((num * (2LL * box - 1)) % (4LL * n * M)) / den) / sinpi((double)num / den);
  };
  // theta / 2 = pi (q'/n -+ a'/M), 2 q' and 2 a' whole
  const long long x = (long long)(even ? 2 * q + 1 : 2 * q) * M, y = (long long)(2 * a + 1) * n;
  A[i] = (!even && q == 0 ? 1.0 : 2.0) / ((double)n * M) * (0.5 * (dirichlet(x - y) + dirichlet(x + y)));
}
size_t compact_matrix_size(int n, int M) { return (size_t)((n + 1) / 2) * (M / 2); }
int launch_compact_matrix(double* A, int n, int M, int box, cudaStream_t st) {
  COUNT_LAUNCH();
  k_compact_matrix<<<(unsigned)((compact_matrix_size(n, M) + 127) / 128), 128, 0, st>>>(A, n, M, box);
  return (int)cudaGetLastError();
}

// Columns of S that a CTA of k_compact_table takes.
static int compact_slice(int H) { return H <= 40 ? H : H == 80 ? 40 : 32; }

// Bytes of launch_compact_table's scratch, 0 where the tables fill the SMs and
// are bound by the FP64 pipe either way.  Tables of 128 points to length 80, whole
// solves of one bounce: 3 tables 371 us in two launches, 554 in one; 96 tables
// 461 and 545.
size_t compact_tmp_bytes(int n, int M, int ntab, int nfreq) {
  const int Q = (n + 1) / 2, H = M / 2;
  if ((long long)ntab * nfreq * (H / compact_slice(H)) >= sm_count()) return 0;
  return sizeof(double2) * (size_t)ntab * nfreq * Q * H;
}

int launch_compact_table(bool fp64, void* out, int nfreq, const double* d_freqs, int ntab, int stride,
                         const int* d_regions, const RegionGeo* d_geo, int n, const double* d_kX, const double* d_kY,
                         const double* d_A, int M, double2* tmp, cudaStream_t st) {
  if (ntab <= 0 || nfreq <= 0) return 0;
  const int Q = (n + 1) / 2, H = M / 2, first = n / 2;
  if (tmp) {
    COUNT_LAUNCH();
    k_compact_rows<<<dim3(ntab, nfreq, (Q + kSplitRows - 1) / kSplitRows), 256, sizeof(double2) * kSplitRows * Q, st>>>(
        tmp, d_freqs, d_regions, d_geo, Q, first, d_kX, d_kY, d_A, H);
    COUNT_LAUNCH();
    const dim3 grid(ntab, nfreq, (H * H + 127) / 128);
    if (fp64) k_compact_sums<double2><<<grid, 128, 0, st>>>((double2*)out, tmp, stride, d_A, Q, H);
    else k_compact_sums<float2><<<grid, 128, 0, st>>>((float2*)out, tmp, stride, d_A, Q, H);
    return (int)cudaGetLastError();
  }
  const int BS = compact_slice(H);
  const size_t smem = sizeof(double2) * kChunk * (Q + BS);
  dim3 grid(ntab, nfreq, H / BS);
  auto go = [&](auto* o, auto e) {
    using C = std::remove_pointer_t<decltype(o)>;
    constexpr int E = decltype(e)::value;
    const cudaError_t rc = cudaFuncSetAttribute(k_compact_table<C, E>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
    if (rc != cudaSuccess) return (int)rc;
    COUNT_LAUNCH();
    k_compact_table<C, E><<<grid, 256, smem, st>>>(o, d_freqs, stride, d_regions, d_geo, Q, first, d_kX, d_kY, d_A, H, BS);
    return (int)cudaGetLastError();
  };
  using std::integral_constant;
  const int per = H * BS;
  if (smem > kMaxSmem) return (int)cudaErrorInvalidValue;
  if (fp64) {
    double2* o = (double2*)out;
    return per <= 512 ? go(o, integral_constant<int, 2>()) : per <= 2048 ? go(o, integral_constant<int, 8>())
                                                                       : go(o, integral_constant<int, 16>());
  }
  float2* o = (float2*)out;
  return per <= 512 ? go(o, integral_constant<int, 2>()) : per <= 2048 ? go(o, integral_constant<int, 8>())
                                                                     : go(o, integral_constant<int, 16>());
}

template <typename C>
__global__ void k_tilt_table(C* out, int nfreq, const double* freqs, int nmaps, const int* regions,
                             const RegionGeo* geo, int nbx, int nby, int bx0, int by0, int nx, int ny,
                             const double* X, const double* Y, const double2* surf) {
  const int per = nbx * nby;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  const int m = blockIdx.y, f = blockIdx.z;
  if (idx >= per) return;
  const int iy = idx / nbx, ix = idx % nbx;
  const int x = bx0 + ix, y = by0 + iy;
  const int reg = regions[m];
  const RegionGeo gg = geo[reg];
  const double lambda = SPEED_OF_LIGHT / freqs[f];
  const double2 k0 = k0_of(lambda, gg.eps_re, gg.eps_im);
  double2 v = cmul(phase_k0(k0, gg.tilt_x * X[x]), phase_k0(k0, gg.tilt_y * Y[y]));
  if (surf) v = cmul(v, phase_k0c(k0, surf[((size_t)reg * ny + y) * nx + x]));
  out[((size_t)f * nmaps + m) * per + idx] = from_d_phase<C>(v);
}

int launch_tilt_table(bool fp64, void* out, int nfreq, const double* d_freqs, int nmaps,
                      const int* d_regions, const RegionGeo* d_geo, int nbx, int nby, int bx0,
                      int by0, int nx, int ny, const double* d_X, const double* d_Y,
                      const double2* d_surf, cudaStream_t st) {
  if (nmaps <= 0 || nfreq <= 0) return 0;
  dim3 grid((nbx * nby + 255) / 256, nmaps, nfreq);
  if (fp64) { COUNT_LAUNCH(); k_tilt_table<double2><<<grid, 256, 0, st>>>((double2*)out, nfreq, d_freqs, nmaps, d_regions, d_geo, nbx, nby, bx0, by0, nx, ny, d_X, d_Y, d_surf); }
  else { COUNT_LAUNCH(); k_tilt_table<float2><<<grid, 256, 0, st>>>((float2*)out, nfreq, d_freqs, nmaps, d_regions, d_geo, nbx, nby, bx0, by0, nx, ny, d_X, d_Y, d_surf); }
  return (int)cudaGetLastError();
}

// A line of any other length, as a sum over its pairs: with e_j, o_j = x_j +- x_(n-j),
// X_k, X_(n-k) = x_0 (+ (-1)^k x_(n/2)) + sum_j e_j cos(2 pi jk / n) -+ i sum_j o_j sin(2 pi jk / n),
// a quarter of the products of the plain sum and a sine for every second root; a
// line of zeros (a row off the disk) stays.  Bound by the FP64 pipe and its
// latency: 101 lines of 101 took 26 us plain, 16 us here; 28 x 51 lines of
// 51 64 us plain, 19 us here.
template <typename C>
__device__ __forceinline__ void folded_line_dft(C* line, int n, size_t stride, int inverse, double2* sm) {
  const int H = (n - 1) / 2, half = n / 2;
  // E[0 .. half], O[1 .. H], tw[m] = (cos, sin)(2 pi m / n) for m <= half: 24 n + 16 bytes at most
  double2 *E = sm, *O = sm + half, *tw = O + H + 1;
  bool some = false;
  for (int j = threadIdx.x; j <= half; j += blockDim.x) {
    const double2 x = to_d(line[j * stride]);
    double2 y = make_double2(0.0, 0.0);
    if (j > 0 && j <= H) y = to_d(line[(n - j) * stride]);
    E[j] = cadd(x, y);
    if (j > 0 && j <= H) O[j] = csub(x, y);
    some = some || x.x != 0.0 || x.y != 0.0 || y.x != 0.0 || y.y != 0.0;
  }
  if (!__syncthreads_or(some)) return;
  for (int m = threadIdx.x; m <= half; m += blockDim.x) sincospi(2.0 * m / n, &tw[m].y, &tw[m].x);
  __syncthreads();
  for (int k = threadIdx.x; k <= half; k += blockDim.x) {
    double2 a = E[0], b = make_double2(0.0, 0.0);
    if (half > H) a = (k & 1) ? csub(a, E[half]) : cadd(a, E[half]);
    int m = 0;
    for (int j = 1; j <= H; ++j) {
      m += k;
      if (m >= n) m -= n;
      double2 w = tw[m <= half ? m : n - m];
      if (m > half) w.y = -w.y;
      const double2 e = E[j], o = O[j];
      a.x = fma(e.x, w.x, a.x);
      a.y = fma(e.y, w.x, a.y);
      b.x = fma(o.x, w.y, b.x);
      b.y = fma(o.y, w.y, b.y);
    }
    // X_k = a - i b (forward), X_(n-k) = a + i b; the inverse's the other way round
    const double2 lo = make_double2(a.x + b.y, a.y - b.x), hi = make_double2(a.x - b.y, a.y + b.x);
    line[k * stride] = from_d<C>(inverse ? hi : lo);
    if (k > 0 && k <= H) line[(n - k) * stride] = from_d<C>(inverse ? lo : hi);
  }
}

// ---------------------------------------------------------------------------
// General full-grid path
// ---------------------------------------------------------------------------
// One block transforms one line of length n held in shared memory: radix-2
// Stockham for powers of two, folded O(n^2) evaluation otherwise.  Roots are
// evaluated in FP64 (sincospi) for either field precision.
template <typename C>
__global__ void k_line_dft(C* data, int nx, int ny, int axis, int inverse) {
  extern __shared__ __align__(16) unsigned char sm[];
  const int n = axis == 0 ? nx : ny;
  C* buf0 = reinterpret_cast<C*>(sm);
  C* buf1 = buf0 + n;
  C* tw = buf1 + n;   // tw[m] = exp(-+2 pi i m / n)
  const int line = blockIdx.x, b = blockIdx.y;
  const size_t base = (size_t)b * nx * ny;
  const size_t stride = axis == 0 ? 1 : nx;
  const size_t off = axis == 0 ? (size_t)line * nx : (size_t)line;
  if ((n & (n - 1)) != 0) {
    folded_line_dft(data + base + off, n, stride, inverse, reinterpret_cast<double2*>(sm));
    return;
  }
  const double sgn = inverse ? 2.0 : -2.0;
  // power-of-two lengths up to 1024 take the unit roots from the constant
  // table (FP64, exactly symmetric) instead of one FP64 sincospi per entry
  const bool table = (n & (n - 1)) == 0 && n <= 1024;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    buf0[i] = data[base + off + i * stride];
    if (table) {
      const double2 r = c_root1024_d[i * (1024 / n)];   // exp(-2 pi i k / n)
      tw[i] = from_d<C>(make_double2(r.x, inverse ? -r.y : r.y));
    } else {
      double s, c;
      sincospi(sgn * (double)i / (double)n, &s, &c);
      tw[i] = from_d<C>(make_double2(c, s));
    }
  }
  __syncthreads();
  // Stockham autosort, radix 2
  C* src = buf0;
  C* dst = buf1;
  for (int l = 1; l < n; l <<= 1) {   // l = size of the sub-transforms being combined
    const int tstep = n / (2 * l);
    for (int i = threadIdx.x; i < n / 2; i += blockDim.x) {
      const int j = i % l;            // position within sub-transform
      const int k = i / l;            // sub-transform index
      const C w = tw[j * tstep];
      C u = src[k * l + j];
      C v = cmul(src[k * l + j + n / 2], w);
      dst[2 * k * l + j] = cadd(u, v);
      dst[2 * k * l + j + l] = csub(u, v);
    }
    __syncthreads();
    C* t = src; src = dst; dst = t;
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) data[base + off + i * stride] = src[i];
}

int launch_line_dft(bool fp64, void* data, int nb, int nx, int ny, int axis, int inverse,
                    cudaStream_t st) {
  const int n = axis == 0 ? nx : ny;
  const int nlines = axis == 0 ? ny : nx;
  if (n <= 1) return 0;
  size_t smem = (fp64 ? 16 : 8) * (size_t)(3 * n);
  if (smem > kMaxSmem) return (int)cudaErrorInvalidValue;
  dim3 grid(nlines, nb);
  int thr = n >= 256 ? 256 : ((n + 31) / 32) * 32;
  if ((n & (n - 1)) != 0) {   // folded: a thread takes a pair of outputs
    thr = std::min(256, (n / 2 + 32) / 32 * 32);
    smem = 24 * (size_t)n + (n % 2 ? 8 : 16);
  }
  if (fp64) {
    if (smem > 48 * 1024) cudaFuncSetAttribute(k_line_dft<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
      COUNT_LAUNCH();
      k_line_dft<double2><<<grid, thr, smem, st>>>((double2*)data, nx, ny, axis, inverse);
  } else {
    if (smem > 48 * 1024) cudaFuncSetAttribute(k_line_dft<float2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
      COUNT_LAUNCH();
      k_line_dft<float2><<<grid, thr, smem, st>>>((float2*)data, nx, ny, axis, inverse);
  }
  return (int)cudaGetLastError();
}

template <typename C>
__global__ void k_mul_mask(C* data, size_t total, int npix, const unsigned char* mask) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x)
    if (!mask[i % npix]) data[i] = czero<C>();
}

static dim3 grid1d(size_t n) {
  size_t b = (n + 255) / 256;
  if (b > 65535 * 16) b = 65535 * 16;
  if (b < 1) b = 1;
  return dim3((unsigned)b);
}

int launch_mul_mask(bool fp64, void* data, int nb, int nx, int ny, const unsigned char* d_mask,
                    cudaStream_t st) {
  size_t total = (size_t)nb * nx * ny;
  if (fp64) { COUNT_LAUNCH(); k_mul_mask<double2><<<grid1d(total), 256, 0, st>>>((double2*)data, total, nx * ny, d_mask); }
  else { COUNT_LAUNCH(); k_mul_mask<float2><<<grid1d(total), 256, 0, st>>>((float2*)data, total, nx * ny, d_mask); }
  return (int)cudaGetLastError();
}

__device__ __forceinline__ double lambda_of(const double* freqs, const double* lambdas, int b) {
  return lambdas ? lambdas[b] : SPEED_OF_LIGHT / freqs[b];
}

template <typename C>
__global__ void k_mul_phasor_full(C* data, int nb, int nx, int ny, const double* freqs,
                                  const double* lambdas, RegionGeo g, const double* kX,
                                  const double* kY, int shifted, double scale) {
  const size_t total = (size_t)nb * nx * ny;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % nx);
    const int y = (int)((i / nx) % ny);
    const int b = (int)(i / ((size_t)nx * ny));
    const int sx = shifted ? x : (x + nx / 2) % nx;
    const int sy = shifted ? y : (y + ny / 2) % ny;
    const double2 k0 = k0_of(lambda_of(freqs, lambdas, b), g.eps_re, g.eps_im);
    double2 p = phasor_value(k0, kX[sx], kY[sy], g.dz);
    p.x *= scale; p.y *= scale;
    double2 d = to_d(data[i]);
    data[i] = from_d<C>(cmul(d, p));
  }
}

int launch_mul_phasor_full(bool fp64, void* data, int nb, int nx, int ny, const double* d_freqs,
                           const double* d_lambda, RegionGeo g, const double* d_kX,
                           const double* d_kY, int shifted_layout, double scale, cudaStream_t st) {
  size_t total = (size_t)nb * nx * ny;
  if (fp64) { COUNT_LAUNCH(); k_mul_phasor_full<double2><<<grid1d(total), 256, 0, st>>>((double2*)data, nb, nx, ny, d_freqs, d_lambda, g, d_kX, d_kY, shifted_layout, scale); }
  else { COUNT_LAUNCH(); k_mul_phasor_full<float2><<<grid1d(total), 256, 0, st>>>((float2*)data, nb, nx, ny, d_freqs, d_lambda, g, d_kX, d_kY, shifted_layout, scale); }
  return (int)cudaGetLastError();
}

template <typename C>
__global__ void k_mul_tilt_full(C* data, int nb, int nx, int ny, const double* freqs,
                                const double* lambdas, RegionGeo g, const double* X, const double* Y,
                                const double2* surf, int only_if_nonzero) {
  const size_t total = (size_t)nb * nx * ny;
  const bool do_tilt = !only_if_nonzero || g.tilt_x != 0.0 || g.tilt_y != 0.0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % nx);
    const int y = (int)((i / nx) % ny);
    const int b = (int)(i / ((size_t)nx * ny));
    const double2 k0 = k0_of(lambda_of(freqs, lambdas, b), g.eps_re, g.eps_im);
    double2 d = to_d(data[i]);
    if (do_tilt) d = cmul(d, cmul(phase_k0(k0, g.tilt_x * X[x]), phase_k0(k0, g.tilt_y * Y[y])));
    if (surf) d = cmul(d, phase_k0c(k0, surf[(size_t)y * nx + x]));
    data[i] = from_d<C>(d);
  }
}

int launch_mul_tilt_full(bool fp64, void* data, int nb, int nx, int ny, const double* d_freqs,
                         const double* d_lambda, RegionGeo g, const double* d_X, const double* d_Y,
                         const double2* d_surf, int only_if_nonzero, cudaStream_t st) {
  size_t total = (size_t)nb * nx * ny;
  if (fp64) { COUNT_LAUNCH(); k_mul_tilt_full<double2><<<grid1d(total), 256, 0, st>>>((double2*)data, nb, nx, ny, d_freqs, d_lambda, g, d_X, d_Y, d_surf, only_if_nonzero); }
  else { COUNT_LAUNCH(); k_mul_tilt_full<float2><<<grid1d(total), 256, 0, st>>>((float2*)data, nb, nx, ny, d_freqs, d_lambda, g, d_X, d_Y, d_surf, only_if_nonzero); }
  return (int)cudaGetLastError();
}

template <typename C>
__global__ void k_mul_phase1d(C* data, int nb, int npix, const double* freqs, const double* lambdas,
                              RegionGeo g) {
  const size_t total = (size_t)nb * npix;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int b = (int)(i / npix);
    const double2 k0 = k0_of(lambda_of(freqs, lambdas, b), g.eps_re, g.eps_im);
    data[i] = from_d<C>(cmul(to_d(data[i]), phase_k0(k0, g.dz)));
  }
}

int launch_mul_scalar_phase_1d(bool fp64, void* data, int nb, int nx, int ny, const double* d_freqs,
                               const double* d_lambda, RegionGeo g, cudaStream_t st) {
  size_t total = (size_t)nb * nx * ny;
  if (fp64) { COUNT_LAUNCH(); k_mul_phase1d<double2><<<grid1d(total), 256, 0, st>>>((double2*)data, nb, nx * ny, d_freqs, d_lambda, g); }
  else { COUNT_LAUNCH(); k_mul_phase1d<float2><<<grid1d(total), 256, 0, st>>>((float2*)data, nb, nx * ny, d_freqs, d_lambda, g); }
  return (int)cudaGetLastError();
}

template <typename C>
__global__ void k_roll(const C* in, C* out, int nb, int nx, int ny, int sx, int sy) {
  const size_t total = (size_t)nb * nx * ny;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % nx);
    const int y = (int)((i / nx) % ny);
    const size_t b = i / ((size_t)nx * ny);
    const int xs = ((x - sx) % nx + nx) % nx;
    const int ys = ((y - sy) % ny + ny) % ny;
    out[i] = in[(b * ny + ys) * nx + xs];
  }
}

int launch_roll(bool fp64, const void* in, void* out, int nb, int nx, int ny, int sx, int sy,
                cudaStream_t st) {
  size_t total = (size_t)nb * nx * ny;
  if (fp64) { COUNT_LAUNCH(); k_roll<double2><<<grid1d(total), 256, 0, st>>>((const double2*)in, (double2*)out, nb, nx, ny, sx, sy); }
  else { COUNT_LAUNCH(); k_roll<float2><<<grid1d(total), 256, 0, st>>>((const float2*)in, (float2*)out, nb, nx, ny, sx, sy); }
  return (int)cudaGetLastError();
}

template <typename CI, typename CO>
__global__ void k_convert(const CI* in, CO* out, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    out[i] = from_d<CO>(to_d(in[i]));
}

int launch_convert(const void* in, bool in_fp64, void* out, bool out_fp64, size_t n, cudaStream_t st) {
  if (in_fp64 && out_fp64) { COUNT_LAUNCH(); k_convert<double2, double2><<<grid1d(n), 256, 0, st>>>((const double2*)in, (double2*)out, n); }
  else if (in_fp64) { COUNT_LAUNCH(); k_convert<double2, float2><<<grid1d(n), 256, 0, st>>>((const double2*)in, (float2*)out, n); }
  else if (out_fp64) { COUNT_LAUNCH(); k_convert<float2, double2><<<grid1d(n), 256, 0, st>>>((const float2*)in, (double2*)out, n); }
  else { COUNT_LAUNCH(); k_convert<float2, float2><<<grid1d(n), 256, 0, st>>>((const float2*)in, (float2*)out, n); }
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------
// exits, broadcast, reductions
// ---------------------------------------------------------------------------
__global__ void k_exit_combine(double2* out, const double2* full, const double2* direct, double2 coef,
                               int nfreq, int npix) {
  const size_t total = (size_t)nfreq * npix;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    double2 v = cmul(coef, full[i]);
    if (direct) {
      double2 d = direct[i % npix];
      v = make_double2(v.x + d.x, v.y + d.y);
    }
    out[i] = v;
  }
}

int launch_exit_combine(double2* out, const double2* full, const double2* direct, double2 coef,
                        int nfreq, int npix, cudaStream_t st) {
  size_t total = (size_t)nfreq * npix;
  COUNT_LAUNCH();
  k_exit_combine<<<grid1d(total), 256, 0, st>>>(out, full, direct, coef, nfreq, npix);
  return (int)cudaGetLastError();
}

// boxes of nbx x nby pixels, `total` in all, times exp(i alpha (x + y)): what k_embed_box takes out again
__global__ void k_modulate(double2* boxes, size_t total, int nbx, int plane, double alpha) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int p = (int)(i % plane);
    boxes[i] = cmul(boxes[i], dcexp(0.0, alpha * (p / nbx + p % nbx)));
  }
}

int launch_modulate(double2* boxes, size_t total, int nbx, int nby, double alpha, cudaStream_t st) {
  if (!total) return 0;
  COUNT_LAUNCH();
  k_modulate<<<grid1d(total), 256, 0, st>>>(boxes, total, nbx, nbx * nby, alpha);
  return (int)cudaGetLastError();
}

__global__ void k_embed_box(double2* full, const double2* box, int nfreq, int nx, int ny, int nbx,
                            int nby, int bx0, int by0, double alpha) {
  const size_t total = (size_t)nfreq * nx * ny;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % nx);
    const int y = (int)((i / nx) % ny);
    const size_t f = i / ((size_t)nx * ny);
    const int ix = x - bx0, iy = y - by0;
    double2 v = make_double2(0.0, 0.0);
    if (ix >= 0 && ix < nbx && iy >= 0 && iy < nby) {
      v = box[(f * nby + iy) * nbx + ix];
      if (alpha != 0.0) v = cmul(v, dcexp(0.0, -alpha * (ix + iy)));   // the stages' fields carry exp(i alpha (x + y))
    }
    full[i] = v;
  }
}

int launch_embed_box(double2* full, const double2* box, int nfreq, int nx, int ny, int nbx, int nby,
                     int bx0, int by0, double alpha, cudaStream_t st) {
  size_t total = (size_t)nfreq * nx * ny;
  COUNT_LAUNCH();
  k_embed_box<<<grid1d(total), 256, 0, st>>>(full, box, nfreq, nx, ny, nbx, nby, bx0, by0, alpha);
  return (int)cudaGetLastError();
}

template <typename C>
__global__ void k_broadcast(C* state, const double2* init, int nfreq, size_t per) {
  const size_t total = (size_t)nfreq * per;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x)
    state[i] = from_d<C>(init[i % per]);
}

int launch_broadcast_state(bool fp64, void* state, const double2* init, int nfreq, size_t per,
                           cudaStream_t st) {
  size_t total = (size_t)nfreq * per;
  if (fp64) { COUNT_LAUNCH(); k_broadcast<double2><<<grid1d(total), 256, 0, st>>>((double2*)state, init, nfreq, per); }
  else { COUNT_LAUNCH(); k_broadcast<float2><<<grid1d(total), 256, 0, st>>>((float2*)state, init, nfreq, per); }
  return (int)cudaGetLastError();
}

__global__ void k_beta2(double* beta2, const double2* E, int npix, double scale) {
  __shared__ double red[256];
  const int f = blockIdx.x;
  double s = 0.0;
  for (int i = threadIdx.x; i < npix; i += blockDim.x) {
    double2 v = E[(size_t)f * npix + i];
    s += v.x * v.x + v.y * v.y;
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) beta2[f] = red[0] * scale;
}

int launch_beta2(double* beta2, const double2* E, int nfreq, int npix, double scale, cudaStream_t st) {
  if (nfreq <= 0) return 0;
  COUNT_LAUNCH();
  k_beta2<<<nfreq, 256, 0, st>>>(beta2, E, npix, scale);
  return (int)cudaGetLastError();
}

template <typename C>
__global__ void k_maxabs(unsigned long long* out, const C* data, size_t n) {
  __shared__ double red[256];
  double m = 0.0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    double2 v = to_d(data[i]);
    m = fmax(m, hypot(v.x, v.y));
  }
  red[threadIdx.x] = m;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + w]);
    __syncthreads();
  }
  // non-negative doubles order like their bit patterns
  if (threadIdx.x == 0) atomicMax(out, (unsigned long long)__double_as_longlong(red[0]));
}

int launch_maxabs(double* d_out, const void* data, bool fp64, size_t n, cudaStream_t st) {
  cudaMemsetAsync(d_out, 0, sizeof(double), st);
  unsigned blocks = (unsigned)((n + 255) / 256);
  if (blocks > 1024) blocks = 1024;
  if (blocks < 1) blocks = 1;
  if (fp64) { COUNT_LAUNCH(); k_maxabs<double2><<<blocks, 256, 0, st>>>((unsigned long long*)d_out, (const double2*)data, n); }
  else { COUNT_LAUNCH(); k_maxabs<float2><<<blocks, 256, 0, st>>>((unsigned long long*)d_out, (const float2*)data, n); }
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------
// 1D propagator solvers: the field at every pixel bounces independently
// (prop = propagator1D multiplies by exp(-i k0 dz) and applies no mask).
// FP64 for both precisions.
// ---------------------------------------------------------------------------
__global__ void k_rfp1d(Rfp1dArgs a) {
  const size_t total = (size_t)a.nfreq * a.npix;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
    const int f = (int)(t / a.npix);
    const int p = (int)(t % a.npix);
    const int nd = a.nd;
    const double2* ph = a.phase + (size_t)f * nd;
    double2* S = (double2*)a.state;
    if (a.kind == 0) {
      // cheerleader (src/boost_fractor_recurprop.jl:226-363); exits in out[f][0]=right, [1]=left
      auto s_at = [&](int j) -> double2& { return S[((size_t)f * nd + j) * a.npix + p]; };
      double2* outR = a.out + ((size_t)f * 2 + 0) * a.npix + p;
      double2* outL = a.out + ((size_t)f * 2 + 1) * a.npix + p;
      auto em = [&](int j, int d) { return a.emit[((size_t)j * 2 + d) * a.npix + p]; };
      auto cf = [&](int i, int k) { return a.coef[4 * i + k]; };  // r_r, t_l, r_l, t_r
      if (a.do_init) {
        for (int j = 0; j < nd; ++j) s_at(j) = em(j, 0);
        for (int i = 1; i <= nd - 2; ++i) {
          s_at(i) = cmul(s_at(i), ph[i]);
          s_at(i + 1) = cadd(s_at(i + 1), cmul(cf(i, 3), s_at(i)));
          s_at(i) = cmul(s_at(i), cf(i, 0));
        }
        for (int j = 0; j <= nd - 2; ++j) s_at(j) = cadd(s_at(j), em(j, 1));
        s_at(nd - 2) = cadd(s_at(nd - 2), cmul(cf(nd - 2, 1), em(nd - 1, 1)));
        s_at(nd - 1) = cadd(s_at(nd - 1), cmul(cf(nd - 2, 2), em(nd - 1, 1)));
        *outR = s_at(nd - 1);
        *outL = s_at(0);
        // the exit regions live in out[] from here on
        s_at(nd - 1) = make_double2(0.0, 0.0);
        s_at(0) = make_double2(0.0, 0.0);
      }
      double2 eR = *outR, eL = *outL;
      for (int n = a.n_begin; n < a.n_end; ++n) {
        double2 f1 = cmul(s_at(1), ph[1]);
        eL = cadd(eL, cmul(cf(0, 1), f1));
        s_at(1) = cmul(f1, cf(0, 2));
        for (int i = 1; i <= nd - 3; ++i) {
          double2 fi = cmul(s_at(i), ph[i]);
          double2 fn = cmul(s_at(i + 1), ph[i + 1]);
          s_at(i + 1) = cadd(cmul(cf(i, 2), fn), cmul(cf(i, 3), fi));
          s_at(i) = cadd(cmul(cf(i, 0), fi), cmul(cf(i, 1), fn));
        }
        const int i = nd - 2;
        double2 fi = cmul(s_at(i), ph[i]);
        eR = cadd(eR, cmul(cf(i, 3), fi));
        s_at(i) = cmul(fi, cf(i, 0));
      }
      *outR = eR;
      *outL = eL;
    } else {
      // dancer (src/boost_fractor_recurprop.jl:25-146): nd trimmed regions,
      // boundaries 0..nd with r[nd] = 0 appended; coef[i].x = r[i]
      auto s_at = [&](int j, int d) -> double2& { return S[(((size_t)f * nd + j) * 2 + d) * a.npix + p]; };
      for (int n = a.n_begin; n < a.n_end; ++n) {
        const int rm = (n + a.rm_phase) & 1, lm = rm ^ 1;
        for (int i = 0; i <= nd; ++i) {
          if (i > 0) s_at(i - 1, rm) = cmul(s_at(i - 1, rm), ph[i - 1]);
          if (i < nd) s_at(i, lm) = cmul(s_at(i, lm), ph[i]);
          const double2 r = a.coef[4 * i];
          const double2 one_p = make_double2(1.0 + r.x, r.y), one_m = make_double2(1.0 - r.x, -r.y);
          const double2 mr = make_double2(-r.x, -r.y);
          if (i == 0) {
            s_at(0, lm) = cmul(s_at(0, lm), mr);
          } else if (i == nd) {
            double2 e = cmul(one_p, s_at(nd - 1, rm));
            double2* o = a.out + ((size_t)f * a.nout + (a.per_iter_out ? n : 0)) * a.npix + p;
            if (a.per_iter_out) *o = e;
            else *o = cadd(*o, e);
            s_at(nd - 1, rm) = cmul(s_at(nd - 1, rm), r);
          } else {
            double2 c = s_at(i - 1, rm);
            s_at(i - 1, rm) = cadd(cmul(r, c), cmul(one_m, s_at(i, lm)));
            s_at(i, lm) = cadd(cmul(mr, s_at(i, lm)), cmul(one_p, c));
          }
        }
      }
    }
  }
}

int launch_rfp1d(bool fp64, const Rfp1dArgs& a, cudaStream_t st) {
  (void)fp64;
  size_t total = (size_t)a.nfreq * a.npix;
  unsigned blocks = (unsigned)((total + 127) / 128);
  if (blocks < 1) blocks = 1;
  COUNT_LAUNCH();
  k_rfp1d<<<blocks, 128, 0, st>>>(a);
  return (int)cudaGetLastError();
}

}  // namespace bf
