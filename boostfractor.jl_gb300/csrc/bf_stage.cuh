// The fused stage kernels of the bounce loop and their launches, templated on
// the transform length; instantiated by bf_device.cu (powers of two) and
// bf_five_f.cu / bf_five_d.cu (lengths 40, 80 and 160), which compile in
// parallel.
#pragma once

#include <math.h>

#include <algorithm>
#include <vector>

#include "bf_common.cuh"
#include "bf_device.cuh"
#include "bf_fft.cuh"

namespace bf {

// Round an FP64 complex value to complex64 so that the modulus error is as
// small as possible: of the float pairs within one ulp of (re, im) take the one
// whose squared modulus is closest to the FP64 one.  Plain rounding leaves a
// random modulus error of ~6e-8 per value, and a phasor or twiddle that is
// applied to the same k-bin on every bounce turns that into a systematic gain
// or loss that compounds over hundreds of bounces.
__host__ __device__ inline float2 round_c64_host_device(double re, double im) {
  const float fr = (float)re, fi = (float)im;
  const double m2 = re * re + im * im;
  float best_r = fr, best_i = fi;
  double best = 1e300;
  for (int a = -1; a <= 1; ++a)
    for (int b = -1; b <= 1; ++b) {
      float cr = a == 0 ? fr : nextafterf(fr, a > 0 ? INFINITY : -INFINITY);
      float ci = b == 0 ? fi : nextafterf(fi, b > 0 ? INFINITY : -INFINITY);
      double d = fabs((double)cr * cr + (double)ci * ci - m2);
      // prefer the plain rounding on ties (keeps exact values exact)
      if (d < best || (d == best && a == 0 && b == 0)) {
        best = d;
        best_r = cr;
        best_i = ci;
      }
    }
  return make_float2(best_r, best_i);
}

template <typename C> __device__ __forceinline__ C from_d(double2 v);
template <> __device__ __forceinline__ float2 from_d<float2>(double2 v) {
  return make_float2((float)v.x, (float)v.y);
}
template <> __device__ __forceinline__ double2 from_d<double2>(double2 v) { return v; }
// phase factors: modulus-aware rounding to complex64
template <typename C> __device__ __forceinline__ C from_d_phase(double2 v);
template <> __device__ __forceinline__ float2 from_d_phase<float2>(double2 v) {
  return round_c64_host_device(v.x, v.y);
}
template <> __device__ __forceinline__ double2 from_d_phase<double2>(double2 v) { return v; }
template <typename C> __device__ __forceinline__ C czero() { return from_d<C>(make_double2(0.0, 0.0)); }

// ---------------------------------------------------------------------------
// Fused box stage kernel
// ---------------------------------------------------------------------------
constexpr int kFusedThreads = 256;
constexpr int kSmemHeader = 128;

// Row pitch of a tile, in elements.  Lengths 80 and 160: 4 mod 16, so that
// both the row pass (4 teams of a half-warp on successive rows, threads 5 or
// 10 bins apart) and the column pass (4 successive columns, threads one row
// apart) spread over the banks; 40: 9 mod 16, for the same reason at 2 threads
// a team.
__host__ __device__ constexpr int pitch_of(int N) { return N == 80 || N == 160 ? N + 4 : N == 40 ? 41 : N + 2; }
template <int N> __host__ __device__ constexpr int fused_pitch() { return pitch_of(N); }

// Elements of `tiles` row tiles, rounded up so that the teams' regions behind
// them start on 16 bytes (the destinations of cp.async).
template <int N> __host__ __device__ constexpr int tile_elements(int tiles, int nby) {
  return (tiles * nby * fused_pitch<N>() + 1) & ~1;
}

// Kernel-shape options of the fused stage (a bit mask): the inter-pass
// twiddles from a shared table instead of registers; team exchanges in two
// halves through half-size scratch; each column task's folded phasor row
// copied into the team's shared buffer (cp.async) while the team runs the
// forward transform, instead of loaded from L2 after it.  None changes the
// arithmetic.
constexpr int kModeTwShared = 1, kModeHalf = 2, kModeStage = 4;

// Complex elements of one team's shared region: its exchange scratch, then
// (kModeStage) the N/2-entry phasor row buffer.
template <int N, int MODE> __host__ __device__ constexpr int team_region() {
  return Team<N>::template scratch<(MODE & kModeHalf) != 0>() + ((MODE & kModeStage) ? N / 2 : 0);
}

__device__ __forceinline__ void cp_async16(void* dst_smem, const void* src_global) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst_smem)),
               "l"(src_global)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// Place of entry ky < N / 2 in a folded phasor row.  Lengths 40, 80 and 160: the
// entries that a team's thread multiplies its bins by lie together (thread g:
// ky = g CC + j + RR q, q < G / 2), so it loads them 16 bytes at a time; other
// lengths: in order.
__host__ __device__ inline int folded_at(int N, int ky) {
  if (N % 5) return ky;
  const int G = N == 40 ? 2 : 4, RR = N / G, CC = RR / G;
  return (ky % RR / CC) * (CC * G / 2) + ky / RR * CC + ky % CC;
}

// v (a thread's bins after the forward transform) times the folded phasor row
// Qrow: bins k and N - 1 - k share an entry.
template <int N, typename C>
__device__ __forceinline__ void mul_folded(C (&v)[Team<N>::RR], const C* Qrow, int g) {
  constexpr int G = Team<N>::G, RR = Team<N>::RR, CC = Team<N>::C;
  if constexpr (N % 5 == 0) {
    constexpr int E = CC * G / 2;   // entries of a thread; its mirrored bins use those of thread G - 1 - g, backwards
    static_assert(E % 2 == 0, "16-byte loads");
    const C* own = Qrow + g * E;
    const C* mir = Qrow + (G - 1 - g) * E;
    auto pair = [](const C* p, C& a, C& b) {
      if constexpr (sizeof(C) == 8) {
        const float4 t = *reinterpret_cast<const float4*>(p);
        a = mk(t.x, t.y);
        b = mk(t.z, t.w);
      } else {
        a = p[0];
        b = p[1];
      }
    };
#pragma unroll
    for (int e = 0; e < E; e += 2) {
      C a, b;
      pair(own + e, a, b);
      v[(e % CC) * G + e / CC] = cmul(v[(e % CC) * G + e / CC], a);
      v[((e + 1) % CC) * G + (e + 1) / CC] = cmul(v[((e + 1) % CC) * G + (e + 1) / CC], b);
      pair(mir + e, a, b);
      const int ma = (CC - 1 - e % CC) * G + G - 1 - e / CC, mb = (CC - 1 - (e + 1) % CC) * G + G - 1 - (e + 1) / CC;
      v[ma] = cmul(v[ma], a);
      v[mb] = cmul(v[mb], b);
    }
  } else {
    // ky = g*CC + j + RR*q < N/2 exactly when q < G/2
#pragma unroll
    for (int j = 0; j < CC; ++j)
#pragma unroll
      for (int q = 0; q < G; ++q) {
        const int ky = g * CC + j + RR * q;
        v[j * G + q] = cmul(v[j * G + q], Qrow[q < G / 2 ? ky : N - 1 - ky]);
      }
  }
}

template <typename C, int N>
struct FusedCtx {
  using T = Team<N>;
  static constexpr int G = T::G, RR = T::RR, CC = T::C;
  static constexpr int P = fused_pitch<N>();
};

// Add a line's points x = g + G r < nbx to its FP64 exit sums: the loads of a
// group together, before its stores (which may alias them, as far as the
// compiler knows), so that a group waits for memory once.
template <int NZ, int G, int RR, typename C>
__device__ __forceinline__ void exit_add(double2* acc, const C (&v)[RR], int g, int nbx) {
  constexpr int S = NZ < 3 ? NZ : 3;
  double2 o[S];
#pragma unroll
  for (int r0 = 0; r0 < NZ; r0 += S) {
#pragma unroll
    for (int k = 0; k < S; ++k)
      if (r0 + k < NZ && g + G * (r0 + k) < nbx) o[k] = acc[g + G * (r0 + k)];
#pragma unroll
    for (int k = 0; k < S; ++k)
      if (r0 + k < NZ && g + G * (r0 + k) < nbx) {
        const double2 d = to_d(v[r0 + k]);
        acc[g + G * (r0 + k)] = make_double2(o[k].x + d.x, o[k].y + d.y);
      }
  }
}

// Phase 1 of one propagation: forward FFT along x of every box row.  Fields
// are stored pre-masked, so only register slots r < ceil(nbx/G) can hold box
// pixels.  A slot feeding an exit adds its (masked) input to the FP64 exit
// accumulator on the way.
template <typename C, int N, int NZ, int NT, bool HALF = false>
__device__ __forceinline__ void fused_phase1(const FusedArgs<C>& a, int f, int slot, int exitk, C* M,
                                             C* scr, const C* tw, int team, int g) {
  using X = FusedCtx<C, N>;
  constexpr int G = X::G, RR = X::RR, CC = X::CC, P = X::P;
  constexpr int NTEAM = NT;
  const int nbx = a.nbx, nby = a.nby;
  const C* src = a.state + ((size_t)f * a.nslots + slot) * (size_t)(nby * nbx);
  double2* acc = exitk >= 0 ? a.exitacc + ((size_t)exitk * a.nfreq + f) * (size_t)(nby * nbx) : nullptr;
  const int rv = (nbx + G - 1) / G;
  for (int base = 0; base < nby; base += NTEAM) {
    const int y = base + team;
    const bool act = y < nby;
    if (!__any_sync(0xffffffffu, act)) continue;   // the whole warp is idle
    const C* row = src + y * nbx;
    double2* arow = acc ? acc + y * nbx : nullptr;
    C v[RR];
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      v[r] = czero<C>();
      if (r < NZ && r < rv) {
        const int x = g + G * r;
        if (act && x < nbx) v[r] = row[x];
      }
    }
    if (act && arow) exit_add<NZ, G>(arow, v, g, nbx);
    X::T::template forward<NZ, HALF>(v, tw, scr, g);
    if (act) {
#pragma unroll
      for (int j = 0; j < CC; ++j)
#pragma unroll
        for (int q = 0; q < G; ++q) M[y * P + g * CC + j + RR * q] = v[j * G + q];
    }
  }
  __syncthreads();
}

// Phase 2: per column kx, forward FFT along y, phasor, inverse FFT along y,
// in place in M (only the nby box rows are read and written).  STAGE: the
// column's folded phasor row is copied into the team's buffer behind its
// scratch (cp.async, issued before the forward transform) and read from there.
template <typename C, int N, int NZ, int NT, bool HALF = false, bool STAGE = false>
__device__ __forceinline__ void fused_phase2(const FusedArgs<C>& a, const C* Q, C* M, C* scr,
                                             const C* tw, int team, int g) {
  using X = FusedCtx<C, N>;
  constexpr int G = X::G, RR = X::RR, CC = X::CC, P = X::P;
  constexpr int NTEAM = NT;
  const int nby = a.nby;
  const int QW = a.fold ? N / 2 : N;
  const int rv = (nby + G - 1) / G;
  C* qb = STAGE ? scr + X::T::template scratch<HALF>() : nullptr;
  for (int base = 0; base < N; base += NTEAM) {
    const int kx = base + team;
    const bool act = kx < N;
    if (!__any_sync(0xffffffffu, act)) continue;
    if constexpr (STAGE) {
      if (act && a.fold) {
        constexpr int E = 16 / sizeof(C);   // elements per 16-byte chunk
        const C* row = Q + (size_t)(kx < N / 2 ? kx : N - 1 - kx) * QW;
        for (int c = g; c < (N / 2) / E; c += G) cp_async16(qb + c * E, row + c * E);
      }
      cp_async_commit();
    }
    C v[RR];
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      v[r] = czero<C>();
      if (r < NZ && r < rv) {
        const int y = g + G * r;
        if (act && y < nby) v[r] = M[y * P + kx];
      }
    }
    X::T::template forward<NZ, HALF>(v, tw, scr, g);
    if constexpr (STAGE) {
      cp_async_wait_all();
      __syncwarp();
    }
    if (act) {
      if (a.fold) {
        mul_folded<N>(v, STAGE ? qb : Q + (size_t)(kx < N / 2 ? kx : N - 1 - kx) * QW, g);
      } else {
        const C* Qrow = Q + (size_t)kx * QW;
#pragma unroll
        for (int j = 0; j < CC; ++j)
#pragma unroll
          for (int q = 0; q < G; ++q) v[j * G + q] = cmul(v[j * G + q], Qrow[g * CC + j + RR * q]);
      }
    }
    // (the inverse's exchange syncs the warp: every lane has read the buffer
    // before the next task's copies overwrite it)
    X::T::template inverse<HALF>(v, tw, scr, g);
    if (act) {
#pragma unroll
      for (int r = 0; r < RR; ++r) {
        if (r < NZ && r < rv) {
          const int y = g + G * r;
          if (y < nby) M[y * P + kx] = v[r];
        }
      }
    }
  }
  __syncthreads();
}

// Phase 3: inverse FFT along x of every box row, tilt/surface map, then the
// epilogue: store the propagated field into obuf (first of two propagations)
// or apply the boundary mix and write the new (masked) fields.
template <typename C, int N, bool MIX, int NZ, int NT, bool HALF = false>
__device__ __forceinline__ void fused_phase3(const FusedArgs<C>& a, const StepDesc& sd, int f, int region,
                                             bool prop_is_b, C* M, C* scr, C* obuf,
                                             const C* tw, int team, int g) {
  using X = FusedCtx<C, N>;
  constexpr int G = X::G, RR = X::RR, CC = X::CC, P = X::P;
  constexpr int NTEAM = NT;
  const int nbx = a.nbx, nby = a.nby;
  const size_t plane = (size_t)nby * nbx;
  const int ti = a.tilt_idx[region];
  const C* tmap = ti >= 0 ? a.tilt + ((size_t)f * a.ntilt + ti) * plane : nullptr;
  C* stA = sd.sa >= 0 ? a.state + ((size_t)f * a.nslots + sd.sa) * plane : nullptr;
  C* stB = sd.sb >= 0 ? a.state + ((size_t)f * a.nslots + sd.sb) * plane : nullptr;
  const C* add = (MIX && sd.addA >= 0) ? a.addbuf + (size_t)sd.addA * plane : nullptr;
  C cAA, cAB, cBA, cBB;
  if (MIX) {
    const C* cf = a.coefs + 4 * sd.coef;
    cAA = cf[0]; cAB = cf[1]; cBA = cf[2]; cBB = cf[3];
  }
  // the boundary's other operand: A~ parked in obuf, or a slot's stored field
  const C* oth = MIX ? (prop_is_b ? (sd.ra >= 0 ? obuf : stA) : stB) : nullptr;
  for (int base = 0; base < nby; base += NTEAM) {
    const int y = base + team;
    const bool act = y < nby;
    if (!__any_sync(0xffffffffu, act)) continue;
    C v[RR];
#pragma unroll
    for (int j = 0; j < CC; ++j)
#pragma unroll
      for (int q = 0; q < G; ++q) v[j * G + q] = act ? M[y * P + g * CC + j + RR * q] : czero<C>();
    X::T::template inverse<HALF>(v, tw, scr, g);
    if (!act) continue;
    // The operands of S points are loaded together before any is used or a
    // result stored: a load per point between the stores (which may alias it)
    // waited for memory once per point, 42 % of the warps' time at N = 80.
    constexpr int S = NZ < 3 ? NZ : 3;
#pragma unroll
    for (int r0 = 0; r0 < NZ; r0 += S) {
      C tm[S], ot[S], ad[S];
      bool in[S];
#pragma unroll
      for (int k = 0; k < S; ++k) {
        const int x = g + G * (r0 + k), i = y * nbx + x;
        if (r0 + k >= NZ || x >= nbx) continue;
        if (tmap) tm[k] = tmap[i];
        if (MIX) {
          ot[k] = oth ? oth[i] : czero<C>();
          in[k] = a.mask[i] != 0;
          if (add) ad[k] = add[i];
        }
      }
#pragma unroll
      for (int k = 0; k < S; ++k) {
        const int x = g + G * (r0 + k), i = y * nbx + x;
        if (r0 + k >= NZ || x >= nbx) continue;
        C p = v[r0 + k];
        if (tmap) p = cmul(p, tm[k]);
        if (!MIX) {
          obuf[i] = p;
        } else {
          // new fields are stored masked (their next propagation masks them anyway)
          const C tA = prop_is_b ? ot[k] : p, tB = prop_is_b ? p : ot[k];
          if (stA) {
            C o = cadd(cmul(cAA, tA), cmul(cAB, tB));
            if (add) o = cadd(o, ad[k]);
            stA[i] = in[k] ? o : czero<C>();
          }
          if (stB) stB[i] = in[k] ? cadd(cmul(cBA, tA), cmul(cBB, tB)) : czero<C>();
        }
      }
    }
  }
}

// ---- joint step: both slots processed together ------------------------------
// The rows of A and of B form one task list (2 nby rows), and so do their
// columns (2 N), so the teams stay busy where a single field's nby rows leave
// most of them idle in the last round; the propagated fields stay in the row
// tiles MA, MB and the boundary mix runs as one pass over the box.  A team
// takes the tasks t0 + team, t0 + team + ts, ... (the fused kernel: t0 = 0,
// ts = its teams; the split-phase kernels spread the tasks over CTAs); the
// tasks of a slot that is not propagated (pa / pb false) are skipped.

// Phase 1, joint: forward FFT along x of the box rows of A (tasks < nby) and B.
template <typename C, int N, int NZ, int NT, bool SPLIT, bool HALF = false>
__device__ __forceinline__ void joint_phase1(const FusedArgs<C>& a, const StepDesc& sd, int f, C* MA, C* MB,
                                             C* scr, const C* tw, int team, int g, int t0, int ts,
                                             bool pa, bool pb) {
  using X = FusedCtx<C, N>;
  constexpr int G = X::G, RR = X::RR, CC = X::CC, P = X::P;
  const int nbx = a.nbx, nby = a.nby, ntask = 2 * nby;
  const int rv = (nbx + G - 1) / G;
  // the fused kernel's joint steps: all tasks of the CTA, both slots propagated
  const int T0 = SPLIT ? t0 : 0, TS = SPLIT ? ts : NT;
  for (int base = T0; base < ntask; base += TS) {
    const int t = base + team;
    const bool act = t < ntask && (!SPLIT || (t >= nby ? pb : pa));
    if (!__any_sync(0xffffffffu, act)) continue;
    const bool isb = act && t >= nby;
    const int y = act ? (isb ? t - nby : t) : 0;
    const int slot = isb ? sd.sb : sd.sa, exitk = isb ? sd.exitB : sd.exitA;
    const C* row = a.state + (((size_t)f * a.nslots + slot) * nby + y) * (size_t)nbx;
    double2* arow = exitk >= 0 ? a.exitacc + (((size_t)exitk * a.nfreq + f) * nby + y) * (size_t)nbx : nullptr;
    C v[RR];
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      v[r] = czero<C>();
      if (r < NZ && r < rv) {
        const int x = g + G * r;
        if (act && x < nbx) v[r] = row[x];
      }
    }
    if (act && arow) exit_add<NZ, G>(arow, v, g, nbx);
    X::T::template forward<NZ, HALF>(v, tw, scr, g);
    if (act) {
      C* M = isb ? MB : MA;
#pragma unroll
      for (int j = 0; j < CC; ++j)
#pragma unroll
        for (int q = 0; q < G; ++q) M[y * P + g * CC + j + RR * q] = v[j * G + q];
    }
  }
  __syncthreads();
}

// Ask L2 for the phasor row of column task t (rows of 128-byte lines, one per
// thread g of the team), so that it is there when the team reaches that task.
// QA / QB are null for a slot that is not propagated.
template <typename C, int N, bool MAYBE_NULL>
__device__ __forceinline__ void prefetch_qrow(const FusedArgs<C>& a, const C* QA, const C* QB, int t, int g) {
  if (t >= 2 * N) return;
  const int QW = a.fold ? N / 2 : N;
  const int kx = t < N ? t : t - N;
  const C* Q = t < N ? QA : QB;
  if (MAYBE_NULL && !Q) return;
  const C* row = Q + (size_t)(a.fold ? (kx < N / 2 ? kx : N - 1 - kx) : kx) * QW;
  const int lines = (int)((sizeof(C) * QW + 127) / 128);
  if (g < lines) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(row) + 128 * g));
}

// Phase 2, joint: columns of A (tasks < N) and of B, each with its region's phasor.
// STAGE as fused_phase2 (the fused kernel only).
template <typename C, int N, int NZ, int NT, bool SPLIT, bool HALF = false, bool STAGE = false>
__device__ __forceinline__ void joint_phase2(const FusedArgs<C>& a, const C* QA, const C* QB, C* MA, C* MB, C* scr,
                                             const C* tw, int team, int g, int t0, int ts) {
  using X = FusedCtx<C, N>;
  constexpr int G = X::G, RR = X::RR, CC = X::CC, P = X::P;
  static_assert(!(SPLIT && STAGE), "staged phasor rows: fused kernel only");
  const int nby = a.nby;
  const int QW = a.fold ? N / 2 : N;
  const int rv = (nby + G - 1) / G;
  const int T0 = SPLIT ? t0 : 0, TS = SPLIT ? ts : NT;
  C* qb = STAGE ? scr + X::T::template scratch<HALF>() : nullptr;
  for (int base = T0; base < 2 * N; base += TS) {
    const int t = base + team;
    const bool act = t < 2 * N && (!SPLIT || (t >= N ? QB : QA) != nullptr);
    if (!__any_sync(0xffffffffu, act)) continue;
    const bool isb = act && t >= N;
    const int kx = act ? (isb ? t - N : t) : 0;
    C* M = isb ? MB : MA;
    const C* Q = isb ? QB : QA;
    if constexpr (STAGE) {
      if (act && a.fold) {
        constexpr int E = 16 / sizeof(C);   // elements per 16-byte chunk
        const C* row = Q + (size_t)(kx < N / 2 ? kx : N - 1 - kx) * QW;
        for (int c = g; c < (N / 2) / E; c += G) cp_async16(qb + c * E, row + c * E);
      }
      cp_async_commit();
      if (!a.fold) prefetch_qrow<C, N, SPLIT>(a, QA, QB, t + TS, g);
    } else {
      prefetch_qrow<C, N, SPLIT>(a, QA, QB, t + TS, g);
    }
    C v[RR];
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      v[r] = czero<C>();
      if (r < NZ && r < rv) {
        const int y = g + G * r;
        if (act && y < nby) v[r] = M[y * P + kx];
      }
    }
    X::T::template forward<NZ, HALF>(v, tw, scr, g);
    if constexpr (STAGE) {
      cp_async_wait_all();
      __syncwarp();
    }
    if (act) {
      if (a.fold) {
        mul_folded<N>(v, STAGE ? qb : Q + (size_t)(kx < N / 2 ? kx : N - 1 - kx) * QW, g);
      } else {
        const C* Qrow = Q + (size_t)kx * QW;
#pragma unroll
        for (int j = 0; j < CC; ++j)
#pragma unroll
          for (int q = 0; q < G; ++q) v[j * G + q] = cmul(v[j * G + q], Qrow[g * CC + j + RR * q]);
      }
    }
    // (the inverse's exchange syncs the warp before the buffer is refilled)
    X::T::template inverse<HALF>(v, tw, scr, g);
    if (act) {
#pragma unroll
      for (int r = 0; r < RR; ++r) {
        if (r < NZ && r < rv) {
          const int y = g + G * r;
          if (y < nby) M[y * P + kx] = v[r];
        }
      }
    }
  }
  __syncthreads();
}

// Phase 3, joint: inverse FFT along x of the box rows of A and B, written back
// in place into the row's first nbx entries (the team's exchange has already
// consumed the row).
template <typename C, int N, int NZ, int NT, bool SPLIT, bool HALF = false>
__device__ __forceinline__ void joint_phase3(const FusedArgs<C>& a, C* MA, C* MB, C* scr, const C* tw, int team,
                                             int g, int t0, int ts, bool pa, bool pb) {
  using X = FusedCtx<C, N>;
  constexpr int G = X::G, RR = X::RR, CC = X::CC, P = X::P;
  const int nbx = a.nbx, nby = a.nby, ntask = 2 * nby;
  const int T0 = SPLIT ? t0 : 0, TS = SPLIT ? ts : NT;
  for (int base = T0; base < ntask; base += TS) {
    const int t = base + team;
    const bool act = t < ntask && (!SPLIT || (t >= nby ? pb : pa));
    if (!__any_sync(0xffffffffu, act)) continue;
    const bool isb = act && t >= nby;
    const int y = act ? (isb ? t - nby : t) : 0;
    C* M = isb ? MB : MA;
    C v[RR];
#pragma unroll
    for (int j = 0; j < CC; ++j)
#pragma unroll
      for (int q = 0; q < G; ++q) v[j * G + q] = act ? M[y * P + g * CC + j + RR * q] : czero<C>();
    X::T::template inverse<HALF>(v, tw, scr, g);
    if (!act) continue;
#pragma unroll
    for (int r = 0; r < NZ; ++r)
      if (g + G * r < nbx) M[y * P + g + G * r] = v[r];
  }
  __syncthreads();
}

// Boundary mix of a step over the box: A' = cAA A~ + cAB B~ (+ add),
// B' = cBA A~ + cBB B~, stored masked; X~ is the propagated field (row tile)
// of a propagated slot times its region's tilt/surface map, else the slot's
// stored field.  Pixels i0, i0 + is, ... below `end`, K at a time: the loads of K pixels
// come before their stores (which may alias them, as far as the compiler
// knows), so memory is waited for once per K pixels instead of once per pixel.
template <typename C, int N, int K>
__device__ __forceinline__ void joint_mix(const FusedArgs<C>& a, const StepDesc& sd, int f, const C* MA,
                                          const C* MB, bool pa, bool pb, int i0, int is, int end = 1 << 30) {
  constexpr int P = FusedCtx<C, N>::P;
  const int nbx = a.nbx, plane = nbx * a.nby;
  end = min(end, plane);
  const unsigned magic = 0xffffffffu / (unsigned)nbx + 1u;   // i / nbx = umulhi(i, magic) for i < 2^16, nbx > 1
  C* stA = sd.sa >= 0 ? a.state + ((size_t)f * a.nslots + sd.sa) * plane : nullptr;
  C* stB = sd.sb >= 0 ? a.state + ((size_t)f * a.nslots + sd.sb) * plane : nullptr;
  const C* add = sd.addA >= 0 ? a.addbuf + (size_t)sd.addA * plane : nullptr;
  const int tiA = pa ? a.tilt_idx[sd.ra] : -1, tiB = pb ? a.tilt_idx[sd.rb] : -1;
  const C* tmA = tiA >= 0 ? a.tilt + ((size_t)f * a.ntilt + tiA) * plane : nullptr;
  const C* tmB = tiB >= 0 ? a.tilt + ((size_t)f * a.ntilt + tiB) * plane : nullptr;
  const C* cf = a.coefs + 4 * sd.coef;
  const C cAA = cf[0], cAB = cf[1], cBA = cf[2], cBB = cf[3];
  for (int b = i0; b < end; b += K * is) {
    C tA[K], tB[K], A[K], B[K], ad[K];
    bool in[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = b + k * is;
      if (i >= end) continue;
      if (tmA) tA[k] = tmA[i];
      if (tmB) tB[k] = tmB[i];
      if (!pa) A[k] = stA ? stA[i] : czero<C>();
      if (!pb) B[k] = stB ? stB[i] : czero<C>();
      if (add) ad[k] = add[i];
      in[k] = a.mask[i] != 0;
      const int y = nbx > 1 ? (int)__umulhi(i, magic) : i, x = i - y * nbx;
      if (pa) A[k] = MA[y * P + x];
      if (pb) B[k] = MB[y * P + x];
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = b + k * is;
      if (i >= end) continue;
      if (tmA) A[k] = cmul(A[k], tA[k]);
      if (tmB) B[k] = cmul(B[k], tB[k]);
      if (stA) {
        C o = cadd(cmul(cAA, A[k]), cmul(cAB, B[k]));
        if (add) o = cadd(o, ad[k]);
        stA[i] = in[k] ? o : czero<C>();
      }
      if (stB) stB[i] = in[k] ? cadd(cmul(cBA, A[k]), cmul(cBB, B[k])) : czero<C>();
    }
  }
}

// One bounce stage: grid = (steps of the stage, frequencies).  JOINT: steps
// with both slots propagated take the joint path (twice the row tile in
// shared memory).  NZ: box lines occupy at most NZ of a thread's RR register
// slots (x = g + G r < nbx, y = g + G r < nby only for r < NZ), so the first
// forward pass is pruned and the inverse stores only NZ slots.  MINB: CTAs
// per SM the registers are sized for.  MODE: kModeTwShared | kModeHalf |
// kModeStage (fewer registers or less shared memory per warp, so more warps
// per SM, and phasor rows staged ahead); the arithmetic, and so every result,
// is the same.
template <typename R, int N, bool JOINT, int NZ, int THREADS, int MINB, int MODE>
__global__ void __launch_bounds__(THREADS, MINB) k_fused_stage(FusedArgs<cplx_t<R>> a) {
  using C = cplx_t<R>;
  using X = FusedCtx<C, N>;
  constexpr int G = X::G, RR = X::RR, P = X::P;
  constexpr int NTEAM = THREADS / G;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int nby = a.nby;
  C* M = reinterpret_cast<C*>(smem_raw + kSmemHeader);
  C* scr_all = M + tile_elements<N>(JOINT ? 2 : 1, nby);
  const int tid = threadIdx.x, team = tid / G, g = tid % G;
  constexpr bool HALF = (MODE & kModeHalf) != 0, STAGE = (MODE & kModeStage) != 0;
  C* scr = scr_all + team * team_region<N, MODE>();
  const StepDesc sd = a.steps[blockIdx.x];
  const int f = blockIdx.y;
  C twr[RR];
  const C* tw = twr;
  if constexpr ((MODE & kModeTwShared) != 0) {
    // tw[g][s] = W_N^(g s) behind the teams' regions, rows RR + 1 apart so
    // that the G threads of a team reading their s-th twiddle hit distinct banks
    C* tws = scr_all + NTEAM * team_region<N, MODE>();
    for (int i = tid; i < G * RR; i += THREADS)
      tws[(i / RR) * (RR + 1) + i % RR] = root_n<N, C>((i / RR) * (i % RR));
    __syncthreads();
    tw = tws + g * (RR + 1);
  } else {
    team_twiddles<N>(twr, g);
  }
  const int QW = a.fold ? N / 2 : N;
  auto qptr = [&](int region) -> const C* {
    return a.phasor + ((size_t)f * a.ntab + a.tab_idx[region]) * (size_t)(QW * QW);
  };
  const bool pa = sd.ra >= 0, pb = sd.rb >= 0;
  if (JOINT && pa && pb) {
    C* MB = M + nby * P;
    prefetch_qrow<C, N, false>(a, qptr(sd.ra), qptr(sd.rb), team, g);
    joint_phase1<C, N, NZ, NTEAM, false, HALF>(a, sd, f, M, MB, scr, tw, team, g, 0, NTEAM, true, true);
    joint_phase2<C, N, NZ, NTEAM, false, HALF, STAGE>(a, qptr(sd.ra), qptr(sd.rb), M, MB, scr, tw, team, g, 0,
                                                      NTEAM);
    joint_phase3<C, N, NZ, NTEAM, false, HALF>(a, M, MB, scr, tw, team, g, 0, NTEAM, true, true);
    joint_mix<C, N, sizeof(C) == 8 ? 5 : 2>(a, sd, f, M, MB, true, true, threadIdx.x, THREADS);
  } else if (pa && pb) {
    // A~ is parked in the A slot itself until the boundary mix
    C* obuf = a.state + ((size_t)f * a.nslots + sd.sa) * (size_t)(nby * a.nbx);
    fused_phase1<C, N, NZ, NTEAM, HALF>(a, f, sd.sa, sd.exitA, M, scr, tw, team, g);
    fused_phase2<C, N, NZ, NTEAM, HALF, STAGE>(a, qptr(sd.ra), M, scr, tw, team, g);
    fused_phase3<C, N, false, NZ, NTEAM, HALF>(a, sd, f, sd.ra, false, M, scr, obuf, tw, team, g);
    // no barrier: B's forward row pass writes row y of M through the same
    // team (y mod NTEAM) and the same per-thread elements that A's inverse row
    // pass just read from it, and A~ goes to global memory, read back in B's
    // mix by the same thread; program order already orders every access
    fused_phase1<C, N, NZ, NTEAM, HALF>(a, f, sd.sb, sd.exitB, M, scr, tw, team, g);
    fused_phase2<C, N, NZ, NTEAM, HALF, STAGE>(a, qptr(sd.rb), M, scr, tw, team, g);
    fused_phase3<C, N, true, NZ, NTEAM, HALF>(a, sd, f, sd.rb, true, M, scr, obuf, tw, team, g);
  } else if (pa) {
    fused_phase1<C, N, NZ, NTEAM, HALF>(a, f, sd.sa, sd.exitA, M, scr, tw, team, g);
    fused_phase2<C, N, NZ, NTEAM, HALF, STAGE>(a, qptr(sd.ra), M, scr, tw, team, g);
    fused_phase3<C, N, true, NZ, NTEAM, HALF>(a, sd, f, sd.ra, false, M, scr, nullptr, tw, team, g);
  } else if (pb) {
    fused_phase1<C, N, NZ, NTEAM, HALF>(a, f, sd.sb, sd.exitB, M, scr, tw, team, g);
    fused_phase2<C, N, NZ, NTEAM, HALF, STAGE>(a, qptr(sd.rb), M, scr, tw, team, g);
    fused_phase3<C, N, true, NZ, NTEAM, HALF>(a, sd, f, sd.rb, true, M, scr, nullptr, tw, team, g);
  }
}

// ---- split-phase stage: for stages with fewer steps x frequencies than SMs --
// The four phases of a step (forward rows, columns, inverse rows, boundary
// mix) run as four launches whose tasks are spread over blockIdx.z, so a
// stage with a handful of steps (one frequency, a short stack) still spreads
// its FFT work over many SMs.  The row tiles of step s, frequency f live in
// global memory at a.mg + (s nfreq + f) 2 nby P (A, then B) and stay in L2.
constexpr int kSplitThreads = 64;

template <typename R, int N, int NZ>
__global__ void __launch_bounds__(kSplitThreads) k_split_phase(FusedArgs<cplx_t<R>> a, int phase) {
  using C = cplx_t<R>;
  using X = FusedCtx<C, N>;
  constexpr int G = X::G, RR = X::RR, P = X::P;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int tid = threadIdx.x, team = tid / G, g = tid % G, nteam = blockDim.x / G;
  // programmatic dependent launch: let the next phase launch now, and wait for
  // the previous phase (its writes visible) before reading anything it wrote
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  C tw[RR];
  team_twiddles<N>(tw, g);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const StepDesc sd = a.steps[blockIdx.x];
  const int f = blockIdx.y;
  C* MA = a.mg + ((size_t)blockIdx.x * a.nfreq + f) * 2 * (size_t)a.nby * P;
  C* MB = MA + (size_t)a.nby * P;
  const bool pa = sd.ra >= 0, pb = sd.rb >= 0;
  if (phase == 3) {
    joint_mix<C, N, 1>(a, sd, f, MA, MB, pa, pb, blockIdx.z * blockDim.x + tid, gridDim.z * blockDim.x);
    return;
  }
  C* scr = reinterpret_cast<C*>(smem_raw) + team * X::T::template scratch<false>();
  const int t0 = blockIdx.z * nteam, ts = gridDim.z * nteam;
  if (phase == 0) {
    joint_phase1<C, N, NZ, kSplitThreads / G, true>(a, sd, f, MA, MB, scr, tw, team, g, t0, ts, pa, pb);
  } else if (phase == 1) {
    const int QW = a.fold ? N / 2 : N;
    const C* QA = pa ? a.phasor + ((size_t)f * a.ntab + a.tab_idx[sd.ra]) * (size_t)(QW * QW) : nullptr;
    const C* QB = pb ? a.phasor + ((size_t)f * a.ntab + a.tab_idx[sd.rb]) * (size_t)(QW * QW) : nullptr;
    joint_phase2<C, N, NZ, kSplitThreads / G, true>(a, QA, QB, MA, MB, scr, tw, team, g, t0, ts);
  } else {
    joint_phase3<C, N, NZ, kSplitThreads / G, true>(a, MA, MB, scr, tw, team, g, t0, ts, pa, pb);
  }
}

// ---- a run of split stages in one launch --------------------------------------
// The same phases by one resident grid of single-warp CTAs (the FP64 pipe takes
// 16 cycles a warp instruction, so a phase's warps go to as many SMs as there
// are), with barriers in place of the launches: three a stage, since the warp
// that transforms a row of A and B back also mixes it.  Bound by latency: the
// one-frequency dancer at 64^2 (4 steps a stage) took 35 us a stage with four
// launches, 29 us here, of which the barriers are 4 (1.3 us each).

// Every CTA of the (cooperatively launched) grid arrives; false when the wait
// gave up after `limit` cycles or another CTA's did.
__device__ __forceinline__ bool run_barrier(unsigned* bar, unsigned target, long long limit, int* err) {
  __syncwarp();
  bool ok = true;
  if ((threadIdx.x & 31) == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    const long long t0 = clock64();
    for (;;) {
      unsigned n;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(bar) : "memory");
      if (n >= target) break;
      if (*reinterpret_cast<volatile unsigned*>(bar + 1)) {
        ok = false;
        break;
      }
      if (clock64() - t0 > limit) {
        atomicExch(err, 1);
        atomicExch(bar + 1, 1u);
        ok = false;
        break;
      }
    }
    __threadfence();
  }
  __syncwarp();
  return __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
}

template <typename R, int N, int NZ>
__global__ void __launch_bounds__(32) k_split_run(FusedArgs<cplx_t<R>> a) {
  using C = cplx_t<R>;
  using X = FusedCtx<C, N>;
  constexpr int G = X::G, RR = X::RR, CC = X::CC, P = X::P, NT = 32 / G;
  constexpr int RW = NT > 1 ? NT / 2 : 1;   // rows of a warp's last phase, of A and of B
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int lane = threadIdx.x, team = lane / G, g = lane % G;
  const int nbx = a.nbx, nby = a.nby;
  C* scr = reinterpret_cast<C*>(smem_raw) + team * X::T::template scratch<false>();
  C tw[RR];
  team_twiddles<N>(tw, g);
  const int z[3] = {(2 * nby + NT - 1) / NT, (2 * N + NT - 1) / NT, (nby + RW - 1) / RW};
  unsigned target = 0;
  for (int k = 0; k < a.run_len; ++k) {
    const int off = a.run_tab[k], ns = a.run_tab[k + 1] - off;
    for (int ph = 0; ph < 3; ++ph) {
      const int total = ns * a.nfreq * z[ph];
      for (int vb = blockIdx.x; vb < total; vb += gridDim.x) {
        const int zi = vb % z[ph], s = vb / z[ph] % ns, f = vb / (z[ph] * ns);
        const StepDesc sd = a.steps[off + s];
        C* MA = a.mg + ((size_t)s * a.nfreq + f) * 2 * (size_t)nby * P;
        C* MB = MA + (size_t)nby * P;
        const bool pa = sd.ra >= 0, pb = sd.rb >= 0;
        if (ph == 0) {
          joint_phase1<C, N, NZ, NT, true>(a, sd, f, MA, MB, scr, tw, team, g, zi * NT, 2 * nby, pa, pb);
        } else if (ph == 1) {
          const int QW = a.fold ? N / 2 : N;
          const C* QA = pa ? a.phasor + ((size_t)f * a.ntab + a.tab_idx[sd.ra]) * (size_t)(QW * QW) : nullptr;
          const C* QB = pb ? a.phasor + ((size_t)f * a.ntab + a.tab_idx[sd.rb]) * (size_t)(QW * QW) : nullptr;
          joint_phase2<C, N, NZ, NT, true>(a, QA, QB, MA, MB, scr, tw, team, g, zi * NT, 2 * N);
        } else {
          const int y0 = zi * RW;
#pragma unroll
          for (int h = 0; h < 2 * RW / NT; ++h) {
            const int q = h * NT + team, y = y0 + q / 2;
            const bool isb = q & 1, act = y < nby && (isb ? pb : pa);
            C* row = (isb ? MB : MA) + (act ? y : 0) * P;
            C v[RR];
#pragma unroll
            for (int j = 0; j < CC; ++j)
#pragma unroll
              for (int i = 0; i < G; ++i) v[j * G + i] = act ? row[g * CC + j + RR * i] : czero<C>();
            X::T::template inverse<false>(v, tw, scr, g);
            if (act)
#pragma unroll
              for (int r = 0; r < NZ; ++r)
                if (g + G * r < nbx) row[g + G * r] = v[r];
          }
          __syncwarp();
          joint_mix<C, N, 1>(a, sd, f, MA, MB, pa, pb, y0 * nbx + lane, 32, (y0 + RW) * nbx);
        }
      }
      if (k + 1 == a.run_len && ph == 2) break;
      target += gridDim.x;
      if (!run_barrier(a.run_bar, target + a.run_late, a.run_limit, a.err)) return;
    }
  }
}

static const size_t kMaxSmem = 227 * 1024;

// Shared memory of one SM (bytes) and what the driver reserves per CTA.
static const size_t kSmemPerSM = 228 * 1024, kSmemReservedPerCta = 1024;

// The dynamic shared-memory limit of a kernel is raised to the per-block
// maximum, the same value for every launch: launches of one kernel with
// different sizes from several host threads (the serving engine's workers)
// must not lower it under one another.
template <typename R, int N, bool JOINT, int NZ, int THREADS = kFusedThreads,
          int MINB = (sizeof(R) == 4 && N <= 128) ? 2 : 1, int MODE = 0>
static int launch_fused_v(const FusedArgs<cplx_t<R>>& a, dim3 grid, size_t smem, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(k_fused_stage<R, N, JOINT, NZ, THREADS, MINB, MODE>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
  if (e != cudaSuccess) return (int)e;
  k_fused_stage<R, N, JOINT, NZ, THREADS, MINB, MODE><<<grid, THREADS, smem, st>>>(a);
  return (int)cudaGetLastError();
}

template <typename R, int N, int NZ>
static int launch_split_run(const FusedArgs<cplx_t<R>>& a, int nsteps, cudaStream_t st) {
  using T = Team<N>;
  constexpr int NT = 32 / T::G;
  const size_t smem = sizeof(cplx_t<R>) * NT * T::template scratch<false>();
  int dev = 0, sms = 0, per = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_split_run<R, N, NZ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_split_run<R, N, NZ>, 32, smem);
  if (e != cudaSuccess) return (int)e;
  if (a.max_ctas > 0) sms = std::min(sms, a.max_ctas);
  // no more CTAs than the widest phase has warps: each one more lengthens the barriers
  const long long widest = (long long)nsteps * a.nfreq * std::max((2 * N + NT - 1) / NT, a.nby);
  const int grid = (int)std::min<long long>(widest, (long long)sms * std::min(per, 4));
  e = cudaMemsetAsync(a.run_bar, 0, 2 * sizeof(unsigned), st);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  note_launch();
  return (int)cudaLaunchKernelEx(&cfg, k_split_run<R, N, NZ>, a);
}

template <typename R, int N, int NZ>
static int launch_split(const FusedArgs<cplx_t<R>>& a, int nsteps, cudaStream_t st) {
  if (a.run_len > 0) return launch_split_run<R, N, NZ>(a, nsteps, st);
  using T = Team<N>;
  const int nteam = kSplitThreads / T::G;
  const size_t smem = sizeof(cplx_t<R>) * nteam * T::template scratch<false>();
  const int zr = (2 * a.nby + nteam - 1) / nteam, zc = (2 * N + nteam - 1) / nteam;
  const int zm = (a.nbx * a.nby + kSplitThreads - 1) / kSplitThreads;
  const int z[4] = {zr, zc, zr, zm};
  // each phase may launch while the previous one drains (programmatic
  // dependent launch); the kernel waits for it before touching its data
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  for (int ph = 0; ph < 4; ++ph) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nsteps, a.nfreq, z[ph]);
    cfg.blockDim = dim3(kSplitThreads);
    cfg.dynamicSmemBytes = ph == 3 ? 0 : smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    note_launch();
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_split_phase<R, N, NZ>, a, ph);
    if (e != cudaSuccess) return (int)e;
  }
  return 0;
}

template <int N, int MODE = 0>
static size_t fused_smem_for(int nby, size_t csz, int tiles = 1, int threads = kFusedThreads) {
  const size_t nteam = threads / Team<N>::G;
  const size_t twt = (MODE & kModeTwShared) ? (size_t)Team<N>::G * (Team<N>::RR + 1) : 0;   // twiddle table
  return kSmemHeader + csz * ((size_t)tile_elements<N>(tiles, nby) + nteam * team_region<N, MODE>() + twt);
}

// Fill this translation unit's unit-root tables on the current device.
static inline void upload_roots() {
  static double2 hd[1024];
  static float2 hf[1024];
  fill_roots(1024, hd, hf);
  cudaMemcpyToSymbol(c_root1024_d, hd, sizeof(hd));
  cudaMemcpyToSymbol(c_root1024_f, hf, sizeof(hf));
  fill_roots(160, hd, hf);
  cudaMemcpyToSymbol(c_root160_d, hd, 160 * sizeof(double2));
  cudaMemcpyToSymbol(c_root160_f, hf, 160 * sizeof(float2));
}

}  // namespace bf
