// Register-resident FFT building blocks for the fused propagation kernels.
//
// A line of N = C*G*G points (N a power of two) is transformed by a "team" of
// G threads holding RR = C*G points each:
//   pass 1  every thread does an RR-point DFT over the points x[g + G*r]
//           (r = 0..RR-1) in registers and multiplies by W_N^(g*s);
//   exchange through a swizzled shared-memory tile (one write + one read);
//   pass 2  every thread does C G-point DFTs in registers.
// Afterwards thread g holds X[(g*C + j) + RR*q] in v[j*G + q].  The inverse is
// the exact adjoint (same exchange, conjugate roots) and returns the points to
// the x[g + G*r] layout, unnormalised (a factor N).
// With C = 2 the exchange can also run in two halves through a scratch tile of
// half the size (HALF): the same data movement, two more warp syncs.
//
// Lengths 40, 80 and 160 (5 2^a) hold RR = 20 or 40 points per thread.  Their
// RR-point DFT is a prime-factor one (5 x 4 or 5 x 8, no twiddles between the
// factors), so a 20-point DFT costs about what a 16-point radix-2 one does
// (112 packed adds and FMAs against 64 adds and ~40 twiddle operations).
#pragma once

#include "bf_common.cuh"

namespace bf {

// Unit roots W_1024^k = exp(-2 pi i k / 1024), filled from the host in FP64.
// Register FFTs index them with compile-time offsets, so they compile into
// constant-bank operands.  One copy per translation unit (upload_roots).
static __constant__ double2 c_root1024_d[1024];
static __constant__ float2 c_root1024_f[1024];

// Unit roots W_160^k of the lengths 40, 80 and 160.
static __constant__ double2 c_root160_d[160];
static __constant__ float2 c_root160_f[160];

template <typename C> __device__ __forceinline__ C root1024(int k);
template <> __device__ __forceinline__ float2 root1024<float2>(int k) { return c_root1024_f[k]; }
template <> __device__ __forceinline__ double2 root1024<double2>(int k) { return c_root1024_d[k]; }

template <typename C> __device__ __forceinline__ C root160(int k);
template <> __device__ __forceinline__ float2 root160<float2>(int k) { return c_root160_f[k]; }
template <> __device__ __forceinline__ double2 root160<double2>(int k) { return c_root160_d[k]; }
// W_N^k, 0 <= k < N
template <int N, typename C> __device__ __forceinline__ C root_n(int k) {
  static_assert(1024 % N == 0 || 160 % N == 0, "root table");
  if constexpr (1024 % N == 0) return root1024<C>(k * (1024 / N));
  else return root160<C>(k * (160 / N));
}

// Butterfly adds.  For complex64 both halves go through one packed FP32x2
// instruction (add/sub.rn.f32x2, Blackwell): an FFT is mostly complex adds, so
// this halves its add instructions.  Each lane rounds exactly like a scalar add.
template <typename C> __device__ __forceinline__ C vadd(C a, C b) { return cadd(a, b); }
template <typename C> __device__ __forceinline__ C vsub(C a, C b) { return csub(a, b); }
template <> __device__ __forceinline__ float2 vadd<float2>(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 pa, pb, pd;\n\tmov.b64 pa, {%2, %3};\n\tmov.b64 pb, {%4, %5};\n\t"
      "add.rn.f32x2 pd, pa, pb;\n\tmov.b64 {%0, %1}, pd;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
template <> __device__ __forceinline__ float2 vsub<float2>(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 pa, pb, pd;\n\tmov.b64 pa, {%2, %3};\n\tmov.b64 pb, {%4, %5};\n\t"
      "sub.rn.f32x2 pd, pa, pb;\n\tmov.b64 {%0, %1}, pd;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}

// a s + b, s real
__device__ __forceinline__ double2 vfma(double2 a, double s, double2 b) { return mk(fma(a.x, s, b.x), fma(a.y, s, b.y)); }
__device__ __forceinline__ float2 vfma(float2 a, float s, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 pa, pb, ps, pd;\n\tmov.b64 pa, {%2, %3};\n\tmov.b64 pb, {%4, %5};\n\tmov.b64 ps, {%6, %6};\n\t"
      "fma.rn.f32x2 pd, pa, ps, pb;\n\tmov.b64 {%0, %1}, pd;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(s));
  return d;
}

// v[i] *= W_M^k (forward) or conj(W_M^k) (inverse), k compile-time after unrolling.
template <int M, bool INV, typename C>
__device__ __forceinline__ C twiddle_mul(C a, int k) {
  if (k == 0) return a;
  if (4 * k == M) return cmul_mi<INV>(a);
  C w = root1024<C>(k * (1024 / M));
  return INV ? cmulc(a, w) : cmul(a, w);
}

template <int M>
__host__ __device__ constexpr int bitrev(int i) {
  int r = 0;
  for (int b = 1; b < M; b <<= 1) {
    r = (r << 1) | (i & 1);
    i >>= 1;
  }
  return r;
}

// In-register M-point DFT of v[OFF .. OFF+M-1] (radix-2 decimation in
// frequency followed by a static bit-reversal permutation).
template <int M, bool INV, int OFF, int LEN, typename C>
__device__ __forceinline__ void reg_dft(C (&v)[LEN]) {
  if constexpr (M == 1) {
    return;
  } else {
#pragma unroll
    for (int len = M; len >= 2; len >>= 1) {
      const int half = len >> 1;
#pragma unroll
      for (int i = 0; i < M; i += len) {
#pragma unroll
        for (int j = 0; j < half; ++j) {
          C a = v[OFF + i + j];
          C b = v[OFF + i + j + half];
          v[OFF + i + j] = vadd(a, b);
          v[OFF + i + j + half] = twiddle_mul<M, INV>(vsub(a, b), j * (M / len));
        }
      }
    }
#pragma unroll
    for (int i = 0; i < M; ++i) {
      const int r = bitrev<M>(i);
      if (r > i) {
        C t = v[OFF + i];
        v[OFF + i] = v[OFF + r];
        v[OFF + r] = t;
      }
    }
  }
}

// Zero pattern (bit p = point p is exactly zero) at the input of the stage of
// length len of an M-point DIF DFT with zero pattern Z0 at its input: a
// butterfly output is zero only if both of its inputs were.
template <int M, unsigned long long Z0>
__host__ __device__ constexpr unsigned long long dif_zero_mask(int len) {
  unsigned long long z = Z0;
  for (int l = M; l > len; l >>= 1) {
    const int half = l >> 1;
    unsigned long long n = 0;
    for (int p = 0; p < M; ++p)
      if (((z >> p) & 1ull) && ((z >> (p ^ half)) & 1ull)) n |= 1ull << p;
    z = n;
  }
  return z;
}

// Bits NZ .. M-1.
__host__ __device__ constexpr unsigned long long zeros_from(int NZ, int M) {
  unsigned long long z = 0;
  for (int p = NZ; p < M; ++p) z |= 1ull << p;
  return z;
}

// One DIF stage (length LEN) of reg_dft_nz, then the next.
template <int M, bool INV, unsigned long long Z0, int LEN, int VLEN, typename C>
__device__ __forceinline__ void dif_stage_nz(C (&v)[VLEN]) {
  constexpr unsigned long long zm = dif_zero_mask<M, Z0>(LEN);
  constexpr int half = LEN / 2;
#pragma unroll
  for (int i = 0; i < M; i += LEN) {
#pragma unroll
    for (int j = 0; j < half; ++j) {
      const int pa = i + j, pb = pa + half;
      const bool za = (zm >> pa) & 1ull, zb = (zm >> pb) & 1ull;
      const int k = j * (M / LEN);
      if (za && zb) continue;
      const C a = v[pa], b = v[pb];
      if (zb) {
        v[pb] = twiddle_mul<M, INV>(a, k);
      } else if (za) {
        v[pa] = b;
        v[pb] = twiddle_mul<M, INV>(csub(czero_of(b), b), k);
      } else {
        v[pa] = vadd(a, b);
        v[pb] = twiddle_mul<M, INV>(vsub(a, b), k);
      }
    }
  }
  if constexpr (LEN > 2) dif_stage_nz<M, INV, Z0, LEN / 2>(v);
}

// M-point DFT (M a power of two) of v[0 .. M-1] whose inputs in Z0 are zero.
template <int M, bool INV, unsigned long long Z0, typename C>
__device__ __forceinline__ void dft_pow2_z(C (&v)[M]) {
  dif_stage_nz<M, INV, Z0, M>(v);
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const int r = bitrev<M>(i);
    if (r > i) {
      C t = v[i];
      v[i] = v[r];
      v[r] = t;
    }
  }
}

// 5-point DFT in place (four real constants; m and u are the even and odd parts).
template <bool INV, typename C>
__device__ __forceinline__ void dft5(C& x0, C& x1, C& x2, C& x3, C& x4) {
  using R = decltype(x0.x);
  constexpr R c1 = (R)0.30901699437494742410, c2 = (R)-0.80901699437494742410;   // cos(2 pi/5), cos(4 pi/5)
  constexpr R s1 = (R)0.95105651629515357212, s2 = (R)0.58778525229247312917;    // sin(2 pi/5), sin(4 pi/5)
  const C t1 = vadd(x1, x4), t2 = vadd(x2, x3), t3 = vsub(x1, x4), t4 = vsub(x2, x3);
  const C m1 = vfma(t2, c2, vfma(t1, c1, x0)), m2 = vfma(t2, c1, vfma(t1, c2, x0));
  const C z = czero_of(x0);
  const C u1 = vfma(t4, s2, vfma(t3, s1, z)), u2 = vfma(t4, -s1, vfma(t3, s2, z));
  x0 = vadd(x0, vadd(t1, t2));
  const C a1 = cmul_mi<INV>(u1), a2 = cmul_mi<INV>(u2);   // -i u (forward), +i u (inverse)
  x1 = cadd(m1, a1);
  x4 = csub(m1, a1);
  x2 = cadd(m2, a2);
  x3 = csub(m2, a2);
}

// (5 B)-point DFT in registers, B = 4 or 8, by the prime-factor map: input
// r = B a + 5 b, output s = kA k1 + kB k2 (mod 5 B) with kA = 1 mod 5, 0 mod B
// and kB = 0 mod 5, 1 mod B, so W^(r s) = W_5^(a k1) W_B^(b k2) and no twiddle
// stands between the two factors; all index maps are compile-time renamings.
// Forward: inputs v[NZ ..] are zero and the B-point DFTs run first, pruned.
// Inverse: the 5-point DFTs first, so that outputs that the caller does not
// store (r >= NZ) are dead code in the B-point ones.
template <int B> struct PfaMap {
  static_assert(B == 4 || B == 8, "prime-factor DFT");
  static constexpr int M = 5 * B;
  static constexpr int kA = 16, kB = B == 4 ? 5 : 25;
  __host__ __device__ static constexpr int in(int a, int b) { return (B * a + 5 * b) % M; }
  __host__ __device__ static constexpr int out(int k1, int k2) { return (kA * k1 + kB * k2) % M; }
  // inputs b of column a that are zero when v[NZ ..] are
  __host__ __device__ static constexpr unsigned long long zeros(int a, int NZ) {
    unsigned long long z = 0;
    for (int b = 0; b < B; ++b)
      if (in(a, b) >= NZ) z |= 1ull << b;
    return z;
  }
};
template <int B, bool INV, int NZ, int A = 0, typename C>
__device__ __forceinline__ void pfa_columns(C (&v)[5 * B]) {
  using P = PfaMap<B>;
  constexpr unsigned long long Z = P::zeros(A, NZ);
  C w[B];
#pragma unroll
  for (int b = 0; b < B; ++b) w[b] = v[P::in(A, b)];
  dft_pow2_z<B, INV, Z>(w);
#pragma unroll
  for (int b = 0; b < B; ++b) v[P::in(A, b)] = w[b];
  if constexpr (A + 1 < 5) pfa_columns<B, INV, NZ, A + 1>(v);
}
template <int B, bool INV, int NZ, typename C>
__device__ __forceinline__ void pfa_dft(C (&v)[5 * B]) {
  using P = PfaMap<B>;
  if constexpr (!INV) pfa_columns<B, INV, NZ>(v);
#pragma unroll
  for (int b = 0; b < B; ++b)
    dft5<INV>(v[P::in(0, b)], v[P::in(1, b)], v[P::in(2, b)], v[P::in(3, b)], v[P::in(4, b)]);
  if constexpr (INV) pfa_columns<B, INV, P::M>(v);
  C w[P::M];
#pragma unroll
  for (int a = 0; a < 5; ++a)
#pragma unroll
    for (int b = 0; b < B; ++b) w[P::out(a, b)] = v[P::in(a, b)];
#pragma unroll
  for (int i = 0; i < P::M; ++i) v[i] = w[i];
}

// reg_dft<M, INV, 0> of v[0 .. M-1] whose inputs v[NZ ..] are zero: butterflies
// with a zero input reduce to a copy and a twiddle, those with two zero inputs
// vanish.  The results are those of the dense DFT (adding an exact zero
// changes nothing but the sign of a zero).
template <int M, bool INV, int NZ, int LEN, typename C>
__device__ __forceinline__ void reg_dft_nz(C (&v)[LEN]) {
  if constexpr (M % 5 == 0) {
    pfa_dft<M / 5, INV, (NZ < M ? NZ : M)>(v);
  } else if constexpr (NZ >= M || M < 2) {
    reg_dft<M, INV, 0>(v);
  } else {
    dft_pow2_z<M, INV, zeros_from(NZ, M)>(v);
  }
}

template <int N> struct TeamShape;
template <> struct TeamShape<8>   { static constexpr int G = 2,  RR = 4;  };
template <> struct TeamShape<16>  { static constexpr int G = 4,  RR = 4;  };
template <> struct TeamShape<32>  { static constexpr int G = 4,  RR = 8;  };
template <> struct TeamShape<40>  { static constexpr int G = 2,  RR = 20; };
template <> struct TeamShape<80>  { static constexpr int G = 4,  RR = 20; };
template <> struct TeamShape<160> { static constexpr int G = 4,  RR = 40; };
template <> struct TeamShape<64>  { static constexpr int G = 8,  RR = 8;  };
template <> struct TeamShape<128> { static constexpr int G = 8,  RR = 16; };
template <> struct TeamShape<256> { static constexpr int G = 16, RR = 16; };
template <> struct TeamShape<512> { static constexpr int G = 16, RR = 32; };

template <int N>
struct Team {
  static constexpr int G = TeamShape<N>::G;
  static constexpr int RR = TeamShape<N>::RR;
  static constexpr int C = RR / G;
  static_assert(C * G * G == N, "team shape");
  // scratch tile of one team, in complex elements; the pad staggers the tiles
  // of teams sharing a half-warp across shared-memory banks
  static constexpr int SCR = RR * G + (G < 16 ? G : 0);
  // the half-size tile of the two-half exchange: G rows of G points; the pad
  // puts the two teams of a half-warp on opposite halves of the banks
  static constexpr int SCRH = (RR / 2) * G + (G < 16 ? G : 0);
  // C > 2, G = 4 (lengths 80 and 160): the exchange runs in C rounds of G x G
  // points through two buffers used in turn (one warp sync a round); 36
  // elements a team put the 4 teams of a half-warp on distinct banks
  static constexpr bool CHUNKED = C > 2 && G == 4;
  static constexpr int SCRC = 2 * G * G + 4;
  template <bool HALF> __host__ __device__ static constexpr int scratch() { return CHUNKED ? SCRC : HALF ? SCRH : SCR; }

  __device__ static __forceinline__ int swz(int s, int g) { return s * G + (g ^ (s / C)); }

  // forward: v[r] = x[g + G r]  ->  v[j*G + q] = X[(g*C + j) + RR*q];
  // NZ < RR: the caller guarantees v[NZ ..] == 0 (pruned first pass);
  // tw: the thread's RR inter-pass twiddles (registers or shared memory)
  template <int NZ = RR, bool HALF = false, typename Cx>
  __device__ static __forceinline__ void forward(Cx (&v)[RR], const Cx* tw, Cx* scr, int g) {
    reg_dft_nz<RR, false, NZ>(v);
#pragma unroll
    for (int s = 1; s < RR; ++s) v[s] = cmul(v[s], tw[s]);
    if constexpr (CHUNKED) {
      Cx w[RR];
#pragma unroll
      for (int j = 0; j < C; ++j) {
        Cx* b = scr + (j & 1) * G * G;
#pragma unroll
        for (int t = 0; t < G; ++t) b[t * G + (g ^ t)] = v[C * t + j];
        __syncwarp();
#pragma unroll
        for (int gp = 0; gp < G; ++gp) w[j * G + gp] = b[g * G + (gp ^ g)];
      }
      __syncwarp();
#pragma unroll
      for (int s = 0; s < RR; ++s) v[s] = w[s];
    } else if constexpr (HALF) {
      static_assert(C == 2, "two-half exchange");
      // half j moves the points s = C t + j: row t, column g ^ t of the tile
      Cx w[RR];
#pragma unroll
      for (int j = 0; j < C; ++j) {
#pragma unroll
        for (int t = 0; t < G; ++t) scr[t * G + (g ^ t)] = v[C * t + j];
        __syncwarp();
#pragma unroll
        for (int gp = 0; gp < G; ++gp) w[j * G + gp] = scr[g * G + (gp ^ g)];
        __syncwarp();
      }
#pragma unroll
      for (int s = 0; s < RR; ++s) v[s] = w[s];
    } else {
#pragma unroll
      for (int s = 0; s < RR; ++s) scr[swz(s, g)] = v[s];
      __syncwarp();
#pragma unroll
      for (int j = 0; j < C; ++j)
#pragma unroll
        for (int gp = 0; gp < G; ++gp) v[j * G + gp] = scr[swz(g * C + j, gp)];
      __syncwarp();
    }
#pragma unroll
    for (int j = 0; j < C; ++j) reg_dft_sub<false>(v, j);
  }

  // inverse (adjoint of forward, unnormalised): v[j*G + q] = X[(g*C + j) + RR*q] -> v[r] = N x[g + G r]
  template <bool HALF = false, typename Cx>
  __device__ static __forceinline__ void inverse(Cx (&v)[RR], const Cx* tw, Cx* scr, int g) {
#pragma unroll
    for (int j = 0; j < C; ++j) reg_dft_sub<true>(v, j);
    if constexpr (CHUNKED) {
      Cx w[RR];
#pragma unroll
      for (int j = 0; j < C; ++j) {
        Cx* b = scr + (j & 1) * G * G;
#pragma unroll
        for (int gp = 0; gp < G; ++gp) b[g * G + (gp ^ g)] = v[j * G + gp];
        __syncwarp();
#pragma unroll
        for (int t = 0; t < G; ++t) w[C * t + j] = b[t * G + (g ^ t)];
      }
      __syncwarp();
#pragma unroll
      for (int s = 0; s < RR; ++s) v[s] = w[s];
    } else if constexpr (HALF) {
      static_assert(C == 2, "two-half exchange");
      Cx w[RR];
#pragma unroll
      for (int j = 0; j < C; ++j) {
#pragma unroll
        for (int gp = 0; gp < G; ++gp) scr[g * G + (gp ^ g)] = v[j * G + gp];
        __syncwarp();
#pragma unroll
        for (int t = 0; t < G; ++t) w[C * t + j] = scr[t * G + (g ^ t)];
        __syncwarp();
      }
#pragma unroll
      for (int s = 0; s < RR; ++s) v[s] = w[s];
    } else {
#pragma unroll
      for (int j = 0; j < C; ++j)
#pragma unroll
        for (int gp = 0; gp < G; ++gp) scr[swz(g * C + j, gp)] = v[j * G + gp];
      __syncwarp();
#pragma unroll
      for (int s = 0; s < RR; ++s) v[s] = scr[swz(s, g)];
      __syncwarp();
    }
#pragma unroll
    for (int s = 1; s < RR; ++s) v[s] = cmulc(v[s], tw[s]);
    if constexpr (RR % 5 == 0) pfa_dft<RR / 5, true, RR>(v);
    else reg_dft<RR, true, 0>(v);
  }

 private:
  template <bool INV, typename Cx>
  __device__ static __forceinline__ void reg_dft_sub(Cx (&v)[RR], int j) {
    // j is a compile-time constant after unrolling of the caller's loop
    if constexpr (C == 1) {
      reg_dft<G, INV, 0>(v);
    } else if constexpr (C == 2) {
      if (j == 0) reg_dft<G, INV, 0>(v);
      else reg_dft<G, INV, G>(v);
    } else {
      Cx w[G];
#pragma unroll
      for (int q = 0; q < G; ++q) w[q] = v[j * G + q];
      reg_dft<G, INV, 0>(w);
#pragma unroll
      for (int q = 0; q < G; ++q) v[j * G + q] = w[q];
    }
  }
};

// Per-thread inter-pass twiddles W_N^(g*s), s = 0..RR-1 (g*s < N always).
template <int N, typename Cx>
__device__ __forceinline__ void team_twiddles(Cx (&tw)[Team<N>::RR], int g) {
#pragma unroll
  for (int s = 0; s < Team<N>::RR; ++s) tw[s] = root_n<N, Cx>(g * s);
}

}  // namespace bf
