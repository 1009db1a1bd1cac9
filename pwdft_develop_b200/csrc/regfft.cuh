// Register-resident 1-D transforms for sm_100a.
//
// A transform of length N lives in the registers of P lanes, M = N / P
// elements each: one lane up to 48 elements in FP32 (96 registers of data)
// and 24 (or 30) in FP64, two lanes above (80 fields of z pencils, forward, table,
// inverse: 60 in one lane 61 us, in two 53; 72 119 and 85; one lane of 48 in FP64
// would need 192 registers of data).  Nothing goes through shared memory inside
// a transform; the two-lane form exchanges M / 2 elements by shuffles for its
// last (first) radix-2 stage.
//
//   fft_dit  in: v[m] = x[P m + p] (interleaved), out: v[j] = X[kout(p, j)]
//   fft_dif  in: v[j] = X[kout(p, j)],            out: v[m] = x[P m + p]
// Forward transforms take fft_dif and inverse ones fft_dit: on decaying spectra
// that order rounds 2-8 % less at 60 and 72 than the other, and the two fit
// together without a change of layout.
//
// Lanes of one transform are 16 apart (p = lane >> 4), so that each half-warp
// walks 16 consecutive columns: full sectors in global memory and conflict-free
// rows in shared memory.  All lanes of a warp must call a two-lane transform.
#pragma once
#include "fft.cuh"

namespace pwb {

template <typename T, int N> struct RegN {
  static constexpr int P = N <= (sizeof(T) == 4 ? 48 : 24) || N == 30 ? 1 : 2;
  static constexpr int M = N / P;
  static constexpr int CW = 32 / P;    // transforms per warp
  static constexpr bool OK = N % (2 * P) == 0 && M % 2 == 0 && M <= (sizeof(T) == 4 ? 48 : 36);
  // register index j of lane p <-> frequency (kout) / sample P j + p (interleaved)
  static __device__ __forceinline__ constexpr int kout(int p, int j) {
    return P == 1 ? j : (j < M / 2 ? j : j + M / 2) + p * (M / 2);
  }
};

__device__ __forceinline__ float2 shfl_x16(float2 v) {
  return make_float2(__shfl_xor_sync(0xffffffffu, v.x, 16), __shfl_xor_sync(0xffffffffu, v.y, 16));
}
__device__ __forceinline__ double2 shfl_x16(double2 v) {
  return make_double2(__shfl_xor_sync(0xffffffffu, v.x, 16), __shfl_xor_sync(0xffffffffu, v.y, 16));
}
template <typename V> __device__ __forceinline__ V csel(bool c, V a, V b) {
  V r;
  r.x = c ? a.x : b.x;
  r.y = c ? a.y : b.y;
  return r;
}

// Coprime factors of R: the largest power of 2 in it (of 6 in 30) and the rest
template <int R> struct CoprimeFactor {
  static constexpr int pow2(int r) { return r % 2 ? 1 : 2 * pow2(r / 2); }
  static constexpr int v = R == 30 ? 6 : pow2(R);
  static constexpr bool split = v > 1 && v < R;
};
constexpr int inv_mod(int a, int m) {
  for (int x = 1; x < m; ++x)
    if (a * x % m == 1) return x;
  return 1;
}

// In-place DFT of R = A B elements in registers, natural order in and out, as B
// transforms of length A and A of length B without twiddles between them (the
// prime-factor algorithm of Good and Thomas: inputs B n1 + A n2, outputs by the
// Chinese remainder theorem; the permutations cost nothing in registers).  Every
// twiddle is a rounded product: against DFT<R> the coarse transforms of 20 .. 72
// points come 3-16 % closer to the exact ones, and at 20, 30, 40 and 60 only so
// as close as the shared-memory transforms were (FP32, damped bands, kinetic
// term 60: four-step 1.54e-6, DFT 1.58e-6, this 1.44e-6; Teter 40: 1.51e-7, 1.84e-7,
// 1.40e-7).
template <int R, int DIR, typename V> struct PDFT {
  static __device__ __forceinline__ void run(V* v) {
    if constexpr (!CoprimeFactor<R>::split) {
      DFT<R, DIR, V>::run(v);
    } else {
      constexpr int A = CoprimeFactor<R>::v, B = R / A;
      V t[R];
      sfor<0, B>([&](auto bI) {
        constexpr int n2 = decltype(bI)::value;
        V a_[A];
        sfor<0, A>([&](auto aI) { a_[decltype(aI)::value] = v[(B * decltype(aI)::value + A * n2) % R]; });
        PDFT<A, DIR, V>::run(a_);
        sfor<0, A>([&](auto aI) { t[decltype(aI)::value * B + n2] = a_[decltype(aI)::value]; });
      });
      constexpr int ea = B * inv_mod(B % A, A), eb = A * inv_mod(A % B, B);
      sfor<0, A>([&](auto aI) {
        constexpr int k1 = decltype(aI)::value;
        V b_[B];
        sfor<0, B>([&](auto bI) { b_[decltype(bI)::value] = t[k1 * B + decltype(bI)::value]; });
        PDFT<B, DIR, V>::run(b_);
        sfor<0, B>([&](auto bI) { v[(ea * k1 + eb * decltype(bI)::value) % R] = b_[decltype(bI)::value]; });
      });
    }
  }
};

// A twiddle left on an input of the next butterfly: w v = kap u with
// u = v + (tan or cot) i v, two FMAs instead of four products; the factor kap goes
// into the butterfly's own FMAs (the fused multiply-add butterflies of Linzer and
// Feig, 1993).
template <int R, int M_, int DIR, typename V> struct PendTw {
  using T = typename RealOf<V>::t;
  static constexpr int m = M_ % R;
  static constexpr double c = TwR<R>::c[m], s = DIR * TwR<R>::s[m];
  static constexpr bool big = (c < 0 ? -c : c) >= (s < 0 ? -s : s);
  static constexpr double kap = big ? c : s;
  static constexpr double t = big ? s / c : c / s;
  static __device__ __forceinline__ V u(V v) {
    if constexpr (big) {
      if constexpr (t == 0) return v;
      return mkc<V>(v.x - (T)t * v.y, v.y + (T)t * v.x);
    } else {
      if constexpr (t == 0) return mkc<V>(-v.y, v.x);
      return mkc<V>((T)t * v.x - v.y, (T)t * v.y + v.x);
    }
  }
};
template <typename V> __device__ __forceinline__ V cfma(typename RealOf<V>::t k, V u, V a) {
  return mkc<V>(a.x + k * u.x, a.y + k * u.y);
}

// In-place DFT of R elements in registers, natural order in and out, decimated
// in time with the twiddles folded into the radix-4, -3 and -2 butterflies:
// about 680 FP32 pipe operations at R = 48 against 800 of DFT<48>.
template <int R, int DIR, typename V> struct RDFT {
  using T = typename RealOf<V>::t;
  static constexpr int B = R <= 5 ? R : (R % 4 == 0 ? 4 : (R % 3 == 0 ? 3 : (R % 2 == 0 ? 2 : 5)));
  static constexpr int A = R / B;
  static __device__ __forceinline__ void run(V* v) {
    if constexpr (R <= 5) {
      DFT<R, DIR, V>::run(v);
    } else {
      V t[R];
      sfor<0, B>([&](auto bI) {
        constexpr int b = decltype(bI)::value;
        V a_[A];
        sfor<0, A>([&](auto aI) { a_[decltype(aI)::value] = v[B * decltype(aI)::value + b]; });
        RDFT<A, DIR, V>::run(a_);
        sfor<0, A>([&](auto aI) { t[b * A + decltype(aI)::value] = a_[decltype(aI)::value]; });
      });
      sfor<0, A>([&](auto kI) {
        constexpr int k = decltype(kI)::value;
        if constexpr (B == 4) {
          using P1 = PendTw<R, k, DIR, V>;
          using P2 = PendTw<R, 2 * k, DIR, V>;
          using P3 = PendTw<R, 3 * k, DIR, V>;
          const V u1 = P1::u(t[A + k]), u2 = P2::u(t[2 * A + k]), u3 = P3::u(t[3 * A + k]);
          const V a = cfma((T)P2::kap, u2, t[k]), b = cfma((T)-P2::kap, u2, t[k]);
          constexpr double r = P3::kap / P1::kap;
          const V s = cfma((T)r, u3, u1), d = cmuli<DIR>(cfma((T)-r, u3, u1));
          v[k] = cfma((T)P1::kap, s, a);
          v[k + 2 * A] = cfma((T)-P1::kap, s, a);
          v[k + A] = cfma((T)P1::kap, d, b);
          v[k + 3 * A] = cfma((T)-P1::kap, d, b);
        } else if constexpr (B == 3) {
          using P1 = PendTw<R, k, DIR, V>;
          using P2 = PendTw<R, 2 * k, DIR, V>;
          const V u1 = P1::u(t[A + k]), u2 = P2::u(t[2 * A + k]);
          constexpr double r = P2::kap / P1::kap;
          const V s = cfma((T)r, u2, u1), d = cmuli<DIR>(cfma((T)-r, u2, u1));
          const V h = cfma((T)(-0.5 * P1::kap), s, t[k]);
          constexpr double q = TwR<3>::s[1] * P1::kap;
          v[k] = cfma((T)P1::kap, s, t[k]);
          v[k + A] = cfma((T)q, d, h);
          v[k + 2 * A] = cfma((T)-q, d, h);
        } else if constexpr (B == 2) {
          using P1 = PendTw<R, k, DIR, V>;
          const V u1 = P1::u(t[A + k]);
          v[k] = cfma((T)P1::kap, u1, t[k]);
          v[k + A] = cfma((T)-P1::kap, u1, t[k]);
        } else {
          V c_[B];
          sfor<0, B>([&](auto bI) {
            constexpr int b = decltype(bI)::value;
            c_[b] = twmul<R, b * k, DIR>(t[b * A + k]);
          });
          DFT<B, DIR, V>::run(c_);
          sfor<0, B>([&](auto bI) { v[k + A * decltype(bI)::value] = c_[decltype(bI)::value]; });
        }
      });
    }
  }
};

// FUSE takes RDFT for the local part: 8 % faster where the FP32 / FP64 pipe binds
// (the fine planes); the memory-bound passes gain nothing from it and take PDFT,
// which is closer to the exact transform.  So do lengths with a factor of 5, whose
// radix-5 step RDFT does not fuse.
template <int R, bool FUSE, int DIR, typename V> __device__ __forceinline__ void local_dft(V* v) {
  if constexpr (FUSE && R % 5 != 0) RDFT<R, DIR, V>::run(v);
  else PDFT<R, DIR, V>::run(v);
}

template <typename T, int N, int DIR, bool FUSE = false> __device__ __forceinline__ void fft_dit(typename C2<T>::t* v, int p) {
  using V = typename C2<T>::t;
  using R = RegN<T, N>;
  local_dft<R::M, FUSE, DIR>(v);
  if constexpr (R::P == 2) {
    constexpr int H = R::M / 2;
    const bool q = p != 0;
    sfor<0, H>([&](auto jI) {
      constexpr int j = decltype(jI)::value;
      const V keep = csel(q, v[j + H], v[j]);
      const V recv = shfl_x16(csel(q, v[j], v[j + H]));
      const V e = csel(q, recv, keep);
      V o = twmul<N, j, DIR>(csel(q, keep, recv));
      o = csel(q, cmuli<DIR>(o), o);
      v[j] = cadd(e, o);
      v[j + H] = csub(e, o);
    });
  }
}

template <typename T, int N, int DIR, bool FUSE = false> __device__ __forceinline__ void fft_dif(typename C2<T>::t* v, int p) {
  using V = typename C2<T>::t;
  using R = RegN<T, N>;
  if constexpr (R::P == 2) {
    constexpr int H = R::M / 2;
    const bool q = p != 0;
    sfor<0, H>([&](auto jI) {
      constexpr int j = decltype(jI)::value;
      const V a = cadd(v[j], v[j + H]);
      V b = twmul<N, j, DIR>(csub(v[j], v[j + H]));
      b = csel(q, cmuli<DIR>(b), b);
      const V recv = shfl_x16(csel(q, a, b));
      const V keep = csel(q, b, a);
      v[j] = csel(q, recv, keep);
      v[j + H] = csel(q, keep, recv);
    });
  }
  local_dft<R::M, FUSE, DIR>(v);
}

}  // namespace pwb
