// H*psi, Teter and exchange passes with register-resident transforms
// (regfft.cuh); included by pipeline.cuh.
//
// The shared-memory passes these replace wrote and read every element three
// to nine times there and were bound by that; these are bound by HBM, the fine
// plane by the FP32 / FP64 pipe and its barriers.  Times below: Si64, 80 pairs,
// 48^3 / 96^3, before -> now.
//
// Layouts: spectra are [z][kx][ky] (ky fastest) so that both passes of a plane
// load and store whole rows with one transform per lane and one exchange
// through shared memory, and a z pencil needs none.  Slot fields are
// [zf][kx slot][ky slot].  Tables that multiply a spectrum come in the same
// order (the *_t buffers of the context).
//
// A padded transform to the fine axis (2 N points from N + 1 slots) is two
// length-N transforms: the even fine points take the coarse spectrum as it is,
// the odd ones the spectrum times e^{i pi k / N}; the "+" and "-" Nyquist
// slots share index N/2 with weights (1, 1) and (i, -i).  The way back is the
// transpose: X_k = E_k + e^{-i pi k / N} O_k.  No zero is ever loaded, stored
// or multiplied, and along z the even planes are the coarse values themselves.
#pragma once

namespace pwb {

constexpr int ceil32(int x) { return (x + 31) / 32 * 32; }
// resident CTAs per SM asked of the compiler: data registers of M complex
// elements and about 70 more
template <typename T, int M> constexpr int reg_min_ctas(int threads) {
  const int regs = M * 2 * (int)sizeof(T) / 4 + 72;
  const int n = 65536 / (regs * threads);
  return n < 1 ? 1 : (n > 8 ? 8 : n);
}

// planes per CTA of the plane kernels: the fewest whose lanes fill at least
// 93 % of whole warps, with at least 96 threads (small grids) and at most 192
template <typename T, int N0, int N1> constexpr int rplane_npl() {
  const int p = RegN<T, N0>::P > RegN<T, N1>::P ? RegN<T, N0>::P : RegN<T, N1>::P;
  const int n = N0 > N1 ? N0 : N1;
  int best = 1;
  for (int k = 1; k <= 8; ++k) {
    const int lanes = k * n * p;
    if (k > 1 && lanes > 192) break;
    best = k;
    if (lanes >= 96 && lanes * 100 >= 93 * ceil32(lanes)) break;
  }
  return best;
}
template <typename T, int N0, int N1> struct RPlane {
  using R0 = RegN<T, N0>;
  using R1 = RegN<T, N1>;
  static constexpr int NPL = rplane_npl<T, N0, N1>();
  static constexpr int PS = N0 + 1;                           // odd: rows and columns free of bank conflicts
  static constexpr int LX = (NPL * N0 + R1::CW - 1) / R1::CW * 32;   // threads of the y transforms
  static constexpr int LY = (NPL * N1 + R0::CW - 1) / R0::CW * 32;   // threads of the x transforms
  static constexpr int TH = LX > LY ? LX : LY;
  static constexpr int MINB = reg_min_ctas<T, (R0::M > R1::M ? R0::M : R1::M)>(TH);
  static constexpr size_t smem = sizeof(typename C2<T>::t) * NPL * N1 * PS;
};

// Plane forward: values -> [z][kx][ky].  MODE 0: two real bands per field,
// 1: complex bands, 2: exchange pairs psi_k (phi_ja + i phi_jb).  Bound by
// memory: one read and one write of the field, one pass through shared memory
// (FP32 62 -> 27 us, 5.2 TB/s; FP64 124 -> 49 us; exchange pairs 697 -> 248 us per
// 1213 fields, bound by the three 4-byte reads per element from L2).
struct RExx {
  int k0, ldp, j0, nphi, njp;
};
template <typename T, int N0, int N1, int MODE>
__global__ void __launch_bounds__(RPlane<T, N0, N1>::TH, RPlane<T, N0, N1>::MINB)
k_rfwd(const T* __restrict__ psi, int ld, int nband, int band0, const T* __restrict__ phi, RExx ex,
       VT<T>* __restrict__ A, int n2) {
  using V = VT<T>;
  using L = RPlane<T, N0, N1>;
  using R0 = RegN<T, N0>;
  using R1 = RegN<T, N1>;
  constexpr int PS = L::PS, NP = N0 * N1;
  extern __shared__ __align__(16) unsigned char smraw[];
  V* S = reinterpret_cast<V*>(smraw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int z0 = blockIdx.x * L::NPL, f = blockIdx.y;
  {
    const int p = R1::P == 1 ? 0 : lane >> 4;
    const int q = warp * R1::CW + (lane & (R1::CW - 1));
    const int pl = q / N0, x = q - pl * N0;
    const bool act = q < L::NPL * N0 && z0 + pl < n2;
    V v[R1::M];
    const long o = (long)(z0 + pl) * NP + R1::kout(p, 0) * N0 + x;
    if (act) {
      if constexpr (MODE == 1) {
        const V* a = reinterpret_cast<const V*>(psi) + (long)(band0 + f) * ld + o;
#pragma unroll
        for (int m = 0; m < R1::M; ++m) v[m] = a[R1::kout(0, m) * N0];
      } else if constexpr (MODE == 0) {
        const int ba = band0 + 2 * f;
        const T* a = psi + (long)ba * ld + o;
        const bool hb = ba + 1 < nband;
        const T* b = hb ? a + ld : a;
#pragma unroll
        for (int m = 0; m < R1::M; ++m) v[m] = mkc<V>(a[R1::kout(0, m) * N0], b[R1::kout(0, m) * N0]);
        if (!hb) {
#pragma unroll
          for (int m = 0; m < R1::M; ++m) v[m].y = 0;
        }
      } else {
        const int kk = f / ex.njp, ja = ex.j0 + 2 * (f - kk * ex.njp);
        const T* s = psi + (long)(ex.k0 + kk) * ld + o;
        const T* a = phi + (long)ja * ex.ldp + o;
        const bool hb = ja + 1 < ex.nphi;
        const T* b = hb ? a + ex.ldp : a;
#pragma unroll
        for (int m = 0; m < R1::M; ++m) {
          const T w = s[R1::kout(0, m) * N0];
          v[m] = mkc<V>(w * a[R1::kout(0, m) * N0], w * b[R1::kout(0, m) * N0]);
        }
        if (!hb) {
#pragma unroll
          for (int m = 0; m < R1::M; ++m) v[m].y = 0;
        }
      }
    }
    fft_dif<T, N1, -1>(v, p);
    if (act) {
      V* s = S + pl * (N1 * PS) + p * PS + x;
#pragma unroll
      for (int m = 0; m < R1::M; ++m) s[R1::P * m * PS] = v[m];
    }
  }
  __syncthreads();
  {
    const int p = R0::P == 1 ? 0 : lane >> 4;
    const int q = warp * R0::CW + (lane & (R0::CW - 1));
    const int pl = q / N1, ky = q - pl * N1;
    const bool act = q < L::NPL * N1 && z0 + pl < n2;
    V v[R0::M];
    if (act) {
      const V* s = S + (pl * N1 + ky) * PS + R0::kout(p, 0);
#pragma unroll
      for (int j = 0; j < R0::M; ++j) v[j] = s[R0::kout(0, j)];
    }
    fft_dif<T, N0, -1>(v, p);
    if (act) {
      V* a = A + ((long)f * n2 + z0 + pl) * NP + p * N1 + ky;
#pragma unroll
      for (int m = 0; m < R0::M; ++m) a[m * (R0::P * N1)] = v[m];
    }
  }
}

// Plane inverse: [z][kx][ky] -> values; CPLX as MODE 1 above (FP32 54 -> 27 us, FP64
// 120 -> 50 us)
template <typename T, int N0, int N1, bool CPLX>
__global__ void __launch_bounds__(RPlane<T, N0, N1>::TH, RPlane<T, N0, N1>::MINB)
k_rinv(const VT<T>* __restrict__ D, T* __restrict__ out, int ldo, int nband, int band0, int accumulate, int n2) {
  using V = VT<T>;
  using L = RPlane<T, N0, N1>;
  using R0 = RegN<T, N0>;
  using R1 = RegN<T, N1>;
  constexpr int PS = L::PS, NP = N0 * N1;
  extern __shared__ __align__(16) unsigned char smraw[];
  V* S = reinterpret_cast<V*>(smraw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int z0 = blockIdx.x * L::NPL, f = blockIdx.y;
  {
    const int p = R0::P == 1 ? 0 : lane >> 4;
    const int q = warp * R0::CW + (lane & (R0::CW - 1));
    const int pl = q / N1, ky = q - pl * N1;
    const bool act = q < L::NPL * N1 && z0 + pl < n2;
    V v[R0::M];
    if (act) {
      const V* a = D + ((long)f * n2 + z0 + pl) * NP + p * N1 + ky;
#pragma unroll
      for (int m = 0; m < R0::M; ++m) v[m] = a[m * (R0::P * N1)];
    }
    fft_dit<T, N0, +1>(v, p);
    if (act) {
      V* s = S + (pl * N1 + ky) * PS + R0::kout(p, 0);
#pragma unroll
      for (int j = 0; j < R0::M; ++j) s[R0::kout(0, j)] = v[j];
    }
  }
  __syncthreads();
  {
    const int p = R1::P == 1 ? 0 : lane >> 4;
    const int q = warp * R1::CW + (lane & (R1::CW - 1));
    const int pl = q / N0, x = q - pl * N0;
    const bool act = q < L::NPL * N0 && z0 + pl < n2;
    V v[R1::M];
    if (act) {
      const V* s = S + pl * (N1 * PS) + p * PS + x;
#pragma unroll
      for (int m = 0; m < R1::M; ++m) v[m] = s[m * (R1::P * PS)];
    }
    fft_dit<T, N1, +1>(v, p);
    if (act) {
      const long o = (long)(z0 + pl) * NP + R1::kout(p, 0) * N0 + x;
      if constexpr (CPLX) {
        V* oc = reinterpret_cast<V*>(out) + (long)(band0 + f) * ldo + o;
        if (accumulate) {
#pragma unroll
          for (int j = 0; j < R1::M; ++j) v[j] = cadd(v[j], oc[R1::kout(0, j) * N0]);
        }
#pragma unroll
        for (int j = 0; j < R1::M; ++j) oc[R1::kout(0, j) * N0] = v[j];
      } else {
        const int ba = band0 + 2 * f;
        T* oa = out + (long)ba * ldo + o;
        const bool hb = ba + 1 < nband;
        T* ob = oa + ldo;
        if (accumulate) {
#pragma unroll
          for (int j = 0; j < R1::M; ++j) v[j].x += oa[R1::kout(0, j) * N0];
          if (hb) {
#pragma unroll
            for (int j = 0; j < R1::M; ++j) v[j].y += ob[R1::kout(0, j) * N0];
          }
        }
#pragma unroll
        for (int j = 0; j < R1::M; ++j) oa[R1::kout(0, j) * N0] = v[j].x;
        if (hb) {
#pragma unroll
          for (int j = 0; j < R1::M; ++j) ob[R1::kout(0, j) * N0] = v[j].y;
        }
      }
    }
  }
}

// Exchange plane inverse: out_k (+)= sum_jp w_ja phi_ja Re + w_jb phi_jb Im of
// the njp fields of band k0 + blockIdx.y; each lane owns its column's sums (in
// shared memory, touched by no other lane: in registers they took 518-757 us for
// 1024 fields against 433).  1213 fields: 1128 -> 463 us, bound by the two barriers
// per field and 12 warps per SM
template <typename T, int N0, int N1>
__global__ void __launch_bounds__(RPlane<T, N0, N1>::TH, RPlane<T, N0, N1>::MINB)
k_rexx_inv(const VT<T>* __restrict__ A, const T* __restrict__ phi, RExx ex, const T* __restrict__ wj,
           T* __restrict__ out, int ldo, int accumulate, int n2) {
  using V = VT<T>;
  using L = RPlane<T, N0, N1>;
  using R0 = RegN<T, N0>;
  using R1 = RegN<T, N1>;
  constexpr int PS = L::PS, NP = N0 * N1;
  extern __shared__ __align__(16) unsigned char smraw[];
  V* S = reinterpret_cast<V*>(smraw);
  T* acc = reinterpret_cast<T*>(smraw + L::smem) + threadIdx.x;   // [M][TH]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int z0 = blockIdx.x * L::NPL, kk = blockIdx.y;
#pragma unroll
  for (int j = 0; j < R1::M; ++j) acc[j * L::TH] = 0;
  const int p0 = R0::P == 1 ? 0 : lane >> 4, p1 = R1::P == 1 ? 0 : lane >> 4;
  const int q0 = warp * R0::CW + (lane & (R0::CW - 1)), q1 = warp * R1::CW + (lane & (R1::CW - 1));
  const int pla = q0 / N1, ky = q0 - pla * N1, plb = q1 / N0, x = q1 - plb * N0;
  const bool acta = q0 < L::NPL * N1 && z0 + pla < n2, actb = q1 < L::NPL * N0 && z0 + plb < n2;
  const long o = (long)(z0 + plb) * NP + R1::kout(p1, 0) * N0 + x;
  for (int jp = 0; jp < ex.njp; ++jp) {
    V v[R0::M > R1::M ? R0::M : R1::M];
    if (acta) {
      const V* a = A + ((long)(kk * ex.njp + jp) * n2 + z0 + pla) * NP + p0 * N1 + ky;
#pragma unroll
      for (int m = 0; m < R0::M; ++m) v[m] = a[m * (R0::P * N1)];
    }
    fft_dit<T, N0, +1>(v, p0);
    __syncthreads();
    if (acta) {
      V* s = S + (pla * N1 + ky) * PS + R0::kout(p0, 0);
#pragma unroll
      for (int j = 0; j < R0::M; ++j) s[R0::kout(0, j)] = v[j];
    }
    __syncthreads();
    if (actb) {
      const V* s = S + plb * (N1 * PS) + p1 * PS + x;
#pragma unroll
      for (int m = 0; m < R1::M; ++m) v[m] = s[m * (R1::P * PS)];
    }
    fft_dit<T, N1, +1>(v, p1);
    if (actb) {
      const int ja = ex.j0 + 2 * jp;
      const bool hb = ja + 1 < ex.nphi;
      const T wa = wj[ja], wb = hb ? wj[ja + 1] : (T)0;
      const T* pa = phi + (long)ja * ex.ldp + o;
      const T* pb = hb ? pa + ex.ldp : pa;
#pragma unroll
      for (int j = 0; j < R1::M; ++j)
        acc[j * L::TH] += wa * pa[R1::kout(0, j) * N0] * v[j].x + wb * pb[R1::kout(0, j) * N0] * v[j].y;
    }
  }
  if (actb) {
    T* oc = out + (long)(ex.k0 + kk) * ldo + o;
#pragma unroll
    for (int j = 0; j < R1::M; ++j) {
      const T s = acc[j * L::TH];
      oc[R1::kout(0, j) * N0] = accumulate ? oc[R1::kout(0, j) * N0] + s : s;
    }
  }
}

// z pencils: one transform per lane (pair), columns (kx, ky) across lanes; no
// shared memory
template <typename T, int NZ> struct RPencil {
  using R = RegN<T, NZ>;
  static constexpr int TH = 96;
  static constexpr int COLS = TH / R::P;
  static constexpr int MINB = reg_min_ctas<T, R::M>(TH);
  // the padding pencils keep three streams of addresses as well: registers
  // before residency (48, 80 pairs: 168 registers and spills 69 us, 210 60 us;
  // FP64 124 -> 102 us)
  static constexpr int THP = 128;
  static constexpr int COLSP = THP / R::P;
  static constexpr int MINBP = R::M * (int)sizeof(T) >= 144 ? 2 : reg_min_ctas<T, R::M>(THP);
};

// Teter / exchange kernel: FFT z, * table / N_c, IFFT z, in place: one read and one
// write of the field (1213 fields of 48^3: 1107 -> 288 us, 7.4 TB/s).  The plane
// size is a template argument: with a run-time stride the 48 addresses shared
// by loads and stores stay live and spill (54 us instead of 21 for 80 fields).
template <typename T, int N0, int N1, int NZ>
__global__ void __launch_bounds__(RPencil<T, NZ>::TH, RPencil<T, NZ>::MINB)
k_rzmul(VT<T>* __restrict__ A, const T* __restrict__ tab, T inv_nc) {
  using V = VT<T>;
  using R = RegN<T, NZ>;
  constexpr int np = N0 * N1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int p = R::P == 1 ? 0 : lane >> 4;
  const int t = blockIdx.x * RPencil<T, NZ>::COLS + warp * R::CW + (lane & (R::CW - 1));
  const bool act = t < np;
  V v[R::M];
  V* a = A + (long)blockIdx.y * NZ * np + (long)R::kout(p, 0) * np + t;
  if (act) {
#pragma unroll
    for (int j = 0; j < R::M; ++j) v[j] = a[(long)R::kout(0, j) * np];
  }
  fft_dif<T, NZ, -1>(v, p);
  if (act) {
    const T* tb = tab + (long)p * np + t;
#pragma unroll
    for (int m = 0; m < R::M; ++m) v[m] = cscale(v[m], tb[(long)(R::P * m) * np] * inv_nc);
  }
  fft_dit<T, NZ, +1>(v, p);
  if (act) {
#pragma unroll
    for (int j = 0; j < R::M; ++j) a[(long)R::kout(0, j) * np] = v[j];
  }
}

// e^{DIR i pi k / N} v for the signed frequency k of index s (s <= N/2: s,
// else s - N): literals for one lane, the table twf[m] = e^{-2 pi i m / 2N} for two
template <int N, int s, int DIR, typename V> __device__ __forceinline__ V half_shift(V v) {
  constexpr int k = s <= N / 2 ? s : s + N;      // (s - N) mod 2N
  return twmul<2 * N, k, DIR>(v);
}
template <int N, int DIR, typename V> __device__ __forceinline__ V half_shift_tab(V v, int s, const V* twf) {
  V w = twf[s <= N / 2 ? s : s + N];
  if (DIR > 0) w.y = -w.y;
  return cmul(v, w);
}
// an interleaved spectrum shifted by half a fine point; the Nyquist element
// (register M / 2 of lane 0) is left alone
template <typename T, int N, int DIR>
__device__ __forceinline__ void half_shift_all(typename C2<T>::t* v, int p, const typename C2<T>::t* twf) {
  using R = RegN<T, N>;
  if constexpr (R::P == 1) {
    sfor<1, N>([&](auto sI) {
      constexpr int s = decltype(sI)::value;
      if constexpr (s != N / 2) v[s] = half_shift<N, s, DIR>(v[s]);
    });
  } else {
#pragma unroll
    for (int j = 0; j < R::M; ++j) {
      const int s = R::P * j + p;
      const auto w = half_shift_tab<N, DIR>(v[j], s, twf);
      v[j] = (j == R::M / 2 && p == 0) ? v[j] : w;
    }
  }
}

// z pencils up: coarse FFT z, kinetic term -> K, fine z values of the "+" (and,
// on Nyquist rows and columns, "-") slots -> B.  The even fine planes are the
// coarse values themselves, so the pencil costs two transforms of length NZ
// (FP32 141 -> 60 us for 289 MB, FP64 285 -> 102 us; bound by the 96 strided stores
// of each lane).  Slot rows stay N1 + 1 long: lanes run over row ends, and rows
// padded to whole sectors were slower (72 us).
template <typename T, int N0, int N1, int NZ>
__global__ void __launch_bounds__(RPencil<T, NZ>::THP, RPencil<T, NZ>::MINBP)
k_rzpad(const VT<T>* __restrict__ A, VT<T>* __restrict__ K, VT<T>* __restrict__ B, const T* __restrict__ ekin,
        T inv_nc, const VT<T>* __restrict__ twf, int cplx, int kf0, int fpk, long kstride) {
  using V = VT<T>;
  using R = RegN<T, NZ>;
  constexpr int np = N0 * N1, ns = N1 + 1, sp = (N0 + 1) * (N1 + 1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int p = R::P == 1 ? 0 : lane >> 4;
  const int t = blockIdx.x * RPencil<T, NZ>::COLSP + warp * R::CW + (lane & (R::CW - 1));
  const int f = blockIdx.y;
  const bool act = t < np;
  const int kx = t / N1, ky = t - kx * N1;
  const bool split = !cplx && (kx == N0 / 2 || ky == N1 / 2);
  const int kxm = kx == N0 / 2 ? N0 : kx, kym = ky == N1 / 2 ? N1 : ky;
  const int zp = R::kout(p, 0);     // lane's first plane
  V v[R::M];
  V* bp = B + (long)f * (2 * NZ) * sp + kx * ns + ky;
  V* bm = B + (long)f * (2 * NZ) * sp + kxm * ns + kym;
  const bool corner = kx == N0 / 2 && ky == N1 / 2;
  if (act) {
    const V* a = A + (long)f * NZ * np + (long)R::kout(p, 0) * np + t;
#pragma unroll
    for (int j = 0; j < R::M; ++j) v[j] = cscale(a[(long)R::kout(0, j) * np], inv_nc);
    const T se = split ? (T)NZ * (T)0.5 : (T)NZ;
#pragma unroll
    for (int j = 0; j < R::M; ++j) bp[(long)(2 * (R::kout(0, j) + zp)) * sp] = cscale(v[j], se);
    if (split) {
#pragma unroll
      for (int j = 0; j < R::M; ++j) bm[(long)(2 * (R::kout(0, j) + zp)) * sp] = cscale(v[j], se);
    }
  }
  fft_dif<T, NZ, -1>(v, p);
  if (act && K) {
    // k-point batches: field kf0 + f belongs to k-point (kf0 + f) / fpk
    const T* ek = ekin + (long)((kf0 + f) / fpk) * kstride + (long)p * np + t;
    V* kp = K + (long)f * NZ * np + (long)p * np + t;
#pragma unroll
    for (int m = 0; m < R::M; ++m)
      kp[(long)(R::P * m) * np] = cscale(v[m], ek[(long)(R::P * m) * np]);
  }
  half_shift_all<T, NZ, +1>(v, p, twf);
  // Nyquist along z: i X_h / 2 at "+" and -i X_h / 2 at "-" cancel on plain
  // columns, go to one slot each on split ones; complex bands take "+" only
  V nq = cmuli<+1>(v[R::M / 2]);
  if (p == 0) v[R::M / 2] = cplx ? nq : mkc<V>(0, 0);
  nq = split ? cscale(nq, (T)0.5) : mkc<V>(0, 0);
  if constexpr (R::P == 2) nq = csel(p != 0, shfl_x16(nq), nq);
  fft_dit<T, NZ, +1>(v, p);
  if (act) {
    if (!split) {
#pragma unroll
      for (int j = 0; j < R::M; ++j) bp[(long)(2 * (R::kout(0, j) + zp) + 1) * sp] = v[j];
      if (cplx && (kx == N0 / 2 || ky == N1 / 2)) {
        // complex bands leave the "-" slots empty
#pragma unroll 4
        for (int m = 0; m < 2 * R::M; ++m) bm[(long)(R::P * m + p) * sp] = mkc<V>(0, 0);
      }
    } else {
#pragma unroll
      for (int j = 0; j < R::M; ++j) {
        const int z = R::kout(0, j) + zp;
        const V h = cscale(v[j], (T)0.5), s = cscale(nq, (z & 1) ? (T)-1 : (T)1);
        bp[(long)(2 * z + 1) * sp] = cadd(h, s);
        bm[(long)(2 * z + 1) * sp] = csub(h, s);
      }
    }
    if (corner) {
      // the two mixed corner slots that no coefficient reaches
      V* c0 = B + (long)f * (2 * NZ) * sp + (long)p * sp;
#pragma unroll 4
      for (int m = 0; m < 2 * R::M; ++m) {
        c0[(long)(R::P * m) * sp + N0 * ns + N1 / 2] = mkc<V>(0, 0);
        c0[(long)(R::P * m) * sp + (N0 / 2) * ns + N1] = mkc<V>(0, 0);
      }
    }
  }
}

// z pencils down: fold the fine z planes of the slots onto the coarse spectrum
// (IP_f2c), add the kinetic term, inverse FFT z.  The even planes enter the
// result as they are unless the cut-off mask needs their spectrum too (FP32 133 ->
// 53 us, with the mask 62 us; FP64 265 -> 95 us; bound by memory).
template <typename T, int N0, int N1, int NZ, bool MASK>
__global__ void __launch_bounds__(RPencil<T, NZ>::TH, RPencil<T, NZ>::MINB)
k_rzfold(const VT<T>* __restrict__ C, const VT<T>* __restrict__ K, VT<T>* __restrict__ D,
         const VT<T>* __restrict__ twf, int cplx, const T* __restrict__ mask) {
  using V = VT<T>;
  using R = RegN<T, NZ>;
  constexpr int np = N0 * N1, ns = N1 + 1, sp = (N0 + 1) * (N1 + 1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int p = R::P == 1 ? 0 : lane >> 4;
  const int t = blockIdx.x * RPencil<T, NZ>::COLS + warp * R::CW + (lane & (R::CW - 1));
  const int f = blockIdx.y;
  const bool act = t < np;
  const int kx = t / N1, ky = t - kx * N1;
  const bool split = !cplx && (kx == N0 / 2 || ky == N1 / 2);
  const int kxm = kx == N0 / 2 ? N0 : kx, kym = ky == N1 / 2 ? N1 : ky;
  const V* cp = C + (long)f * (2 * NZ) * sp + kx * ns + ky;
  const V* cm = C + (long)f * (2 * NZ) * sp + kxm * ns + kym;
  const int zp = R::kout(p, 0);
  V v[R::M];
  V nq = mkc<V>(0, 0);
  if (act) {
#pragma unroll
    for (int j = 0; j < R::M; ++j) v[j] = cp[(long)(2 * (R::kout(0, j) + zp) + 1) * sp];
    if (split) {
      // (O+ + O-) / 2 everywhere; the z Nyquist takes -i / 2 (O+ - O-)
#pragma unroll
      for (int j = 0; j < R::M; ++j) {
        const int z = R::kout(0, j) + zp;
        const V o = cm[(long)(2 * z + 1) * sp];
        const V d = csub(v[j], o);
        nq = (z & 1) ? csub(nq, d) : cadd(nq, d);
        v[j] = cscale(cadd(v[j], o), (T)0.5);
      }
    }
  }
  if constexpr (R::P == 2) nq = cadd(nq, shfl_x16(nq));
  fft_dif<T, NZ, -1>(v, p);
  half_shift_all<T, NZ, -1>(v, p, twf);
  if (p == 0) v[R::M / 2] = cplx ? cmuli<-1>(v[R::M / 2]) : cscale(cmuli<-1>(nq), (T)0.5);
  if (act) {
    if (K) {
      const V* kp = K + (long)f * NZ * np + (long)p * np + t;
#pragma unroll
      for (int m = 0; m < R::M; ++m) v[m] = cadd(v[m], kp[(long)(R::P * m) * np]);
    }
  }
  fft_dit<T, NZ, +1>(v, p);
  if (act) {
#pragma unroll
    for (int j = 0; j < R::M; ++j) {
      const int z = R::kout(0, j) + zp;
      V e = cp[(long)(2 * z) * sp];
      if (split) e = cscale(cadd(e, cm[(long)(2 * z) * sp]), (T)0.5);
      // the even planes' share of the spectrum, returned by the inverse NZ-fold
      v[j] = mkc<V>(v[j].x + (T)NZ * e.x, v[j].y + (T)NZ * e.y);
    }
  }
  if constexpr (MASK) {
    fft_dif<T, NZ, -1>(v, p);
    if (act) {
      const T* mk = mask + (long)p * np + t;
#pragma unroll
      for (int m = 0; m < R::M; ++m) v[m] = cscale(v[m], mk[(long)(R::P * m) * np] * (T)(1.0 / NZ));
    }
    fft_dit<T, NZ, +1>(v, p);
  }
  if (act) {
    V* d = D + (long)f * NZ * np + (long)zp * np + t;
#pragma unroll
    for (int j = 0; j < R::M; ++j) d[(long)R::kout(0, j) * np] = v[j];
  }
}

// ---------------------------------------------------------------------------
// Fine plane: slots -> fine values, * V_loc, -> slots, in place.  Axis A (the
// slow slot index, coarse length NA) is transformed by lanes walking the slots
// of axis B, then axis B by lanes walking the 2 NA fine points of A (V rows and
// shared-memory columns both run along the lanes).  Even and odd fine points
// are separate tasks of the two halves of the CTA; on the way back the halves
// swap one half of their outputs through shared memory and add.
// Shared memory per plane: 2 NA (NB + 1) elements written and read about three
// times, against nine in k_floc2.  FP32 280 -> 234 us, FP64 617 -> 508 us, 144 x 144
// planes (80 pairs, FP32) 1326 -> 1021 us: the FP32 pipe is busy 48 % of the time
// (12 warps of 158 registers; barriers are the first stall, the instruction
// cache the next: the four transforms are about 50 KB of code).  Slower: packed
// two-value FP32 instructions (244-274 us: register moves), one shared copy of the
// transform in a loop (255-272), 96 or 128 threads (263, 260), 128 registers (272).
// ---------------------------------------------------------------------------
template <typename T, int NA, int NB> struct RFine {
  using RA = RegN<T, NA>;
  using RB = RegN<T, NB>;
  static constexpr int PM = RA::P > RB::P ? RA::P : RB::P;
  static constexpr int PS = NB + 1;
  static constexpr size_t smem = sizeof(typename C2<T>::t) * (2 * NA * PS + (PM > 1 ? 2 * NA + 2 * NB : 0));
  // threads: all 2 x 2 NA rows of a plane in one pass where that takes at most
  // 320 lanes, else in the fewest equal passes of at most 320 (80 pairs, 192 / 256
  // / 320 threads: FP32 72 1080 / 1178 / 1021 us, 60 - / 552 / 680, FP64 36 252 / 283
  // / 242, 48 512 / 554 / 976); planes that leave room for one CTA only take 384
  // (FP64 60, 40 pairs: 256 threads 897 us, 384 737)
  static constexpr int LANES = 4 * NA * RB::P, NPASS = (LANES + 319) / 320;
  static constexpr bool ALONE = 2 * (smem + 1024) > 227 * 1024;
  static constexpr int TH = PM == 1 ? ceil32(4 * NA) : (ALONE ? 384 : (LANES / NPASS + 63) / 64 * 64);
  // FP32: only the two warps that share rows wait for one another (48: 239 ->
  // 234 us on 80 pairs of 96 x 96); FP64 stays in step (506, with pairs 551 us)
  static constexpr bool PAIR = sizeof(T) == 4 && TH % 64 == 0;
  static constexpr int CPP = TH / (2 * RA::P);   // columns (slots of B) per pass
  static constexpr int RPP = TH / (2 * RB::P);   // rows (fine points of A) per pass
  // one lane per row: 48 registers beside the data are enough (40: three CTAs
  // instead of two, 164 -> 141 us on 80 pairs)
  static constexpr int REGS = (RA::M > RB::M ? RA::M : RB::M) * 2 * (int)sizeof(T) / 4 + 48;
  static constexpr int MINB = PM == 2 ? (ALONE ? 1 : 2) : (65536 / (REGS * TH) < 1 ? 1 : 65536 / (REGS * TH));
};

__device__ __forceinline__ void bar_pair(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

// the halves' exchange: par 0 finishes the registers below M / 2, par 1 those
// from M / 2 on; S(j) is the shared element of register j, out(j, X) receives the sum
// and nyq(X+, X-) the two Nyquist slots
template <typename R, typename V, typename SY, typename SF, typename OF, typename NF>
__device__ __forceinline__ void fold_halves(V* v, int p, int par, bool act, SY&& sync, SF&& S, OF&& out, NF&& nyq) {
  constexpr int H = R::M / 2;
  sync();
  if (act) {
    if (par == 0) {
#pragma unroll
      for (int j = H; j < R::M; ++j) *S(j) = v[j];
    } else {
#pragma unroll
      for (int j = 0; j < H; ++j) *S(j) = v[j];
    }
  }
  sync();
  if (act) {
    if (par == 0) {
#pragma unroll
      for (int j = 0; j < H; ++j) out(j, cadd(v[j], *S(j)));
    } else {
      const V e = *S(H);
      if (p == 0) nyq(cadd(e, cmuli<-1>(v[H])), cadd(e, cmuli<+1>(v[H])));
      else out(H, cadd(v[H], e));
#pragma unroll
      for (int j = H + 1; j < R::M; ++j) out(j, cadd(v[j], *S(j)));
    }
  }
}

template <typename T, int NA, int NB>
__global__ void __launch_bounds__(RFine<T, NA, NB>::TH, RFine<T, NA, NB>::MINB)
k_rfloc(VT<T>* __restrict__ BC, const T* __restrict__ vt, T inv_nf, const VT<T>* __restrict__ twa_g,
        const VT<T>* __restrict__ twb_g) {
  using V = VT<T>;
  using L = RFine<T, NA, NB>;
  using RA = RegN<T, NA>;
  using RB = RegN<T, NB>;
  constexpr int PS = L::PS, ns = NB + 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  V* S = reinterpret_cast<V*>(smraw);
  V* twa = S + 2 * NA * PS;
  V* twb = twa + 2 * NA;
  if constexpr (L::PM > 1) {
    load_tw(twa, twa_g, 2 * NA);
    load_tw(twb, twb_g, 2 * NB);
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int zf = blockIdx.x;
  V* Bp = BC + ((long)blockIdx.y * gridDim.x + zf) * ((NA + 1) * ns);
  const int pa = RA::P == 1 ? 0 : lane >> 4, pb = RB::P == 1 ? 0 : lane >> 4;
  const int ua = warp * RA::CW + (lane & (RA::CW - 1)), ub = warp * RB::CW + (lane & (RB::CW - 1));
  const int parb = ub >= L::RPP, rb = ub - parb * L::RPP;
  // warps w and w + TH / 64 hold the two parities of the same rows or columns
  auto sync = [&] {
    if constexpr (L::PAIR) bar_pair(1 + (warp < L::TH / 64 ? warp : warp - L::TH / 64));
    else __syncthreads();
  };

  // A up
  for (int c0 = 0; c0 < ns; c0 += L::CPP) {
    // the last pass packs its few columns of both parities into the first warps
    const int nc = L::PAIR ? L::CPP : min(L::CPP, ns - c0);
    const int para = ua >= nc, c = c0 + ua - para * nc;
    const bool act = ua < 2 * nc && c < ns;
    if (RA::P == 1 ? !act : !__any_sync(0xffffffffu, act)) continue;
    V v[RA::M];
    if (act) {
#pragma unroll
      for (int m = 0; m < RA::M; ++m) v[m] = Bp[(RA::P * m + pa) * ns + c];
      if (pa == 0) {
        const V h = v[RA::M / 2], n = Bp[NA * ns + c];
        v[RA::M / 2] = para ? cmuli<+1>(csub(h, n)) : cadd(h, n);
      }
    }
    if (para) half_shift_all<T, NA, +1>(v, pa, twa);
    fft_dit<T, NA, +1, true>(v, pa);
    if (act) {
      V* s = S + (2 * RA::kout(pa, 0) + para) * PS + c;
#pragma unroll
      for (int j = 0; j < RA::M; ++j) s[2 * RA::kout(0, j) * PS] = v[j];
    }
  }
  __syncthreads();

  // B up, * V, B down
  const T* vz = vt + (long)zf * (4 * NA * NB);
  for (int r0 = 0; r0 < 2 * NA; r0 += L::RPP) {
    const int r = r0 + rb;
    const bool act = rb < L::RPP && r < 2 * NA;
    V v[RB::M];
    V* srow = S + r * PS;
    if (act) {
#pragma unroll
      for (int m = 0; m < RB::M; ++m) v[m] = srow[RB::P * m + pb];
      if (pb == 0) {
        const V h = v[RB::M / 2], n = srow[NB];
        v[RB::M / 2] = parb ? cmuli<+1>(csub(h, n)) : cadd(h, n);
      }
    }
    if (parb) half_shift_all<T, NB, +1>(v, pb, twb);
    fft_dit<T, NB, +1, true>(v, pb);
    if (act) {
      const T* vr = vz + (long)(2 * RB::kout(pb, 0) + parb) * (2 * NA) + r;
#pragma unroll
      for (int j = 0; j < RB::M; ++j) v[j] = cscale(v[j], vr[2 * RB::kout(0, j) * (2 * NA)]);
    }
    fft_dif<T, NB, -1, true>(v, pb);
    if (parb) half_shift_all<T, NB, -1>(v, pb, twb);
    fold_halves<RB>(v, pb, parb, act, sync, [&](int j) { return srow + RB::P * j + pb; },
                    [&](int j, V x) { srow[RB::P * j + pb] = x; },
                    [&](V xp, V xm) { srow[NB / 2] = xp; srow[NB] = xm; });
  }
  __syncthreads();

  // A down
  for (int c0 = 0; c0 < ns; c0 += L::CPP) {
    const int nc = L::PAIR ? L::CPP : min(L::CPP, ns - c0);
    const int para = ua >= nc, c = c0 + ua - para * nc;
    const bool act = ua < 2 * nc && c < ns;
    V v[RA::M];
    V* scol = S + c;
    if (RA::P == 1 ? act : __any_sync(0xffffffffu, act)) {
      if (act) {
        const V* s = scol + (2 * RA::kout(pa, 0) + para) * PS;
#pragma unroll
        for (int j = 0; j < RA::M; ++j) v[j] = s[2 * RA::kout(0, j) * PS];
      }
      fft_dif<T, NA, -1, true>(v, pa);
      if (para) half_shift_all<T, NA, -1>(v, pa, twa);
    }
    V* bc = Bp + c;
    fold_halves<RA>(v, pa, para, act, sync, [&](int j) { return scol + (RA::P * j + pa) * PS; },
                    [&](int j, V x) { bc[(RA::P * j + pa) * ns] = cscale(x, inv_nf); },
                    [&](V xp, V xm) {
                      bc[(NA / 2) * ns] = cscale(xp, inv_nf);
                      bc[NA * ns] = cscale(xm, inv_nf);
                    });
  }
}

}  // namespace pwb
