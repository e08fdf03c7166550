// In-register radix-R DFTs and a Stockham autosort engine for batched length-N complex FFTs.
//
// Thread model: one FFT of length N is computed by NT = N / E cooperating threads, each holding
// E elements.  The first stage is radix E (one butterfly per thread); later stages are radix E
// except a shorter last one (N need not be a power of E).  Between stages the threads exchange
// through a caller-provided shared-memory column (element p at sbuf[p * sstride]).
//
// Register contract of fft_run():
//   on entry  a[m] = x[j + NT*m]      (m = 0..E-1, j = this thread's index within the FFT)
//   on return a[m] = X[j + NT*m]      (same positions, transformed)
// so a thread's outputs sit at exactly the positions of its inputs; a forward transform can be
// chained after an inverse one with no exchange in between.
//
// Twiddles for stages >= 1 come from a table tw[p] = exp(-2 pi i p / N), p < N, computed on the
// host in FP64 (and rounded once to the element type), read directly, or through a copy in the
// thread's own order: registers (TwRegs) or shared memory (TwLane).  The radix-R butterflies use
// the exact constants cos(2 pi m / 16), sin(2 pi m / 16).
//
// The other lengths N = 12 R2 R3 (360 = 12 5 6, 384 = 12 8 4, 192 = 12 4 4, 96 = 12 4 2) take
// twelve elements per thread and three in-place stages with two exchanges (fft_run_12).
#pragma once
#include <cmath>
#include <type_traits>

#include "ld_common.cuh"

namespace ld {

__host__ __device__ constexpr int ipow(int b, int e) { return e == 0 ? 1 : b * ipow(b, e - 1); }
__host__ __device__ constexpr int nstages(int n, int e) { return n <= e ? 1 : 1 + nstages(n / e, e); }

template <int N, int E> struct FftShape {
  static_assert((N & (N - 1)) == 0 && (E & (E - 1)) == 0, "powers of two only");
  static_assert(E >= 2 && E <= 16 && E <= N, "radix 2..16");
  static constexpr int NT = N / E;
  static constexpr int S = nstages(N, E);
  static constexpr int RL = N / ipow(E, S - 1);  // radix of the last stage
  static __host__ __device__ constexpr int radix(int s) { return s < S - 1 ? E : RL; }
  static __host__ __device__ constexpr int ns(int s) { return ipow(E, s); }
};

// W_16^m, W_16 = exp(-2 pi i / 16): W = c2 (1 -+ i) for even m, c1 (+-1 -+ i t) or c1 (+-t -+ i) for odd
// m, with c2 = cos(pi/4), c1 = cos(pi/8), t = tan(pi/8), s1 = c1 t.
template <typename T> struct W16 {
  static constexpr double C1 = 0.92387953251128675613;
  static constexpr T c1 = T(C1), s1 = T(0.38268343236508977173), t = T(0.41421356237309504880),
                     c2 = T(0.70710678118654752440);
  // c1 rounded to FP32 is almost as far off as a rounded number can be (3.1e-8), in every second
  // butterfly of the radix-16 steps, so rows of 128 = 16 x 8 and 256 = 16 x 16 add its remainder l1
  // (EXACT below).  Error against 64 bits of a right-hand side at 256^3 / 128^3: 4.56e-7 / 3.55e-7 without
  // it and without the fused products, 4.27e-7 / 3.38e-7 now, 4.40e-7 / 3.50e-7 with rows of 8 x 8 x 4 and
  // 8 x 8 x 2; time 363 -> 365 us and 58.8 -> 59.1 us.  In the columns too: 3.92e-7, 367 us.
  static constexpr T l1 = T(C1 - double(T(C1)));
  static constexpr bool exact(int n, int e, bool row) { return sizeof(T) == 4 && row && e == 16 && n <= 256; }
};

// q W_16^m for m = 0..7 (INV: by its conjugate)
template <typename T, bool INV> __device__ __forceinline__ cplx<T> w16mul(cplx<T> x, int m) {
  using W = W16<T>;
  constexpr T c1 = W::c1, s1 = W::s1, c2 = W::c2;
  const T sg = INV ? T(1) : T(-1);  // sign of the sine part
  switch (m) {
    case 0: return x;
    case 4: return INV ? cmk(-x.y, x.x) : cmk(x.y, -x.x);  // * (+-i)
    case 2: { T a = x.x, b = x.y;                            // * c2 (1 -+ i)
      return INV ? cmk(c2 * (a - b), c2 * (a + b)) : cmk(c2 * (a + b), c2 * (b - a)); }
    case 6: { T a = x.x, b = x.y;                            // * c2 (-1 -+ i)
      return INV ? cmk(-c2 * (a + b), c2 * (a - b)) : cmk(c2 * (b - a), -c2 * (a + b)); }
    default: {
      T wr, wi;
      switch (m) {
        case 1: wr = c1;  wi = s1; break;
        case 3: wr = s1;  wi = c1; break;
        case 5: wr = -s1; wi = c1; break;
        default: wr = -c1; wi = s1; break;  // m == 7
      }
      wi *= sg;
      return cmk(x.x * wr - x.y * wi, x.x * wi + x.y * wr);
    }
  }
}

// The odd products: W v = c1 (ka a, kb b).
template <bool INV> struct OddW16 {
  static constexpr float sg = INV ? -1.f : 1.f, st = sg * W16<float>::t;
  float ta, ka, kb;
  bool xy;  // a = v.x + ta v.y, b = v.y - ta v.x; else a = v.y + ta v.x, b = v.x - ta v.y
  __device__ __forceinline__ explicit OddW16(int m)
      : ta(m == 1 || m == 3 ? st : -st), ka(m == 1 ? 1.f : (m == 7 ? -1.f : sg)),
        kb(m == 1 ? 1.f : (m == 7 ? -1.f : -sg)), xy(m == 1 || m == 7) {}
};

// Butterfly p, q <- p +- q W_16^m.  FP32: the products accumulated onto p by fused multiply-adds, six
// operations for an odd m (ten with EXACT) instead of eight with the product rounded first.  FP64 keeps
// the plain form: the fused one has a longer chain (one field forward at 128^3 24.4 -> 25.6 us).
template <typename T, bool INV, bool EXACT> __device__ __forceinline__ void butterfly(cplx<T>& p, cplx<T>& q, int m) {
  using W = W16<T>;
  const cplx<T> u = p, v = q;
  if (sizeof(T) == 8 || m == 0 || m == 4) {
    const cplx<T> w = w16mul<T, INV>(v, m);
    p = cadd(u, w);
    q = csub(u, w);
  } else if (m == 2 || m == 6) {
    const T s = v.x + v.y, d = v.x - v.y;
    // W^2 v = c2 (s, -d) forward, c2 (d, s) inverse; W^6 v = c2 (-d, -s) forward, c2 (-s, d) inverse
    const T a = m == 2 ? (INV ? d : s) : (INV ? s : d), b = m == 2 ? (INV ? s : d) : (INV ? d : s);
    const T ka = m == 2 ? W::c2 : -W::c2, kb = INV ? W::c2 : -W::c2;
    p = cmk(std::fma(a, ka, u.x), std::fma(b, kb, u.y));
    q = cmk(std::fma(a, -ka, u.x), std::fma(b, -kb, u.y));
  } else {
    const OddW16<INV> o(m);
    const T ta = o.ta, ka = o.ka, kb = o.kb;
    const T a = o.xy ? std::fma(v.y, ta, v.x) : std::fma(v.x, ta, v.y);
    const T b = o.xy ? std::fma(v.x, -ta, v.y) : std::fma(v.y, -ta, v.x);
    cplx<T> up = u, uq = u;
    if constexpr (EXACT) {
      up = cmk(std::fma(a, ka * W::l1, u.x), std::fma(b, kb * W::l1, u.y));
      uq = cmk(std::fma(a, -ka * W::l1, u.x), std::fma(b, -kb * W::l1, u.y));
    }
    p = cmk(std::fma(a, ka * W::c1, up.x), std::fma(b, kb * W::c1, up.y));
    q = cmk(std::fma(a, -ka * W::c1, uq.x), std::fma(b, -kb * W::c1, uq.y));
  }
}

__host__ __device__ constexpr int bitrev(int i, int bits) {
  return bits == 0 ? 0 : ((i & 1) << (bits - 1)) | bitrev(i >> 1, bits - 1);
}
__host__ __device__ constexpr int ilog2(int n) { return n <= 1 ? 0 : 1 + ilog2(n / 2); }

// One radix-2 pass (butterfly span LEN) of an in-place length-R DIT DFT, then the next pass.
// LEN is a template constant so every loop has a compile-time trip count and every index into
// a[] is static: the array stays in registers.
template <typename T, int R, int LEN, bool INV, bool EXACT> __device__ __forceinline__ void dft_pass(cplx<T>* a) {
  if constexpr (LEN <= R) {
#pragma unroll
    for (int i = 0; i < R; i += LEN) {
#pragma unroll
      for (int q = 0; q < LEN / 2; ++q) {
        butterfly<T, INV, EXACT>(a[i + q], a[i + q + LEN / 2], q * (16 / LEN));
      }
    }
    dft_pass<T, R, 2 * LEN, INV, EXACT>(a);
  }
}

// Bit-reversal permutation of a[0..R-1], one compile-time swap at a time.
template <typename T, int R, int I> __device__ __forceinline__ void bitrev_swaps(cplx<T>* a) {
  if constexpr (I < R) {
    constexpr int K = bitrev(I, ilog2(R));
    if constexpr (K > I) {
      const cplx<T> t = a[I];
      a[I] = a[K];
      a[K] = t;
    }
    bitrev_swaps<T, R, I + 1>(a);
  }
}

// In-place length-R DFT of a[0..R-1] (natural order in and out), R in {1,2,4,8,16}.
template <typename T, int R, bool INV, bool EXACT = false> __device__ __forceinline__ void dft(cplx<T>* a) {
  if constexpr (R > 1) {
    bitrev_swaps<T, R, 0>(a);
    dft_pass<T, R, 2, INV, EXACT>(a);
  }
}

// Twiddle exp(-+2 pi i p / N) from the FP64-built table.
template <typename T, bool INV> __device__ __forceinline__ cplx<T> twid(const cplx<T>* tw, int p) {
  cplx<T> w = tw[p];
  if (INV) w.y = -w.y;
  return w;
}

// Barrier kinds for the exchanges.
// Each barrier is bracketed by compiler memory clobbers so that no shared-memory access of the
// exchange is moved across it.
struct SyncBlock {
  __device__ __forceinline__ void operator()() const {
    asm volatile("" ::: "memory");
    __syncthreads();
    asm volatile("" ::: "memory");
  }
};
struct SyncWarp {
  __device__ __forceinline__ void operator()() const {
    asm volatile("" ::: "memory");
    __syncwarp();
    asm volatile("" ::: "memory");
  }
};

// Shared-memory slot of element p of a row buffer (sstride = 1) when PAD is set.
//   8-byte elements (complex float), rows of 16 threads or more: p ^ (p / 16 mod 16), a permutation
//   inside each 128-byte line (16 elements) keyed by the line index: the contiguous reads of every
//   stage stay on whole lines and the stride-E writes of stage 0 and the grouped writes of the
//   middle stages spread over the banks, so that the sixteen elements of each half-warp fall in
//   distinct bank pairs.  Rows of 2 to 8 threads (E = 8): one spare slot per 8 elements (p + p / 8),
//   conflict-free for two rows of 8 threads side by side that start 8 slots apart (mod 16).
//   16-byte elements (complex double): one spare slot per E elements (p + p / E), which spreads
//   the stride-E writes; a warp needs four wavefronts for these anyway.
// Without PAD: p (column buffers, sstride = columns per block).
template <typename T, int N, int E, bool PAD> __device__ __forceinline__ int sidx(int p) {
  if constexpr (!PAD) {
    return p;
  } else if constexpr (sizeof(T) == 4 && N / E >= 16) {
    return p ^ ((p >> 4) & 15);
  } else {
    return p + (p >> ilog2(E));
  }
}
// In-place length-3 and length-5 DFTs (forward sign exp(-2 pi i jk / R); INV conjugates).  The
// constants are cos and sin of 2 pi / 3, 2 pi / 5 and 4 pi / 5.
template <typename T, bool INV> __device__ __forceinline__ void dft3(cplx<T>* x) {
  constexpr T s3 = T(0.86602540378443864676);  // sin(2 pi / 3)
  const cplx<T> t1 = cadd(x[1], x[2]);
  const cplx<T> d = csub(x[1], x[2]);
  const cplx<T> m = cmk(x[0].x - T(0.5) * t1.x, x[0].y - T(0.5) * t1.y);
  // -i s3 d (forward) / +i s3 d (inverse)
  const cplx<T> r = INV ? cmk(-s3 * d.y, s3 * d.x) : cmk(s3 * d.y, -s3 * d.x);
  x[0] = cadd(x[0], t1);
  x[1] = cadd(m, r);
  x[2] = csub(m, r);
}

template <typename T, bool INV> __device__ __forceinline__ void dft5(cplx<T>* x) {
  constexpr T c1 = T(0.30901699437494742410);   // cos(2 pi / 5)
  constexpr T c2 = T(-0.80901699437494742410);  // cos(4 pi / 5)
  constexpr T s1 = T(0.95105651629515357212);   // sin(2 pi / 5)
  constexpr T s2 = T(0.58778525229247312917);   // sin(4 pi / 5)
  const cplx<T> a1 = cadd(x[1], x[4]), a2 = cadd(x[2], x[3]);
  const cplx<T> b1 = csub(x[1], x[4]), b2 = csub(x[2], x[3]);
  const cplx<T> t1 = cmk(x[0].x + c1 * a1.x + c2 * a2.x, x[0].y + c1 * a1.y + c2 * a2.y);
  const cplx<T> t2 = cmk(x[0].x + c2 * a1.x + c1 * a2.x, x[0].y + c2 * a1.y + c1 * a2.y);
  const cplx<T> u1 = cmk(s1 * b1.x + s2 * b2.x, s1 * b1.y + s2 * b2.y);
  const cplx<T> u2 = cmk(s2 * b1.x - s1 * b2.x, s2 * b1.y - s1 * b2.y);
  // forward: X1 = t1 - i u1, X4 = t1 + i u1, X2 = t2 - i u2, X3 = t2 + i u2
  const cplx<T> iu1 = INV ? cmk(-u1.y, u1.x) : cmk(u1.y, -u1.x);
  const cplx<T> iu2 = INV ? cmk(-u2.y, u2.x) : cmk(u2.y, -u2.x);
  x[0] = cadd(x[0], cadd(a1, a2));
  x[1] = cadd(t1, iu1);
  x[4] = csub(t1, iu1);
  x[2] = cadd(t2, iu2);
  x[3] = csub(t2, iu2);
}

// In-place length-3 P DFT, P = 2 or 4, by the prime-factor map: no twiddles, input n = 3 a + P b mod
// 3 P and output k = K3 a' + KP b' mod 3 P, with K3 = 1 mod P and 0 mod 3, KP = 1 mod 3 and 0 mod P.
template <typename T, int P, bool INV> __device__ __forceinline__ void dft3p(cplx<T>* x) {
  constexpr int R = 3 * P, K3 = P == 4 ? 9 : 3, KP = 4;
  cplx<T> y[R];
#pragma unroll
  for (int a = 0; a < P; ++a) {
    cplx<T> t[3];
#pragma unroll
    for (int b = 0; b < 3; ++b) t[b] = x[(3 * a + P * b) % R];
    dft3<T, INV>(t);
#pragma unroll
    for (int b = 0; b < 3; ++b) y[P * b + a] = t[b];
  }
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    dft<T, P, INV>(y + P * b);
#pragma unroll
    for (int a = 0; a < P; ++a) x[(K3 * a + KP * b) % R] = y[P * b + a];
  }
}

// Any radix of the mixed-radix pipeline: 2, 4, 8, 16 (bit-reversed passes), 3, 5, 6 or 12.
template <typename T, int R, bool INV> __device__ __forceinline__ void dft_any(cplx<T>* x) {
  if constexpr (R == 3) dft3<T, INV>(x);
  else if constexpr (R == 5) dft5<T, INV>(x);
  else if constexpr (R == 6) dft3p<T, 2, INV>(x);
  else if constexpr (R == 12) dft3p<T, 4, INV>(x);
  else dft<T, R, INV>(x);
}

__host__ __device__ constexpr bool is_pow2(int n) { return n > 0 && (n & (n - 1)) == 0; }

// Lengths N = 12 R2 R3: with k1 = 0..11, a = 0..R3-1, b and c = 0..R2-1, d = 0..R3-1,
//   stage 1  thread j = a + R3 b: radix 12 over x[j + NT m] -> k1, twiddle W_N^(j k1);
//   stage 2  for every (k1, a): radix R2 over b -> c, twiddle W_NT^(a c), in place;
//   stage 3  for every (k1, c): radix R3 over a -> d, output k = k1 + 12 c + 12 R2 d.
// The exchange buffer holds (k1, a + R3 c) at slot S(k1) + a + R3 c.  Stage 3's butterflies t = k1 +
// 12 c = j + NT q leave their outputs at j + NT (q + (12 / R3) d), the thread's own positions (the
// register contract), and stage 2 works in place, so two barriers separate the three stages.
// S(k1) = PITCH k1 + (k1 >> SH), the pitch and skew from an enumeration of the bank groups of each
// half-warp (FP32) or quarter-warp (FP64), rows of a warp side by side: stages 1 and 2 are free of bank
// conflicts (stage 2 of 360 in FP64: 10% more wavefronts), stage 3, whose lanes wrap past k1 = 11, takes
// 4/3 (FP64, FP32 96), 3/2 (FP64 360) or 2 (FP32) times as many.  A transform takes 1.08 (FP64, FP32 96),
// 1.25 (FP32) and, with the copies of lanes 0 and 1 that 360 has in its last quarter-warp, 1.21 (FP64
// 360) times the wavefronts without conflicts.  ROW is the row buffer's length.
template <typename T, int N> struct Len12 {
  static_assert(N == 360 || N == 384 || N == 192 || N == 96, "length 12 R2 R3");
  static constexpr int NT = N / 12;
  static constexpr int R2 = N == 360 ? 5 : (N == 384 ? 8 : 4), R3 = N == 360 ? 6 : (N == 96 ? 2 : 4);
  static constexpr bool F32 = sizeof(T) == 4;
  static constexpr int PITCH = NT + (N == 96 ? 2 : (N == 360 ? (F32 ? 8 : 0) : 4));
  static constexpr int SH = F32 ? (N == 360 ? 3 : 2) : (N == 360 ? 2 : (N == 96 ? 3 : 1));
  static constexpr int ROW = 11 * PITCH + (11 >> SH) + NT;
};

// The twiddles a thread uses, numbered: powers of two stage by stage (s >= 1), then by butterfly q,
// then by r = 1..R-1; N = 12 R2 R3: W_N^(j k1) for k1 = 1..11, then W_NT^(a c) for c = 1..R2-1 (a = j
// mod R3 for every butterfly of thread j).
template <int N, int E, bool P2> struct Pipe_;
template <int N, int E> struct Pipe_<N, E, true> {
  using Sh = FftShape<N, E>;
  static constexpr int NT = N / E, S = Sh::S;
  static __host__ __device__ constexpr int per(int s) { return E / Sh::radix(s); }
  static __host__ __device__ constexpr int first(int s) {
    return s <= 1 ? 0 : first(s - 1) + per(s - 1) * (Sh::radix(s - 1) - 1);
  }
  static constexpr int COUNT = first(S);
  // f(number, table index) over thread j's twiddles
  template <class F, int s = 1> static __device__ __forceinline__ void each(int j, F f) {
    if constexpr (s < S) {
#pragma unroll
      for (int q = 0; q < per(s); ++q)
#pragma unroll
        for (int r = 1; r < Sh::radix(s); ++r)
          f(first(s) + q * (Sh::radix(s) - 1) + r - 1, r * ((j + NT * q) % Sh::ns(s)) * (N / (Sh::ns(s) * Sh::radix(s))));
      each<F, s + 1>(j, f);
    }
  }
};
template <int N, int E> struct Pipe_<N, E, false> {
  using L = Len12<float, N>;
  static constexpr int COUNT = 11 + L::R2 - 1;
  template <class F> static __device__ __forceinline__ void each(int j, F f) {
#pragma unroll
    for (int k = 1; k < 12; ++k) f(k - 1, j * k);
#pragma unroll
    for (int c = 1; c < L::R2; ++c) f(10 + c, 12 * (j % L::R3) * c);
  }
};
template <int N, int E> using Pipe = Pipe_<N, E, is_pow2(N)>;

// A thread's twiddles in registers (loaded once, used by every transform of a persistent kernel).
template <typename T, int N, int E> struct TwRegs {
  cplx<T> w[Pipe<N, E>::COUNT];
  __device__ __forceinline__ void load(const cplx<T>* __restrict__ tab, int j) {
    Pipe<N, E>::each(j, [&](int n, int p) { w[n] = tab[p]; });
  }
};
// The same in shared memory, twiddle n of thread j at p[n * NT] (p already at j): contiguous over
// the threads of a row, where the table's own order would touch a line per thread.
template <typename T, int N, int E> struct TwLane {
  const cplx<T>* p;
  static constexpr int ELEMS = Pipe<N, E>::COUNT * (N / E);
  static __device__ __forceinline__ void fill(cplx<T>* dst, const cplx<T>* __restrict__ tab, int tid, int nthreads) {
    for (int j = tid; j < N / E; j += nthreads)
      Pipe<N, E>::each(j, [&](int n, int q) { dst[n * (N / E) + j] = tab[q]; });
  }
};
// Twiddle number n (table index p) from any of the sources, conjugated for the inverse.
template <typename T, int N, int E, bool INV> __device__ __forceinline__ cplx<T> tw_at(const cplx<T>* tw, int n, int p) {
  (void)n;
  return twid<T, INV>(tw, p);
}
template <typename T, int N, int E, bool INV>
__device__ __forceinline__ cplx<T> tw_at(const TwRegs<T, N, E>& tw, int n, int p) {
  (void)p;
  cplx<T> w = tw.w[n];
  if (INV) w.y = -w.y;
  return w;
}
template <typename T, int N, int E, bool INV>
__device__ __forceinline__ cplx<T> tw_at(const TwLane<T, N, E>& tw, int n, int p) {
  (void)p;
  cplx<T> w = tw.p[n * (N / E)];
  if (INV) w.y = -w.y;
  return w;
}

// The three stages of a length N = 12 R2 R3 (see Len12); without PAD the slots are a + R3 c + NT k1.
// A row buffer (PAD) serves NT lanes of a warp; lanes past its last whole row (360: NT = 30, lanes 30
// and 31) run along as copies of a row's first lanes.  They only read it: stage 2 replaces the values
// it has read, with no barrier in between, so a copy that is not in step with the lane it repeats
// would transform values already transformed.
template <typename T, int N, bool INV, bool PAD, class Tw, class Sync>
__device__ __forceinline__ void fft_run_12(cplx<T>* a, cplx<T>* sbuf, int sstride, int j, const Tw& tw, Sync sync) {
  using L = Len12<T, N>;
  constexpr int NT = L::NT, R2 = L::R2, R3 = L::R3, Q2 = (12 + R2 - 1) / R2, Q3 = 12 / R3;
  auto S = [](int k1) { return PAD ? L::PITCH * k1 + (k1 >> L::SH) : NT * k1; };
  bool own = true;
  if constexpr (PAD && 32 % NT != 0) own = (int)(threadIdx.x & 31) < 32 / NT * NT;
  dft3p<T, 4, INV>(a);
  if (own) {
#pragma unroll
    for (int k = 0; k < 12; ++k)
      sbuf[(S(k) + j) * sstride] = k ? cmul(a[k], tw_at<T, N, 12, INV>(tw, k - 1, j * k)) : a[k];
  }
  sync();
#pragma unroll
  for (int q = 0; q < Q2; ++q) {
    const int u = j + NT * q;
    if (own && (Q2 * R2 == 12 || u < 12 * R3)) {
      const int i = u % R3;
      cplx<T>* p = sbuf + (S(u / R3) + i) * sstride;
      cplx<T> x[R2];
#pragma unroll
      for (int b = 0; b < R2; ++b) x[b] = p[b * R3 * sstride];
      dft_any<T, R2, INV>(x);
#pragma unroll
      for (int c = 0; c < R2; ++c)
        p[c * R3 * sstride] = c ? cmul(x[c], tw_at<T, N, 12, INV>(tw, 10 + c, 12 * i * c)) : x[c];
    }
  }
  sync();
#pragma unroll
  for (int q = 0; q < Q3; ++q) {
    const int t = j + NT * q;
    const cplx<T>* p = sbuf + (S(t % 12) + R3 * (t / 12)) * sstride;
    cplx<T> x[R3];
#pragma unroll
    for (int i = 0; i < R3; ++i) x[i] = p[i * sstride];
    dft_any<T, R3, INV>(x);
#pragma unroll
    for (int d = 0; d < R3; ++d) a[q + Q3 * d] = x[d];
  }
}

// Stage s >= 1 of the Stockham pipeline (compile-time recursion over the stages).
template <typename T, int N, int E, bool INV, bool PAD, int s, class Tw, class Sync>
__device__ __forceinline__ void fft_stage(cplx<T>* a, cplx<T>* sbuf, int sstride, int j, const Tw& tw, Sync sync) {
  using Sh = FftShape<N, E>;
  constexpr int NT = Sh::NT;
  constexpr int S = Sh::S;
  constexpr int R = Sh::radix(s);
  constexpr int Ns = Sh::ns(s);
  constexpr int Q = E / R;
  cplx<T> x[E];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int b = j + NT * q;
#pragma unroll
    for (int r = 0; r < R; ++r) x[q * R + r] = sbuf[sidx<T, N, E, PAD>(b + r * (N / R)) * sstride];
  }
  sync();
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int b = j + NT * q;
    const int k = b % Ns;
#pragma unroll
    for (int r = 1; r < R; ++r) x[q * R + r] = cmul(x[q * R + r], tw_at<T, N, E, INV>(tw, Pipe<N, E>::first(s) + q * (R - 1) + r - 1,
                                                                            r * k * (N / (Ns * R))));
    dft<T, R, INV, W16<T>::exact(N, E, PAD)>(x + q * R);
    if constexpr (s < S - 1) {
      const int base = (b / Ns) * Ns * R + k;
#pragma unroll
      for (int r = 0; r < R; ++r) sbuf[sidx<T, N, E, PAD>(base + r * Ns) * sstride] = x[q * R + r];
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) a[q + r * Q] = x[q * R + r];
    }
  }
  if constexpr (s < S - 1) {
    sync();
    fft_stage<T, N, E, INV, PAD, s + 1>(a, sbuf, sstride, j, tw, sync);
  }
}

// Full FFT of length N; see the register contract at the top of this file.  The caller must
// not touch sbuf between fft_run() calls without a barrier: the last stage reads it.
template <typename T, int N, int E, bool INV, bool PAD, class Tw, class Sync>
__device__ __forceinline__ void fft_run(cplx<T>* a, cplx<T>* sbuf, int sstride, int j, const Tw& tw, Sync sync) {
  if constexpr (is_pow2(N)) {
    using Sh = FftShape<N, E>;
    dft<T, E, INV, W16<T>::exact(N, E, PAD)>(a);  // stage 0: radix E, Ns = 1, no twiddles
    if constexpr (Sh::S > 1) {
#pragma unroll
      for (int r = 0; r < E; ++r) sbuf[sidx<T, N, E, PAD>(j * E + r) * sstride] = a[r];
      sync();
      fft_stage<T, N, E, INV, PAD, 1>(a, sbuf, sstride, j, tw, sync);
    }
  } else {
    static_assert(E == 12, "lengths 12 R2 R3 take twelve elements per thread");
    fft_run_12<T, N, INV, PAD>(a, sbuf, sstride, j, tw, sync);
  }
}

// ------------------------------------------------------------------------------------------
// two FP32 transforms of one length side by side, on packed FP32 pairs
// ------------------------------------------------------------------------------------------
// Element n of both transforms: x = (re0, re1), y = (im0, im1).  Every operation is one packed
// instruction for both (add, multiply, fused multiply-add, each half rounding as the scalar one;
// differences as fma(b, -1, a)), which halves the instructions of the row passes: they issue on two
// thirds of their cycles and their transforms are two thirds of what they issue.
struct C2 {
  float2 x, y;
};
__device__ __forceinline__ float2 f2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, f2(-1.f), a); }

// The butterfly of both transforms.
template <bool INV, bool EXACT> __device__ __forceinline__ void butterfly2(C2& p, C2& q, int m) {
  using W = W16<float>;
  const C2 u = p, v = q;
  if (m == 0) {
    p.x = __fadd2_rn(u.x, v.x);
    p.y = __fadd2_rn(u.y, v.y);
    q.x = sub2(u.x, v.x);
    q.y = sub2(u.y, v.y);
  } else if (m == 4) {  // v -> -i v (forward), i v (inverse)
    const float2 ax = __fadd2_rn(u.x, v.y), sx = sub2(u.x, v.y);
    const float2 ay = __fadd2_rn(u.y, v.x), sy = sub2(u.y, v.x);
    p.x = INV ? sx : ax;
    p.y = INV ? ay : sy;
    q.x = INV ? ax : sx;
    q.y = INV ? sy : ay;
  } else if (m == 2 || m == 6) {
    const float2 s = __fadd2_rn(v.x, v.y), d = sub2(v.x, v.y);
    const float2 a = m == 2 ? (INV ? d : s) : (INV ? s : d), b = m == 2 ? (INV ? s : d) : (INV ? d : s);
    const float ka = m == 2 ? W::c2 : -W::c2, kb = INV ? W::c2 : -W::c2;
    p.x = __ffma2_rn(a, f2(ka), u.x);
    p.y = __ffma2_rn(b, f2(kb), u.y);
    q.x = __ffma2_rn(a, f2(-ka), u.x);
    q.y = __ffma2_rn(b, f2(-kb), u.y);
  } else {
    const OddW16<INV> o(m);
    const float ka = o.ka, kb = o.kb;
    const float2 a = o.xy ? __ffma2_rn(v.y, f2(o.ta), v.x) : __ffma2_rn(v.x, f2(o.ta), v.y);
    const float2 b = o.xy ? __ffma2_rn(v.x, f2(-o.ta), v.y) : __ffma2_rn(v.y, f2(-o.ta), v.x);
    C2 up = u, uq = u;
    if constexpr (EXACT) {
      up = C2{__ffma2_rn(a, f2(ka * W::l1), u.x), __ffma2_rn(b, f2(kb * W::l1), u.y)};
      uq = C2{__ffma2_rn(a, f2(-ka * W::l1), u.x), __ffma2_rn(b, f2(-kb * W::l1), u.y)};
    }
    p.x = __ffma2_rn(a, f2(ka * W::c1), up.x);
    p.y = __ffma2_rn(b, f2(kb * W::c1), up.y);
    q.x = __ffma2_rn(a, f2(-ka * W::c1), uq.x);
    q.y = __ffma2_rn(b, f2(-kb * W::c1), uq.y);
  }
}
template <int R, int LEN, bool INV, bool EXACT> __device__ __forceinline__ void dft_pass2(C2* a) {
  if constexpr (LEN <= R) {
#pragma unroll
    for (int i = 0; i < R; i += LEN)
#pragma unroll
      for (int q = 0; q < LEN / 2; ++q) butterfly2<INV, EXACT>(a[i + q], a[i + q + LEN / 2], q * (16 / LEN));
    dft_pass2<R, 2 * LEN, INV, EXACT>(a);
  }
}
template <int R, int I> __device__ __forceinline__ void bitrev_swaps2(C2* a) {
  if constexpr (I < R) {
    constexpr int K = bitrev(I, ilog2(R));
    if constexpr (K > I) {
      const C2 t = a[I];
      a[I] = a[K];
      a[K] = t;
    }
    bitrev_swaps2<R, I + 1>(a);
  }
}
template <int R, bool INV, bool EXACT> __device__ __forceinline__ void dft2(C2* a) {
  if constexpr (R > 1) {
    bitrev_swaps2<R, 0>(a);
    dft_pass2<R, 2, INV, EXACT>(a);
  }
}

// Exchange buffer of 16-byte elements: p ^ (p / E mod E), conflict-free for the quarter-warps of
// stage 0's writes (E apart) and of the contiguous reads.
template <int E> __device__ __forceinline__ int sidx2(int p) { return p ^ ((p / E) & (E - 1)); }

// Twiddles in shared memory as (wr, wr, wi, wi), in lane order: twiddle n of thread j at p[n * NT].
template <int N, int E> struct TwLane2 {
  const float4* p;
  static constexpr int ELEMS = Pipe<N, E>::COUNT * (N / E);
  static __device__ __forceinline__ void fill(float4* dst, const float2* __restrict__ tab, int tid, int nthreads) {
    for (int j = tid; j < N / E; j += nthreads)
      Pipe<N, E>::each(j, [&](int n, int q) {
        const float2 w = tab[q];
        dst[n * (N / E) + j] = make_float4(w.x, w.x, w.y, w.y);
      });
  }
};
// for a single transform beside the packed ones
template <typename T, int N, int E, bool INV>
__device__ __forceinline__ float2 tw_at(const TwLane2<N, E>& tw, int n, int p) {
  (void)p;
  const float4 w = tw.p[n * (N / E)];
  return make_float2(w.x, INV ? -w.z : w.z);
}
// a W (forward) or a conj(W) (inverse)
template <bool INV> __device__ __forceinline__ C2 cmul2(const C2& a, float4 w) {
  const float2 wr = make_float2(w.x, w.y), wi = make_float2(w.z, w.w), nwi = __fmul2_rn(wi, f2(-1.f));
  C2 r;
  r.x = __ffma2_rn(a.y, INV ? wi : nwi, __fmul2_rn(a.x, wr));
  r.y = __ffma2_rn(a.x, INV ? nwi : wi, __fmul2_rn(a.y, wr));
  return r;
}

// Exchange slot of element p: row buffers (STRIDE = 1) swizzled, column buffers p STRIDE.
template <int E, int STRIDE> __device__ __forceinline__ int slot2(int p) { return STRIDE == 1 ? sidx2<E>(p) : p * STRIDE; }

template <int N, int E, bool INV, int STRIDE, int s, class Sync>
__device__ __forceinline__ void fft_stage2(C2* a, float4* sbuf, int j, const TwLane2<N, E>& tw, Sync sync) {
  using Sh = FftShape<N, E>;
  constexpr int NT = Sh::NT, S = Sh::S, R = Sh::radix(s), Ns = Sh::ns(s), Q = E / R;
  C2 x[E];
#pragma unroll
  for (int q = 0; q < Q; ++q)
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float4 v = sbuf[slot2<E, STRIDE>(j + NT * q + r * (N / R))];
      x[q * R + r] = C2{make_float2(v.x, v.y), make_float2(v.z, v.w)};
    }
  if constexpr (s < S - 1) sync();
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int b = j + NT * q, k = b % Ns;
#pragma unroll
    for (int r = 1; r < R; ++r)
      x[q * R + r] = cmul2<INV>(x[q * R + r], tw.p[(Pipe<N, E>::first(s) + q * (R - 1) + r - 1) * NT]);
    dft2<R, INV, W16<float>::exact(N, E, STRIDE == 1)>(x + q * R);
    if constexpr (s < S - 1) {
      const int base = (b / Ns) * Ns * R + k;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const C2 c = x[q * R + r];
        sbuf[slot2<E, STRIDE>(base + r * Ns)] = make_float4(c.x.x, c.x.y, c.y.x, c.y.y);
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) a[q + r * Q] = x[q * R + r];
    }
  }
  if constexpr (s < S - 1) {
    sync();
    fft_stage2<N, E, INV, STRIDE, s + 1>(a, sbuf, j, tw, sync);
  }
}

// Both transforms, powers of two: the register contract of fft_run().
template <int N, int E, bool INV, int STRIDE, class Sync>
__device__ __forceinline__ void fft_run2(C2* a, float4* sbuf, int j, const TwLane2<N, E>& tw, Sync sync) {
  dft2<E, INV, W16<float>::exact(N, E, STRIDE == 1)>(a);
#pragma unroll
  for (int r = 0; r < E; ++r)
    sbuf[slot2<E, STRIDE>(j * E + r)] = make_float4(a[r].x.x, a[r].x.y, a[r].y.x, a[r].y.y);
  sync();
  fft_stage2<N, E, INV, STRIDE, 1>(a, sbuf, j, tw, sync);
}

}  // namespace ld
