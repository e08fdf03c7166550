// Kernel templates of the DNS step: the three axis passes of the 3D real transform, the fused
// nonlinear-term z pass, the k-space update epilogues, spectra/forcing and the droplet kernels.
//
// Data layout (see include/ld.h): physical fields (N,N,N) z fastest; spectra either in the
// reference's full layout (N, N, Nf) or in the dealiased cube (Mx, My, Mzp).
//
// Transform structure for the DNS (cube layout, c = complex element):
//   inverse : x pass (cube rows kx -> N rows x)  |  y pass (My rows ky -> N rows y)
//             |  z pass (kz <= kc -> N reals z)
//   forward : z pass (N reals -> kz < Mzp)  |  y pass (N rows -> My rows)  |  x pass (N -> Mx)
// Rows that are zero on input (|k| > kc) are never read and rows outside the cube are never
// written, so each pass moves only the data the dealiased spectrum needs.
#pragma once
#include <type_traits>

#include "ld_async.cuh"
#include "ld_fft.cuh"

namespace ld {

// ------------------------------------------------------------------------------------------
// index helpers
// ------------------------------------------------------------------------------------------
// logical FFT index n in [0, N) -> compact cube row, or -1 when |freq| > kc
__device__ __forceinline__ int crow(int n, int N, int kc) {
  return n <= kc ? n : (n >= N - kc ? n - (N - 2 * kc - 1) : -1);
}
// compact cube row -> signed frequency
__device__ __forceinline__ int cfreq(int i, int kc) { return i <= kc ? i : i - (2 * kc + 1); }
// logical FFT index -> signed frequency (fftfreq convention: N/2 -> -N/2)
__device__ __forceinline__ int nfreq(int n, int N) { return n < N / 2 ? n : n - N; }

// 4-vectors for interleaved physical fields (u, v, w, 0)
template <typename T> struct V4T;
template <> struct V4T<float> { using type = float4; };
template <> struct V4T<double> { using type = double4; };
template <typename T> using vec4 = typename V4T<T>::type;
template <typename T> __device__ __forceinline__ vec4<T> mk4(T a, T b, T c, T d) {
  vec4<T> v; v.x = a; v.y = b; v.z = c; v.w = d; return v;
}

// Launch shapes of the column passes by N.  Powers of two: as tuned.  N = 12 R2 R3: twelve elements
// per thread, a CTA of 8 columns (64-byte FP32 / 128-byte FP64 row segments).
template <int N> struct Cfg {
  static constexpr bool P2 = is_pow2(N);
  // column passes: E elements per thread, TB columns per CTA
  static constexpr int EC = P2 ? ((N == 32 || N == 64) ? 8 : 16) : 12;
  static constexpr int NTC = N / EC;
  static constexpr int TB = P2 ? (N == 16 ? 64 : (N == 32 ? 32 : 16)) : 8;
  static constexpr int COL_THREADS = TB * NTC;
  // the dealiased cube of a plan of size N (ld_plan_create: kc = N / 3, rows padded to 8)
  static constexpr int KC = N / 3;
  static constexpr int MY = 2 * KC + 1;
  static constexpr int MZP = (KC + 1 + 7) / 8 * 8;
};

// Shapes of the z passes (contiguous rows).  A row lies inside one warp (N / E <= 32), so
// that its exchanges are warp-level, and a warp takes R rows side by side.  What bounds these
// passes is the shared-memory data path, so E is chosen for few exchanges per transform:
//   powers of two: E = 16 for FP32 rows of 128 and 256 (256 = 16 x 16: one exchange where E = 8
//   needs two), E = 8 for rows of 16..64 and for FP64 (the fused pass keeps three transforms of E
//   elements in registers), E = 16 for 512;
//   N = 12 R2 R3: E = 12, rows of 8, 16, 30 or 32 lanes and two exchanges inside a warp, where E = 8
//   spread a row of 360 over 45 threads (block-wide barriers) and four exchanges.
template <typename T, int N> struct ZCfg {
  static constexpr bool P2 = is_pow2(N);
  static constexpr int E = !P2 ? 12 : (N >= 512 || (sizeof(T) == 4 && (N == 128 || N == 256)) ? 16 : 8);
  static constexpr int NT = N / E;                         // threads per row
  static constexpr int R = 32 / NT;                        // rows per warp (360: lanes 30, 31 repeat lanes 0, 1)
  static constexpr int ZBUF = P2 ? N + N / E : Len12<T, P2 ? 96 : N>::ROW;  // padded row buffer
  // One-shot kernels (C2R, R2C of one pair of rows per unit): a short FP32 row of 128 has too few
  // threads with E = 16 (reference-layout transforms of 128^3: 82 us against 76)
  static constexpr int E1 = sizeof(T) == 4 && N == 128 ? 8 : E;
  static constexpr int THREADS1 = 256;
  static constexpr int UNITS1 = THREADS1 / 32 * (32 / (N / E1));  // row units per block
  static constexpr int ZBUF1 = P2 ? N + N / E1 : ZBUF;
  // twiddles of the fused pass: in registers where three transforms and they fit (FP64 powers of
  // two; FP32 512, whose eight warps per SM run at 255 registers), else in shared memory in lane
  // order (FP32 128 at 168 registers and three CTAs per SM)
  // packed transforms: FP32 rows of 256 (right-hand side 388 -> 366 us, warp instructions down by a
  // quarter); 512 (16 x 16 x 2 at 8 warps per SM: 3.71 -> 3.75 ms), 128 (60.7 -> 64.1 us) and the plane
  // pass of 64 are not faster with them
  static constexpr bool PACK = sizeof(T) == 4 && N == 256;
  static constexpr bool TWREG = sizeof(T) == 4 ? N == 512 : Pipe<N, E>::COUNT <= 13;
};

// ------------------------------------------------------------------------------------------
// column (strided axis) passes
// ------------------------------------------------------------------------------------------
// Plain strided rows: element (f, o, row, col) at f*fs + o*os + row*RS + col.  The row stride RS is
// a template constant (every pass has one fixed by N), so that the rows of a thread are one base
// address and immediate offsets: the y passes spent a third of their instructions on addresses.
template <typename T> struct RowsIO {
  cplx<T>* p;
  long long fs, os;
  __device__ __forceinline__ cplx<T>* at(int f, int o, int col) const {
    return p + ((long long)f * fs + (long long)o * os + col);
  }
};
// Row strides of the passes: y and x passes over cube rows, y and x passes over reference-layout rows
template <int N> struct RowStride {
  static constexpr int YC = Cfg<N>::MZP, XC = Cfg<N>::MY * Cfg<N>::MZP;
  static constexpr int YF = N / 2 + 1, XF = N * (N / 2 + 1);
};

// Strided row loader: rows mapped to compact cube rows through crow (MAP) or taken as they are.
template <typename T, int N, bool MAP, int RS> struct LdRowsC {
  RowsIO<T> io;
  __device__ __forceinline__ cplx<T> operator()(int f, int o, int n, int col) const {
    const int r = MAP ? crow(n, N, Cfg<N>::KC) : n;
    if (r < 0) return czero<cplx<T>>();
    return io.at(f, o, col)[(long long)r * RS];
  }
  // columns col, col + 1 (FP32; RS and col even, rows 16-byte aligned)
  __device__ __forceinline__ float4 two(int f, int o, int n, int col) const {
    const int r = MAP ? crow(n, N, Cfg<N>::KC) : n;
    if (r < 0) return make_float4(0.f, 0.f, 0.f, 0.f);
    return *reinterpret_cast<const float4*>(io.at(f, o, col) + (long long)r * RS);
  }
};

// Strided row storer: rows mapped to compact cube rows through crow (MAP; rows outside the cube
// are not written) or taken as they are.
template <typename T, int N, bool MAP, int RS> struct StRowsC {
  RowsIO<T> io;
  __device__ __forceinline__ void operator()(int f, int o, int n, int col, cplx<T> v) const {
    const int r = MAP ? crow(n, N, Cfg<N>::KC) : n;
    if (r < 0) return;
    io.at(f, o, col)[(long long)r * RS] = v;
  }
  __device__ __forceinline__ void two(int f, int o, int n, int col, float4 v) const {
    const int r = MAP ? crow(n, N, Cfg<N>::KC) : n;
    if (r < 0) return;
    *reinterpret_cast<float4*>(io.at(f, o, col) + (long long)r * RS) = v;
  }
};

// Storer into the cube that also applies the spherical mask round(|k|) <= kc (F:129): the last
// (x) pass of a forward cube transform.  Columns are the flat (ky, kz) index of a kx plane.
template <typename T, int N> struct StCube {
  RowsIO<T> io;
  __device__ __forceinline__ void operator()(int f, int o, int n, int col, cplx<T> v) const {
    constexpr int kc = Cfg<N>::KC, Mzp = Cfg<N>::MZP;
    const int r = crow(n, N, kc);
    if (r < 0) return;
    const int kx = n <= kc ? n : n - N;
    const int iy = col / Mzp;
    const int ky = cfreq(iy, kc), kz = col - iy * Mzp;
    if (kz > kc || kx * kx + ky * ky + kz * kz > kc * kc + kc) v = czero<cplx<T>>();
    io.at(f, o, col)[(long long)r * RowStride<N>::XC] = v;
  }
};

// Inverse x-pass loader producing [u_x, u_y, u_z, w_x, w_y, w_z] from a cube 3-vector:
// w = i k x u (F:295-297).  Columns are the flat (ky, kz) index of a kx plane.
template <typename T, int N> struct LdCurl {
  const cplx<T>* u;
  long long cs;  // component stride (cube elements)
  long long bs;  // box stride (elements): the outer index is the box of a multi-box plan
  static constexpr int kc = Cfg<N>::KC, My = Cfg<N>::MY, Mzp = Cfg<N>::MZP;
  __device__ __forceinline__ cplx<T> operator()(int f, int o, int n, int col) const {
    const int r = crow(n, N, kc);
    if (r < 0) return czero<cplx<T>>();
    const long long b = (long long)o * bs + (long long)r * My * Mzp + col;
    if (f < 3) return u[f * cs + b];
    const T kx = T(n <= kc ? n : n - N);
    const int iy = col / Mzp;
    const T ky = T(cfreq(iy, kc));
    const T kz = T(col - iy * Mzp);
    cplx<T> w;
    if (f == 3) {        // i (ky u_z - kz u_y)
      cplx<T> uy = u[cs + b], uz = u[2 * cs + b];
      w = cmuli(csub(cscale(uz, ky), cscale(uy, kz)));
    } else if (f == 4) { // i (kz u_x - kx u_z)
      cplx<T> ux = u[b], uz = u[2 * cs + b];
      w = cmuli(csub(cscale(ux, kz), cscale(uz, kx)));
    } else {             // i (kx u_y - ky u_x)
      cplx<T> ux = u[b], uy = u[cs + b];
      w = cmuli(csub(cscale(uy, kx), cscale(ux, ky)));
    }
    return w;
  }
  // columns col, col + 1 (FP32; col even, u 16-byte aligned): one ky, two neighbouring kz
  __device__ __forceinline__ float4 two(int f, int o, int n, int col) const {
    const int r = crow(n, N, kc);
    if (r < 0) return make_float4(0.f, 0.f, 0.f, 0.f);
    const cplx<T>* b = u + (long long)o * bs + (long long)r * My * Mzp + col;
    auto get = [&](int c) { return *reinterpret_cast<const float4*>(b + c * cs); };
    if (f < 3) return get(f);
    const float kx = float(n <= kc ? n : n - N);
    const int iy = col / Mzp;
    const float ky = float(cfreq(iy, kc));
    const float kz = float(col - iy * Mzp);
    // i (p a - q b) for the two columns
    auto curl = [](float4 a, float pa0, float pa1, float4 b, float qb0, float qb1) {
      return make_float4(-(a.y * pa0 - b.y * qb0), a.x * pa0 - b.x * qb0, -(a.w * pa1 - b.w * qb1),
                         a.z * pa1 - b.z * qb1);
    };
    if (f == 3) return curl(get(2), ky, ky, get(1), kz, kz + 1.f);  // i (ky u_z - kz u_y)
    if (f == 4) return curl(get(0), kz, kz + 1.f, get(2), kx, kx);  // i (kz u_x - kx u_z)
    return curl(get(1), kx, kx, get(0), ky, ky);                    // i (kx u_y - ky u_x)
  }
};

// One CTA = TB columns x NT threads; blockIdx.x = tile * nf + field (fields of a tile launch
// together so their shared inputs are served from L2), blockIdx.y = outer index.
template <typename T, int N, bool INV, class Ld, class St>
__device__ __forceinline__ void colfft_tile(const Ld& ld, const St& st, int ncols, int nf, const cplx<T>* __restrict__ tw,
                                            unsigned char* smem) {
  constexpr int E = Cfg<N>::EC, TB = Cfg<N>::TB, NT = Cfg<N>::NTC;
  cplx<T>* sbuf = reinterpret_cast<cplx<T>*>(smem);
  const int c = threadIdx.x % TB, j = threadIdx.x / TB;
  __builtin_assume(j >= 0 && j < NT);
  const int field = blockIdx.x % nf;
  const int col = (blockIdx.x / nf) * TB + c;
  const bool ok = col < ncols;
  const int outer = blockIdx.y;
  cplx<T> a[E];
#pragma unroll
  for (int m = 0; m < E; ++m) a[m] = ok ? ld(field, outer, j + NT * m, col) : czero<cplx<T>>();
  fft_run<T, N, E, INV, false>(a, sbuf + c, TB, j, tw, SyncBlock());
  if (ok) {
#pragma unroll
    for (int m = 0; m < E; ++m) st(field, outer, j + NT * m, col, a[m]);
  }
}

template <typename T, int N, bool INV, class Ld, class St>
__global__ void __launch_bounds__(Cfg<N>::COL_THREADS)
k_colfft(Ld ld, St st, int ncols, int nf, const cplx<T>* __restrict__ tw) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  grid_dep();
  colfft_tile<T, N, INV>(ld, st, ncols, nf, tw, smem_raw);
}

// The same tile with five CTAs per SM, for N = 256 in FP32: 48 registers, no spills, 32 KB of shared
// memory each, instead of four CTAs at 56 registers.  These one-shot tiles wait on their loads and
// the extra warps hide that latency (x inverse 0.072 -> 0.067 ms).  Elsewhere k_colfft keeps the
// compiler's own register choice: stating one CTA per SM would let the FP64 tiles grow from about
// 90 to about 150 registers.
template <typename T, int N, bool INV, class Ld, class St>
__global__ void __launch_bounds__(Cfg<N>::COL_THREADS, 5)
k_colfft5(Ld ld, St st, int ncols, int nf, const cplx<T>* __restrict__ tw) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  grid_dep();
  colfft_tile<T, N, INV>(ld, st, ncols, nf, tw, smem_raw);
}

template <typename T, int N, bool INV, class Ld, class St>
constexpr auto colfft_kernel() {
  if constexpr (N == 256 && sizeof(T) == 4) return k_colfft5<T, N, INV, Ld, St>;
  else return k_colfft<T, N, INV, Ld, St>;
}

// The tile with two neighbouring columns per thread, FP32: 16-byte accesses, and their transforms as
// packed pairs (C2), which halves the instructions of a pass.  It pays where the one-column tiles
// queue for issue slots and the load unit (512^3: inverse y 823 -> 736 us, right-hand side 3.70 ->
// 3.43 ms; 128^3 60.5 -> 58.4 us); at 256^3 the passes wait for memory either way (366 -> 361 us).  The twiddles are put into shared
// memory in lane order, behind the exchange buffer.
template <int N> struct Col2 {
  static constexpr int E = Cfg<N>::EC, NT = Cfg<N>::NTC, PAIRS = Cfg<N>::TB / 2;
  static constexpr bool OK = is_pow2(N) && E == 16 && N >= 128;
  static constexpr int THREADS = PAIRS * NT;
  static constexpr int MINB = 640 / THREADS;  // 96 registers (128: five in four at 256^3; 80: spills)
  using Tw = TwLane2<is_pow2(N) ? N : 64, is_pow2(N) ? E : 8>;
  static constexpr size_t BUF = sizeof(float4) * N * PAIRS, SMEM = BUF + sizeof(float4) * Tw::ELEMS;
};
__device__ __forceinline__ C2 pair_of(float4 v) { return C2{make_float2(v.x, v.z), make_float2(v.y, v.w)}; }
__device__ __forceinline__ float4 columns_of(const C2& c) { return make_float4(c.x.x, c.y.x, c.x.y, c.y.y); }

template <int N, bool INV, class Ld, class St>
__device__ __forceinline__ void colfft_tile2(const Ld& ld, const St& st, int ncols, int nf, const float2* __restrict__ tw,
                                             unsigned char* smem) {
  using C = Col2<N>;
  constexpr int E = C::E, NT = C::NT;
  float4* sbuf = reinterpret_cast<float4*>(smem);
  float4* tws = reinterpret_cast<float4*>(smem + C::BUF);
  const int c = threadIdx.x % C::PAIRS, j = threadIdx.x / C::PAIRS;
  __builtin_assume(j >= 0 && j < NT);
  const int field = blockIdx.x % nf;
  const int col = (blockIdx.x / nf) * Cfg<N>::TB + 2 * c;
  const bool ok = col < ncols;  // ncols is even
  const int outer = blockIdx.y;
  float4 v[E];
#pragma unroll
  for (int m = 0; m < E; ++m) v[m] = ok ? ld.two(field, outer, j + NT * m, col) : make_float4(0.f, 0.f, 0.f, 0.f);
  C::Tw::fill(tws, tw, threadIdx.x, C::THREADS);  // before the exchange's first barrier
  typename C::Tw t;
  t.p = tws + j;
  C2 a[E];
#pragma unroll
  for (int m = 0; m < E; ++m) a[m] = pair_of(v[m]);
  fft_run2<N, E, INV, C::PAIRS>(a, sbuf + c, j, t, SyncBlock());
  if (ok) {
#pragma unroll
    for (int m = 0; m < E; ++m) st.two(field, outer, j + NT * m, col, columns_of(a[m]));
  }
}


template <int N, bool INV, class Ld, class St>
__global__ void __launch_bounds__(Col2<N>::THREADS, Col2<N>::MINB)
k_colfft2(Ld ld, St st, int ncols, int nf, const float2* __restrict__ tw) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  grid_dep();
  colfft_tile2<N, INV>(ld, st, ncols, nf, tw, smem_raw);
}

// Sum of 0.5 |u|^2 normalize over the modes listed for shell s (CSR of cube indices), by the block
// in a fixed order (FP64, deterministic); as_factor: the constant-power factor f0 / (2 E_s) of
// F:250-254 instead of E_s.  red: 32 doubles of shared memory.
template <typename T> struct ShellArgs {
  const cplx<T>* u;
  long long cs, ubs;  // component stride, box stride of u
  const int *off, *idx;
  int Mzp, shell0, nshell;
  double norm0, f0;
  int as_factor, obs;  // box stride of out
  double* out;
};
template <typename T> __device__ __forceinline__ void shell_sum(const ShellArgs<T>& A, int s, int box, double* red) {
  const cplx<T>* u = A.u + box * A.ubs;
  const int nthr = (int)blockDim.x & ~31;  // whole warps
  if ((int)threadIdx.x >= nthr) {
    __syncthreads();
    return;
  }
  double acc = 0.0;
  for (int t = A.off[s] + threadIdx.x; t < A.off[s + 1]; t += nthr) {
    const int e = A.idx[t];
    const double w = (e % A.Mzp) ? 2.0 : 1.0;  // Hermitian weight of F:136 (kz < N/2 here)
    double m = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      cplx<T> v = u[c * A.cs + e];
      m += double(v.x) * double(v.x) + double(v.y) * double(v.y);
    }
    acc += 0.5 * m * w * A.norm0;
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, d);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double e = red[0];
    for (int w = 1; w < nthr / 32; ++w) e += red[w];
    if (A.as_factor) {
      if (fabs(e) < 1e-10) e = INFINITY;  // F:250
      e = A.f0 / (2.0 * e);
    }
    A.out[box * A.obs + s] = e;
  }
}

template <typename T> __global__ void k_shell_sum(ShellArgs<T> A) {
  __shared__ double red[32];
  grid_dep();
  shell_sum(A, A.shell0 + (int)blockIdx.x, (int)blockIdx.y, red);
}

// The inverse x pass of the right-hand side (curl on load); the blocks past its tiles compute the
// forcing factors of the stage input, one shell each, which the update pass reads (a launch of its
// own cost 3.3 us, of 31 us for a right-hand side at 32^3).
template <typename T, int N, class St>
__device__ __forceinline__ void xinv_block(const LdCurl<T, N>& ld, const St& st, int ncols, const cplx<T>* __restrict__ tw,
                                           const ShellArgs<T>& F, unsigned char* smem) {
  const int tiles = 6 * ((ncols + Cfg<N>::TB - 1) / Cfg<N>::TB);
  if ((int)blockIdx.x < tiles) colfft_tile<T, N, true>(ld, st, ncols, 6, tw, smem);
  else shell_sum(F, F.shell0 + (int)blockIdx.x - tiles, (int)blockIdx.y, reinterpret_cast<double*>(smem));
}
template <typename T, int N, class St>
__global__ void __launch_bounds__(Cfg<N>::COL_THREADS)
k_xinv(LdCurl<T, N> ld, St st, int ncols, const cplx<T>* __restrict__ tw, ShellArgs<T> F) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  grid_dep();
  xinv_block<T, N>(ld, st, ncols, tw, F, smem_raw);
}
template <typename T, int N, class St>
__global__ void __launch_bounds__(Cfg<N>::COL_THREADS, 5)
k_xinv5(LdCurl<T, N> ld, St st, int ncols, const cplx<T>* __restrict__ tw, ShellArgs<T> F) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  grid_dep();
  xinv_block<T, N>(ld, st, ncols, tw, F, smem_raw);
}
template <int N, class St>
__global__ void __launch_bounds__(Col2<N>::THREADS, Col2<N>::MINB)
k_xinv2(LdCurl<float, N> ld, St st, int ncols, const float2* __restrict__ tw, ShellArgs<float> F) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  grid_dep();
  const int tiles = 6 * ((ncols + Cfg<N>::TB - 1) / Cfg<N>::TB);
  if ((int)blockIdx.x < tiles) colfft_tile2<N, true>(ld, st, ncols, 6, tw, smem_raw);
  else shell_sum(F, F.shell0 + (int)blockIdx.x - tiles, (int)blockIdx.y, reinterpret_cast<double*>(smem_raw));
}
template <typename T, int N, class St> constexpr auto xinv_kernel() {
  if constexpr (N == 256 && sizeof(T) == 4) return k_xinv5<T, N, St>;
  else return k_xinv<T, N, St>;
}

// Pipelined column pass over plain strided rows: a CTA loops over items (column block, field,
// outer index), items of neighbouring CTAs adjacent in memory.  While an item is transformed, the
// rows of the CTA's next item stream into the other shared buffer with 16-byte cp.async copies;
// the buffer an item was staged in serves as its FFT exchange buffer once its values sit in
// registers.  Rows the loader's row map drops (r < 0) and columns past ncols are not copied.
template <typename T, int N, bool INV, class St, bool IN_MAP, int RS>
__global__ void __launch_bounds__(Cfg<N>::COL_THREADS, 3)
k_colfft_pipe(RowsIO<T> in, St st, int ncols, int nf, int nouter, const cplx<T>* __restrict__ tw) {
  constexpr int E = Cfg<N>::EC, TB = Cfg<N>::TB, NT = Cfg<N>::NTC;
  constexpr int CPR = TB * (int)sizeof(cplx<T>) / 16;  // 16-byte chunks of a full row segment
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* buf0 = reinterpret_cast<cplx<T>*>(smem_raw);
  cplx<T>* buf1 = buf0 + N * TB;
  const int c = threadIdx.x % TB, j = threadIdx.x / TB;
  __builtin_assume(j >= 0 && j < NT);
  // item = (column block cb, field f, outer o), cb fastest; the launcher keeps the item count
  // below 2^31, so items are split with 32-bit unsigned division
  const unsigned ncb = (unsigned)((ncols + TB - 1) / TB);
  const unsigned nitems = ncb * (unsigned)nf * (unsigned)nouter;
  struct Item {
    int cb, f, o;
  };
  auto split = [&](unsigned it) {
    const unsigned rest = it / ncb;
    const unsigned fo = rest / (unsigned)nf;
    return Item{(int)(it - rest * ncb), (int)(rest - fo * (unsigned)nf), (int)fo};
  };
  // each thread copies one fixed 16-byte chunk k of rows threadIdx / CPR + (THREADS / CPR) i
  constexpr int THREADS = Cfg<N>::COL_THREADS;
  static_assert(THREADS % CPR == 0 && (N * CPR) % THREADS == 0, "whole rows per pass of the block");
  const int kq = threadIdx.x % CPR, n0 = threadIdx.x / CPR;
  __builtin_assume(n0 >= 0 && n0 < THREADS / CPR);
  auto prefetch = [&](const Item& itm, cplx<T>* dst) {
    const int col0 = itm.cb * TB;
    const int w = ncols - col0 < TB ? ncols - col0 : TB;
    const int cpr = w * (int)sizeof(cplx<T>) / 16;
    if (kq < cpr) {
      const char* src0 = reinterpret_cast<const char*>(in.at(itm.f, itm.o, col0)) + 16 * kq;
      const unsigned d0 = (unsigned)__cvta_generic_to_shared(reinterpret_cast<char*>(dst) + 16 * kq);
#pragma unroll
      for (int i = 0; i < N * CPR / THREADS; ++i) {
        const int n = n0 + (THREADS / CPR) * i;
        const int r = IN_MAP ? crow(n, N, Cfg<N>::KC) : n;
        if (r < 0) continue;
        const char* src = src0 + (long long)r * (RS * (long long)sizeof(cplx<T>));
        const unsigned d = d0 + (unsigned)(n * TB * (int)sizeof(cplx<T>));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  grid_dep();
  unsigned it = blockIdx.x;
  Item cur_item = split(it);
  if (it < nitems) prefetch(cur_item, buf0);
  int b = 0;
  for (; it < nitems; it += gridDim.x) {
    cplx<T>* cur = b ? buf1 : buf0;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int f = cur_item.f, o = cur_item.o;
    const int col = cur_item.cb * TB + c;
    const bool ok = col < ncols;
    cplx<T> a[E];
#pragma unroll
    for (int m = 0; m < E; ++m) {
      const int n = j + NT * m;
      const int r = IN_MAP ? crow(n, N, Cfg<N>::KC) : n;
      a[m] = (ok && r >= 0) ? cur[n * TB + c] : czero<cplx<T>>();
    }
    __syncthreads();  // every value is in registers: cur becomes the exchange buffer
    const unsigned nx = it + gridDim.x;
    const Item next_item = split(nx);
    if (nx < nitems) prefetch(next_item, b ? buf0 : buf1);
    fft_run<T, N, E, INV, false>(a, cur + c, TB, j, tw, SyncBlock());
    if (ok) {
#pragma unroll
      for (int m = 0; m < E; ++m) st(f, o, j + NT * m, col, a[m]);
    }
    __syncthreads();
    b ^= 1;
    cur_item = next_item;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// The pipelined pass with two columns per thread (see colfft_tile2 and k_colfft_pipe).
template <int N, bool INV, class St, bool IN_MAP, int RS>
__global__ void __launch_bounds__(Col2<N>::THREADS, 3)
k_colfft_pipe2(RowsIO<float> in, St st, int ncols, int nf, int nouter, const float2* __restrict__ tw) {
  using C = Col2<N>;
  constexpr int E = C::E, NT = C::NT, PAIRS = C::PAIRS, TB = Cfg<N>::TB, THREADS = C::THREADS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float4* buf0 = reinterpret_cast<float4*>(smem_raw);
  float4* buf1 = buf0 + N * PAIRS;
  float4* tws = buf1 + N * PAIRS;
  const int c = threadIdx.x % PAIRS, j = threadIdx.x / PAIRS;
  __builtin_assume(j >= 0 && j < NT);
  C::Tw::fill(tws, tw, threadIdx.x, THREADS);
  typename C::Tw t;
  t.p = tws + j;
  grid_dep();
  const unsigned ncb = (unsigned)((ncols + TB - 1) / TB);
  const unsigned nitems = ncb * (unsigned)nf * (unsigned)nouter;
  struct Item {
    int cb, f, o;
  };
  auto split = [&](unsigned it) {
    const unsigned rest = it / ncb;
    const unsigned fo = rest / (unsigned)nf;
    return Item{(int)(it - rest * ncb), (int)(rest - fo * (unsigned)nf), (int)fo};
  };
  // this thread copies what it will transform: its two columns of rows j + NT m
  auto prefetch = [&](const Item& itm, float4* dst) {
    if (itm.cb * TB + 2 * c < ncols) {
      const float2* src = in.at(itm.f, itm.o, itm.cb * TB + 2 * c);
      const unsigned d = (unsigned)__cvta_generic_to_shared(dst + c);
#pragma unroll
      for (int m = 0; m < E; ++m) {
        const int n = j + NT * m, r = IN_MAP ? crow(n, N, Cfg<N>::KC) : n;
        if (r < 0) continue;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16u * PAIRS * n), "l"(src + (long long)r * RS)
                     : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  unsigned it = blockIdx.x;
  Item cur_item = split(it);
  if (it < nitems) prefetch(cur_item, buf0);
  int b = 0;
  __syncthreads();  // the twiddles
  for (; it < nitems; it += gridDim.x) {
    float4* cur = b ? buf1 : buf0;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    const int f = cur_item.f, o = cur_item.o;
    const int col = cur_item.cb * TB + 2 * c;
    const bool ok = col < ncols;
    C2 a[E];
#pragma unroll
    for (int m = 0; m < E; ++m) {  // the thread's own copies
      const int n = j + NT * m, r = IN_MAP ? crow(n, N, Cfg<N>::KC) : n;
      a[m] = pair_of(ok && r >= 0 ? cur[n * PAIRS + c] : make_float4(0.f, 0.f, 0.f, 0.f));
    }
    __syncthreads();  // every value is in registers: cur becomes the exchange buffer, the other is free
    const unsigned nx = it + gridDim.x;
    const Item next_item = split(nx);
    if (nx < nitems) prefetch(next_item, b ? buf0 : buf1);
    fft_run2<N, E, INV, PAIRS>(a, cur + c, j, t, SyncBlock());
    if (ok) {
#pragma unroll
      for (int m = 0; m < E; ++m) st.two(f, o, j + NT * m, col, columns_of(a[m]));
    }
    b ^= 1;
    cur_item = next_item;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// ------------------------------------------------------------------------------------------
// k-space update epilogue of the forward x pass (F:304-316 + the time integrators)
// ------------------------------------------------------------------------------------------
enum UpdMode : int {
  UPD_RHS = 0,     // s0 <- P[nl + f] - visc nu k^2 s1               (s1 = stage input)
  UPD_RK2_1 = 1,   // s1 = uk: s0 <- E (uk + h N1) [ustar], s2 <- E (uk + h/2 N1) [acc]
  UPD_RK2_2 = 2,   // s1 = ustar: s0 <- s2 + h/2 N2                   (s0 = uk, s2 = acc)
  UPD_RK4_1 = 3,   // s0 = un, s1 = stage input, s2 = acc, s3 = next stage input
  UPD_RK4_2 = 4,
  UPD_RK4_3 = 5,
  UPD_RK4_4 = 6,
};

template <typename T> struct UpdArgs {
  const cplx<T>* nl;  // forward-transformed (u x w): (3, N, My, Mzp) rows x = N
  long long nls;      // component stride of nl
  cplx<T>* s0;
  cplx<T>* s1;
  cplx<T>* s2;
  cplx<T>* s3;
  long long cs;       // component stride of the cube
  const double* factor;  // forcing factor per shell (FP64), shells kf_lo..kf_hi
  int kf_lo, kf_hi;
  const T* ifac;         // exp(-nu h k^2) by k^2
  T h, nu, visc;
  int kc, My, Mzp;
  unsigned* status;
  // optional slow-manifold velocity of the stage input y (F:319-321):
  // vk = y + tps (k (k . rhs) / k^2 + visc nu k^2 y), minus vg = tps g N^3 on the mean of w
  cplx<T>* vk;
  T tps, vg;
  // stage the cube rows of the CTA's columns that the update reads for every mode (the stage input
  // s1; s2 in the second RK2 stage) into shared memory with cp.async while the x transforms run; the
  // launcher sets it when the (3, Mx, TB) buffer fits beside the exchange buffer at 2 CTAs per SM
  int prefetch;
  // final stages (UPD_RK2_2, UPD_RK4_4): the step epilogue's work on the kz > 0 modes (projection
  // and the non-finite / blow-up checks, as k_epilogue does them) is done here, so that the
  // epilogue that follows needs only the kz = 0 plane (k_epilogue_plane0)
  T blowup;
  // multi-box plans: blockIdx.y is the box; strides of nl, of the cube states and of the forcing
  // factors from one box to the next
  long long nl_bs, cube_bs;
  int fac_bs;
};

// The step epilogue of one kz > 0 mode (k_epilogue's arithmetic): projection with its own k
// inside the mask, zero outside; flags for non-finite values and the blow-up threshold.
template <typename T>
__device__ __forceinline__ void epi_mode(cplx<T> (&v)[3], int kx, int ky, int kz, int kc, T blowup, unsigned& flags) {
  const int k2 = kx * kx + ky * ky + kz * kz;
  if (kz <= kc && k2 <= kc * kc + kc) {
    const T qx = T(kx), qy = T(ky), qz = T(kz);
    cplx<T> kd = cscale(cadd(cadd(cscale(v[0], qx), cscale(v[1], qy)), cscale(v[2], qz)), T(1) / T(k2));
    v[0] = csub(v[0], cscale(kd, qx));
    v[1] = csub(v[1], cscale(kd, qy));
    v[2] = csub(v[2], cscale(kd, qz));
  } else {
    v[0] = v[1] = v[2] = czero<cplx<T>>();
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if (!(isfinite(v[c].x) && isfinite(v[c].y))) flags |= LD_STATUS_NONFINITE;
    if (v[c].x > blowup) flags |= LD_STATUS_BLOWUP;
  }
}

template <typename T, int N, int MODE>
__global__ void __launch_bounds__(Cfg<N>::COL_THREADS, (N == 256 && sizeof(T) == 4) ? 2 : 1)
k_xfwd_update(UpdArgs<T> A, int ncols, const cplx<T>* __restrict__ tw) {
  constexpr int E = Cfg<N>::EC, TB = Cfg<N>::TB, NT = Cfg<N>::NTC;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  grid_dep();
  if (blockIdx.y) {  // box of a multi-box plan
    const long long bo = blockIdx.y;
    A.nl += bo * A.nl_bs;
    if (A.s0) A.s0 += bo * A.cube_bs;
    if (A.s1) A.s1 += bo * A.cube_bs;
    if (A.s2) A.s2 += bo * A.cube_bs;
    if (A.s3) A.s3 += bo * A.cube_bs;
    A.factor += bo * A.fac_bs;
  }
  cplx<T>* sbuf = reinterpret_cast<cplx<T>*>(smem_raw);
  const int c = threadIdx.x % TB, j = threadIdx.x / TB;
  __builtin_assume(j >= 0 && j < NT);
  const int col = blockIdx.x * TB + c;
  const bool ok = col < ncols;
  constexpr int Mx = Cfg<N>::MY;  // A.kc == Cfg<N>::KC, A.My == Cfg<N>::MY, A.Mzp == Cfg<N>::MZP
  cplx<T>* ybuf = sbuf + N * TB;  // (3, Mx, TB) staged rows of s1 (s2 in the second RK2 stage)
  const bool pre = A.prefetch;
  if (pre) {
    constexpr int PER = 16 / (int)sizeof(cplx<T>);  // elements per 16-byte chunk
    const cplx<T>* src = MODE == UPD_RK2_2 ? A.s2 : A.s1;
    const int col0 = blockIdx.x * TB;
    const int w = ncols - col0 < TB ? ncols - col0 : TB;  // a multiple of 8 (Mzp is)
    const int cpr = w / PER;
    constexpr long long rs = (long long)Cfg<N>::MY * Cfg<N>::MZP;
    for (int q = threadIdx.x; q < 3 * Mx * (TB / PER); q += blockDim.x) {
      const int row = q / (TB / PER), k = q - row * (TB / PER);  // row = cc * Mx + r
      if (k >= cpr) continue;
      const int cc = row / Mx, r = row - cc * Mx;
      const cplx<T>* g = src + cc * A.cs + r * rs + col0 + k * PER;
      const unsigned d = (unsigned)__cvta_generic_to_shared(ybuf + row * TB + k * PER);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(g) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // the three components' loads in flight together, then their transforms (the registers of all
  // three are live through the last transform either way)
  cplx<T> res[3][E];
#pragma unroll
  for (int f = 0; f < 3; ++f)
#pragma unroll
    for (int m = 0; m < E; ++m)
      res[f][m] = ok ? A.nl[f * A.nls + col + (long long)(j + NT * m) * RowStride<N>::XC] : czero<cplx<T>>();
#pragma unroll
  for (int f = 0; f < 3; ++f) {
    if (f) __syncthreads();
    fft_run<T, N, E, false, false>(res[f], sbuf + c, TB, j, tw, SyncBlock());
  }
  if (pre) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
  }
  if (!ok) return;
  const int iy = col / Cfg<N>::MZP;
  const int kzi = col - iy * Cfg<N>::MZP;
  const int kyi = cfreq(iy, Cfg<N>::KC);
  const T ky = T(kyi), kz = T(kzi);
  constexpr int kc = Cfg<N>::KC;
  unsigned flags = 0;
#pragma unroll
  for (int m = 0; m < E; ++m) {
    const int n = j + NT * m;
    const int r = crow(n, N, kc);
    if (r < 0) continue;
    const int kxi = n <= kc ? n : n - N;
    const T kx = T(kxi);
    const int k2 = kxi * kxi + kyi * kyi + kzi * kzi;
    const long long idx = (long long)r * (Cfg<N>::MY * Cfg<N>::MZP) + col;
    const bool keep = (kzi <= kc) && (k2 <= kc * kc + kc);  // round(|k|) <= kc  (F:129)
    // forcing on shells kf_lo..kf_hi: factor[kint] * y  (F:253-264)
    T fac = T(0);
    if (keep && k2 <= A.kf_hi * A.kf_hi + A.kf_hi) {
      int s = 0;
      while (s * s + s < k2) ++s;  // s = round(sqrt(k2))
      if (s >= A.kf_lo) fac = T(A.factor[s]);
    }
    // the stage input; the second RK2 stage reads it only for the forcing and the slow manifold
    const bool need_y = MODE != UPD_RK2_2 || A.vk != nullptr || fac != T(0);
    cplx<T> y[3];
#pragma unroll
    for (int cc = 0; cc < 3; ++cc)
      y[cc] = !need_y ? czero<cplx<T>>()
                      : ((MODE != UPD_RK2_2 && pre) ? ybuf[(cc * Mx + r) * TB + c] : A.s1[cc * A.cs + idx]);
    cplx<T> rhs[3];
    cplx<T> kd = czero<cplx<T>>();  // (k . rhs) / k^2 before the projection
    if (keep) {
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) rhs[cc] = cadd(res[cc][m], cscale(y[cc], fac));
      if (k2 > 0) {  // pressure projection, invlap = -1/k^2 (F:309-316)
        const T inv = T(1) / T(k2);
        kd = cadd(cadd(cscale(rhs[0], kx), cscale(rhs[1], ky)), cscale(rhs[2], kz));
        kd = cscale(kd, inv);
        rhs[0] = csub(rhs[0], cscale(kd, kx));
        rhs[1] = csub(rhs[1], cscale(kd, ky));
        rhs[2] = csub(rhs[2], cscale(kd, kz));
      }
    } else {
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) rhs[cc] = czero<cplx<T>>();
    }
    if (A.vk) {
      // -i k pk = -k (k . rhs) / k^2 and -nu k^2 y: the reference's Du/Dt of the slow manifold
      const T lvs = A.visc * A.nu * T(k2);
      const T kk[3] = {kx, ky, kz};
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) {
        cplx<T> v = czero<cplx<T>>();
        if (keep) v = cadd(y[cc], cscale(cadd(cscale(kd, kk[cc]), cscale(y[cc], lvs)), A.tps));
        if (cc == 2 && k2 == 0) v.x -= A.vg;
        A.vk[cc * A.cs + idx] = v;
      }
    }
    const T h = A.h;
    if (MODE == UPD_RHS) {
      const T lv = A.visc * A.nu * T(k2);
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) A.s0[cc * A.cs + idx] = csub(rhs[cc], cscale(y[cc], lv));
    } else if (MODE == UPD_RK2_1) {
      const T Ef = keep ? A.ifac[k2] : T(0);
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) {
        cplx<T> us = cscale(cadd(y[cc], cscale(rhs[cc], h)), Ef);
        cplx<T> ac = cscale(cadd(y[cc], cscale(rhs[cc], T(0.5) * h)), Ef);
        A.s0[cc * A.cs + idx] = us;
        A.s2[cc * A.cs + idx] = ac;
      }
    } else if (MODE == UPD_RK2_2) {
      cplx<T> v[3];
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) {
        const cplx<T> acc = pre ? ybuf[(cc * Mx + r) * TB + c] : A.s2[cc * A.cs + idx];
        v[cc] = cadd(acc, cscale(rhs[cc], T(0.5) * h));
        if (!keep) v[cc] = czero<cplx<T>>();
        if (!(isfinite(v[cc].x) && isfinite(v[cc].y))) flags |= LD_STATUS_NONFINITE;
      }
      if (kzi > 0) epi_mode(v, kxi, kyi, kzi, kc, A.blowup, flags);
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) A.s0[cc * A.cs + idx] = v[cc];
    } else {
      // RK4 (F:341-360): ku = rhs - nu k^2 y ;  y = stage input
      const T lv = A.nu * T(k2);
      cplx<T> ku[3];
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) ku[cc] = csub(rhs[cc], cscale(y[cc], lv));
      if (MODE == UPD_RK4_4) {
        cplx<T> v[3];
#pragma unroll
        for (int cc = 0; cc < 3; ++cc) {
          v[cc] = cadd(A.s2[cc * A.cs + idx], cscale(ku[cc], h / T(6)));
          if (!(isfinite(v[cc].x) && isfinite(v[cc].y))) flags |= LD_STATUS_NONFINITE;
        }
        if (kzi > 0) epi_mode(v, kxi, kyi, kzi, kc, A.blowup, flags);
#pragma unroll
        for (int cc = 0; cc < 3; ++cc) A.s0[cc * A.cs + idx] = v[cc];
      } else {
#pragma unroll
        for (int cc = 0; cc < 3; ++cc) {
          const long long o = cc * A.cs + idx;
          if (MODE == UPD_RK4_1) {
            cplx<T> un = y[cc];
            A.s2[o] = cadd(un, cscale(ku[cc], h / T(6)));
            A.s3[o] = cadd(un, cscale(ku[cc], h / T(2)));
          } else {  // UPD_RK4_2, UPD_RK4_3
            cplx<T> un = A.s0[o];
            A.s2[o] = cadd(A.s2[o], cscale(ku[cc], h / T(3)));
            A.s3[o] = cadd(un, cscale(ku[cc], MODE == UPD_RK4_2 ? h / T(2) : h));
          }
        }
      }
    }
  }
  if (flags) atomicOr(A.status, flags);
}

// ------------------------------------------------------------------------------------------
// z passes (contiguous axis): NT threads per row unit, inside one warp
// ------------------------------------------------------------------------------------------
// Row unit of this lane within its warp, and the lane within the row.
template <int N, int E> __device__ __forceinline__ void z_lane(int& unit, int& j) {
  constexpr int NT = N / E, R = 32 / NT;
  const int lane = threadIdx.x & 31;
  unit = lane / NT;
  j = lane - unit * NT;
  if (R * NT < 32 && unit >= R) unit = 0;  // the lanes left over repeat the first ones of unit 0
  __builtin_assume(j >= 0 && j < NT);
}

// Hermitian-extended load of Y[k] = A[k] + i B[k] (k = j + NT m), A/B spectral rows with Kin
// valid coefficients; imaginary parts of k = 0 and k = N/2 are dropped (pocketfft c2r).
template <typename T, int N, int E>
__device__ __forceinline__ void zload_pair(cplx<T>* a, const cplx<T>* A, const cplx<T>* B, int Kin,
                                           int j, T s) {
  constexpr int NT = N / E;
#pragma unroll
  for (int m = 0; m < E; ++m) {
    const int k = j + NT * m;
    T yr = 0, yi = 0;
    if (k == 0 || k == N / 2) {
      if (k < Kin) {
        yr = A[k].x;
        if (B) yi = B[k].x;
      }
    } else if (k < N / 2) {
      if (k < Kin) {
        cplx<T> av = A[k];
        cplx<T> bv = B ? B[k] : czero<cplx<T>>();
        yr = av.x - bv.y;
        yi = av.y + bv.x;
      }
    } else {
      const int kk = N - k;
      if (kk < Kin) {
        cplx<T> av = A[kk];
        cplx<T> bv = B ? B[kk] : czero<cplx<T>>();
        yr = av.x + bv.y;
        yi = bv.x - av.y;
      }
    }
    a[m] = cmk(yr * s, yi * s);
  }
}

// After a forward FFT of (a + i b): split Y into A[k], B[k] for k < Kout (zero for k >= Kval; B null:
// A alone).  The mirrored coefficients come by shuffles: Y[N - k] (Y[0] for k = 0) is register
// E - 1 - m of lane NT - j (j > 0), or register (E - m) % E of lane 0 (j = 0).
template <typename T, int N, int E>
__device__ __forceinline__ void zstore_pair(const cplx<T>* a, cplx<T>* A, cplx<T>* B, int Kout, int Kval, int j,
                                            bool ok) {
  constexpr int NT = N / E;
  if (B == nullptr) {
#pragma unroll
    for (int m = 0; m < E; ++m) {
      const int k = j + NT * m;
      if (ok && k < Kout) A[k] = k < Kval ? a[m] : czero<cplx<T>>();
    }
    return;
  }
  const int lane = threadIdx.x & 31, src = j == 0 ? lane : lane - j + NT - j;
#pragma unroll
  for (int m = 0; m < E; ++m) {
    const int k = j + NT * m;
    if (NT * m >= Kout) continue;  // uniform
    cplx<T> z;
    z.x = __shfl_sync(0xffffffffu, a[E - 1 - m].x, src);
    z.y = __shfl_sync(0xffffffffu, a[E - 1 - m].y, src);
    if (j == 0) z = a[(E - m) % E];
    if (ok && k < Kout) {
      cplx<T> ra = czero<cplx<T>>(), rb = czero<cplx<T>>();
      if (k < Kval) {
        const cplx<T> y = a[m];
        ra = cmk(T(0.5) * (y.x + z.x), T(0.5) * (y.y - z.y));
        rb = cmk(T(0.5) * (y.y + z.y), T(-0.5) * (y.x - z.x));
      }
      A[k] = ra;
      B[k] = rb;
    }
  }
}

// Row unit of this thread in a one-shot z kernel: unit within the block, lane j within the row,
// and whether this lane's stores are its own (lanes left over repeat others).
template <typename T, int N> __device__ __forceinline__ void z_unit(int& unit, int& j, bool& own) {
  constexpr int E = ZCfg<T, N>::E1, NT = N / E, R = 32 / NT;
  z_lane<N, E>(unit, j);
  unit += (threadIdx.x >> 5) * R;
  own = (threadIdx.x & 31) < R * NT;
}

// Generic C2R: pairs of rows (2p, 2p+1) of nrows rows per field; spectral rows of stride ss
// (Kin valid), real rows of stride N.  Scale s (1/N^3 for the 3D inverse).
template <typename T, int N>
__global__ void __launch_bounds__(256)
k_z_c2r(const cplx<T>* __restrict__ X, T* __restrict__ x, long long nrows, int ss, int Kin, T s,
        long long xfs, long long Xfs, const cplx<T>* __restrict__ tw) {
  using Z = ZCfg<T, N>;
  constexpr int E = Z::E1, NT = N / E;
  grid_dep();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* sbuf = reinterpret_cast<cplx<T>*>(smem_raw);
  int unit, j;
  bool own;
  z_unit<T, N>(unit, j, own);
  cplx<T>* sb = sbuf + unit * Z::ZBUF1;
  const long long pair = (long long)blockIdx.x * Z::UNITS1 + unit;
  const int f = blockIdx.y;
  const bool ok = 2 * pair < nrows;
  const long long r0 = ok ? 2 * pair : 0;
  const cplx<T>* A = X + f * Xfs + r0 * ss;
  const cplx<T>* B = (r0 + 1 < nrows) ? A + ss : nullptr;
  cplx<T> a[E];
  if (ok) zload_pair<T, N, E>(a, A, B, Kin, j, s);
  else for (int m = 0; m < E; ++m) a[m] = czero<cplx<T>>();
  fft_run<T, N, E, true, true>(a, sb, 1, j, tw, SyncWarp());
  if (!ok || !own) return;
  T* xa = x + f * xfs + r0 * N;
#pragma unroll
  for (int m = 0; m < E; ++m) {
    const int n = j + NT * m;
    xa[n] = a[m].x;
    if (B) xa[N + n] = a[m].y;
  }
}

// Generic R2C: pairs of real rows -> spectral rows (stride ss), Kout stored (zeros for k >= Kval).
template <typename T, int N>
__global__ void __launch_bounds__(256)
k_z_r2c(const T* __restrict__ x, cplx<T>* __restrict__ X, long long nrows, int ss, int Kout,
        int Kval, long long xfs, long long Xfs, const cplx<T>* __restrict__ tw) {
  using Z = ZCfg<T, N>;
  constexpr int E = Z::E1, NT = N / E;
  grid_dep();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* sbuf = reinterpret_cast<cplx<T>*>(smem_raw);
  int unit, j;
  bool own;
  z_unit<T, N>(unit, j, own);
  cplx<T>* sb = sbuf + unit * Z::ZBUF1;
  const long long pair = (long long)blockIdx.x * Z::UNITS1 + unit;
  const int f = blockIdx.y;
  const bool ok = 2 * pair < nrows;
  const long long r0 = ok ? 2 * pair : 0;
  const bool hasb = r0 + 1 < nrows;
  const T* xa = x + f * xfs + r0 * N;
  cplx<T> a[E];
#pragma unroll
  for (int m = 0; m < E; ++m) {
    const int n = j + NT * m;
    a[m] = ok ? cmk(xa[n], hasb ? xa[N + n] : T(0)) : czero<cplx<T>>();
  }
  fft_run<T, N, E, false, true>(a, sb, 1, j, tw, SyncWarp());
  cplx<T>* A = X + f * Xfs + r0 * ss;
  zstore_pair<T, N, E>(a, A, hasb ? A + ss : nullptr, Kout, Kval, j, ok && own);
}

// The products and forward half of one row of the fused z pass, from the three inverse transforms
// p0 = (u_x, u_y), p1 = (u_z, w_x), p2 = (w_y, w_z): optional store of physical u, u x w
// (F:299-301), R2C of the three products into A, B, C (kz < Kout stored, zero beyond Kin).
template <typename T, int N, class Tw>
__device__ __forceinline__ void zcross_forward(cplx<T>* p0, cplx<T>* p1, const cplx<T>* p2, cplx<T>* sb, cplx<T>* A,
                                               cplx<T>* B, cplx<T>* C, long long row, T* uphys, int ulayout, int Kout,
                                               int Kin, int j, bool own, const Tw& tw) {
  constexpr int E = ZCfg<T, N>::E, NT = ZCfg<T, N>::NT;
  if (uphys && own) {
    if (ulayout == 0) {  // planar (3, N, N, N)
      const long long NN3 = (long long)N * N * N;
#pragma unroll
      for (int m = 0; m < E; ++m) {
        const int n = j + NT * m;
        uphys[row * N + n] = p0[m].x;
        uphys[NN3 + row * N + n] = p0[m].y;
        uphys[2 * NN3 + row * N + n] = p1[m].x;
      }
    } else {  // interleaved (N, N, N, 4): (u, v, w, 0) per grid point
      vec4<T>* u4 = reinterpret_cast<vec4<T>*>(uphys);
#pragma unroll
      for (int m = 0; m < E; ++m) {
        const int n = j + NT * m;
        u4[row * N + n] = mk4<T>(p0[m].x, p0[m].y, p1[m].x, T(0));
      }
    }
  }
  // products: (u x w) = (uy wz - uz wy, uz wx - ux wz, ux wy - uy wx)
#pragma unroll
  for (int m = 0; m < E; ++m) {
    const T ux = p0[m].x, uy = p0[m].y, uz = p1[m].x, wx = p1[m].y, wy = p2[m].x, wz = p2[m].y;
    p0[m] = cmk(wz * uy - wy * uz, wx * uz - wz * ux);
    p1[m] = cmk(wy * ux - wx * uy, T(0));
  }
  fft_run<T, N, E, false, true>(p0, sb, 1, j, tw, SyncWarp());
  zstore_pair<T, N, E>(p0, A, B, Kout, Kin, j, own);
  __syncwarp();
  fft_run<T, N, E, false, true>(p1, sb, 1, j, tw, SyncWarp());
  __syncwarp();  // C may lie in the exchange buffer
  zstore_pair<T, N, E>(p1, C, (cplx<T>*)nullptr, Kout, Kin, j, own);
}

// The fused z pass of an FP32 row of power-of-two length with packed transforms: (u_x, u_y) and
// (u_z, w_x) transform side by side, (w_y, w_z) alone, the products (two and one) side by side.
// Hermitian-extended load of two pairs of fields (A0, B0), (A1, B1), as zload_pair.
template <int N, int E>
__device__ __forceinline__ void zload_pair2(C2* a, const float2* A0, const float2* B0, const float2* A1, const float2* B1,
                                            int Kin, int j, float s) {
  float2 t0[E], t1[E];
  zload_pair<float, N, E>(t0, A0, B0, Kin, j, s);
  zload_pair<float, N, E>(t1, A1, B1, Kin, j, s);
#pragma unroll
  for (int m = 0; m < E; ++m) a[m] = C2{make_float2(t0[m].x, t1[m].x), make_float2(t0[m].y, t1[m].y)};
}

// zcross_forward from the packed inverse transforms p = ((u_x, u_z), (u_y, w_x)) and p2 = (w_y, w_z).
template <int N, int E>
__device__ __forceinline__ void zcross_forward2(C2* p, const float2* p2, float4* sb, float2* A, float2* B, float2* C,
                                                long long row, float* uphys, int ulayout, int Kout, int Kin, int j,
                                                bool own, const TwLane2<N, E>& tw) {
  constexpr int NT = N / E;
  if (uphys && own) {
    const long long NN3 = (long long)N * N * N;
#pragma unroll
    for (int m = 0; m < E; ++m) {
      const int n = j + NT * m;
      if (ulayout == 0) {  // planar (3, N, N, N)
        uphys[row * N + n] = p[m].x.x;
        uphys[NN3 + row * N + n] = p[m].y.x;
        uphys[2 * NN3 + row * N + n] = p[m].x.y;
      } else {  // interleaved (N, N, N, 4)
        reinterpret_cast<float4*>(uphys)[row * N + n] = make_float4(p[m].x.x, p[m].y.x, p[m].x.y, 0.f);
      }
    }
  }
#pragma unroll
  for (int m = 0; m < E; ++m) {
    const float ux = p[m].x.x, uy = p[m].y.x, uz = p[m].x.y, wx = p[m].y.y, wy = p2[m].x, wz = p2[m].y;
    p[m] = C2{make_float2(wz * uy - wy * uz, wy * ux - wx * uy), make_float2(wx * uz - wz * ux, 0.f)};
  }
  fft_run2<N, E, false, 1>(p, sb, j, tw, SyncWarp());
  SyncWarp()();  // A, B, C may lie in the exchange buffer
  float2 t[E];
#pragma unroll
  for (int m = 0; m < E; ++m) t[m] = make_float2(p[m].x.x, p[m].y.x);
  zstore_pair<float, N, E>(t, A, B, Kout, Kin, j, own);
#pragma unroll
  for (int m = 0; m < E; ++m) t[m] = make_float2(p[m].x.y, p[m].y.y);
  zstore_pair<float, N, E>(t, C, (float2*)nullptr, Kout, Kin, j, own);
}

// Fused z pass: persistent warps walk groups of R rows with a
// stride.  The six field rows of the warp's next group are brought into shared memory by bulk
// asynchronous copies (the TMA engine), one mbarrier per pair of fields, each issued as soon as
// the current group's pair sits in registers, so that the transforms cover it.  Waits are bounded:
// a wait gives up after wait_limit polls (the plan's setting); the warp then raises
// LD_STATUS_WAIT_TIMEOUT, drains its copies in flight (bounded by kWaitLimit) and returns.  With
// `stall` set (a test of that path) each warp first waits on a fourth mbarrier that nothing
// completes, so the wait runs out while the warp's first copies are in flight.
// Shared memory: per warp 6 R rows of Mzp and R exchange rows, then the twiddles in lane order
// (unless they are in registers), then 4 mbarriers per warp.
constexpr unsigned kWaitLimit = 1u << 24;

template <typename T, int N> struct ZPipe {
  using Z = ZCfg<T, N>;
  static constexpr bool PACK = Z::PACK;
  static constexpr int WARPS = 4;
  static constexpr int STAGE = 6 * Z::R * Cfg<N>::MZP;  // elements per warp
  static constexpr int EX = PACK ? 2 * Z::R * N : Z::R * Z::ZBUF;
  static constexpr int TW = PACK ? 2 * TwLane<T, N, Z::E>::ELEMS : (Z::TWREG ? 0 : TwLane<T, N, Z::E>::ELEMS);
  static constexpr size_t SMEM = sizeof(cplx<T>) * ((size_t)WARPS * (STAGE + EX) + TW) + 32 * WARPS;
  // CTAs per SM asked of the compiler: 3 E complex values and what a transform needs besides
  static constexpr int MINB = sizeof(T) == 4 && N != 512 ? 3 : 2;
};

template <typename T, int N>
__global__ void __launch_bounds__(32 * ZPipe<T, N>::WARPS, ZPipe<T, N>::MINB)
k_z_cross_pipe(const cplx<T>* __restrict__ W, cplx<T>* __restrict__ P, T* __restrict__ uphys, int ulayout, T s,
               const cplx<T>* __restrict__ tw, unsigned* status, unsigned wait_limit, int stall, long long NR) {
  using Z = ZCfg<T, N>;
  using ZP = ZPipe<T, N>;
  constexpr int E = Z::E, R = Z::R, WARPS = ZP::WARPS;
  constexpr int MZ = Cfg<N>::MZP, KIN = Cfg<N>::KC + 1;  // the plan's cube (checked at launch)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int unit, j;
  z_lane<N, E>(unit, j);
  const bool own = lane < R * Z::NT;
  cplx<T>* base = reinterpret_cast<cplx<T>*>(smem_raw);
  cplx<T>* stage = base + warp * ZP::STAGE;
  cplx<T>* sb = base + WARPS * ZP::STAGE + warp * ZP::EX + unit * (ZP::PACK ? 2 * N : Z::ZBUF);
  cplx<T>* tws = base + WARPS * (ZP::STAGE + ZP::EX);
  uint64_t* bars = reinterpret_cast<uint64_t*>(tws + ZP::TW) + 4 * warp;
  const long long fs = NR * MZ;
  const long long stride = (long long)gridDim.x * WARPS * R;
  long long row = ((long long)blockIdx.x * WARPS + warp) * R;  // NR is a multiple of R
  if (lane == 0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) mbar_init(&bars[q], 1);
    mbar_init_fence();
  }
  typename std::conditional<ZP::PACK, TwLane2<N, E>,
                            typename std::conditional<Z::TWREG, TwRegs<T, N, E>, TwLane<T, N, E>>::type>::type twr;
  if constexpr (!ZP::PACK && Z::TWREG) {
    twr.load(tw, j);
  } else {
    using Table = decltype(twr);
    using Elem = typename std::remove_const<typename std::remove_pointer<decltype(twr.p)>::type>::type;
    Elem* t = reinterpret_cast<Elem*>(tws);
    Table::fill(t, tw, threadIdx.x, 32 * WARPS);
    twr.p = t + j;
    __syncthreads();
  }
  grid_dep();
  __syncwarp();
  auto issue = [&](long long r, int q) {  // fields 2 q, 2 q + 1 of rows r .. r + R - 1
    if (lane == 0) {
      constexpr unsigned bytes = (unsigned)(R * MZ * sizeof(cplx<T>));
      fence_proxy_async();
      mbar_expect_tx(&bars[q], 2u * bytes);
      bulk_g2s(stage + 2 * q * R * MZ, W + 2 * q * fs + r * MZ, bytes, &bars[q]);
      bulk_g2s(stage + (2 * q + 1) * R * MZ, W + (2 * q + 1) * fs + r * MZ, bytes, &bars[q]);
    }
  };
  if (row < NR) {
    issue(row, 0);
    issue(row, 1);
    issue(row, 2);
  }
  if (stall && row < NR && !__all_sync(0xffffffffu, mbar_wait_bounded(&bars[3], 0u, wait_limit))) {
    if (lane == 0) atomicOr(status, LD_STATUS_WAIT_TIMEOUT);
    for (int q = 0; q < 3; ++q) mbar_wait_bounded(&bars[q], 0u, kWaitLimit);  // the first rows' copies are in flight
    return;
  }
  unsigned ph = 0;
  // waits for pair q of this group; false after a time-out (pairs before q already belong to the next
  // group's phase when there is one and `moved`)
  auto arrived = [&](int q, long long next, bool moved) -> bool {
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&bars[q], ph, wait_limit))) {
      if (lane == 0) atomicOr(status, LD_STATUS_WAIT_TIMEOUT);
      for (int b = 0; b < 3; ++b)
        if (b >= q) mbar_wait_bounded(&bars[b], ph, kWaitLimit);
        else if (moved && next < NR) mbar_wait_bounded(&bars[b], ph ^ 1u, kWaitLimit);
      return false;
    }
    return true;
  };
  // pair q of this group into registers, then its next group's copy
  auto take = [&](cplx<T>* a, int q, long long next) -> bool {
    if (!arrived(q, next, true)) return false;
    const cplx<T>* A = stage + (2 * q * R + unit) * MZ;
    zload_pair<T, N, E>(a, A, A + R * MZ, KIN, j, s);
    __syncwarp();  // every lane has read the pair
    if (next < NR) issue(next, q);
    return true;
  };
  for (; row < NR; row += stride, ph ^= 1u) {
    const long long next = row + stride;
    cplx<T>* out = P + (row + unit) * MZ;
    if constexpr (ZP::PACK) {
      C2 p[E];
      cplx<T> p2[E];
      float4* sb4 = reinterpret_cast<float4*>(sb);
      if (!arrived(0, next, false) || !arrived(1, next, false)) return;
      const cplx<T>* A = stage + unit * MZ;
      zload_pair2<N, E>(p, A, A + R * MZ, A + 2 * R * MZ, A + 3 * R * MZ, KIN, j, s);
      __syncwarp();  // every lane has read the pairs
      if (next < NR) {
        issue(next, 0);
        issue(next, 1);
      }
      fft_run2<N, E, true, 1>(p, sb4, j, twr, SyncWarp());
      if (!take(p2, 2, next)) return;  // (w_y, w_z); its __syncwarp frees the exchange buffer
      fft_run<T, N, E, true, true>(p2, sb, 1, j, twr, SyncWarp());
      __syncwarp();
      zcross_forward2<N, E>(p, p2, sb4, out, out + fs, out + 2 * fs, row + unit, uphys, ulayout, MZ, KIN, j, own, twr);
      __syncwarp();  // every lane is done with the exchange buffer
    } else {
      cplx<T> p0[E], p1[E], p2[E];
      if (!take(p0, 0, next)) return;  // (u_x, u_y)
      fft_run<T, N, E, true, true>(p0, sb, 1, j, twr, SyncWarp());
      if (!take(p1, 1, next)) return;  // (u_z, w_x); its __syncwarp frees the exchange buffer
      fft_run<T, N, E, true, true>(p1, sb, 1, j, twr, SyncWarp());
      if (!take(p2, 2, next)) return;  // (w_y, w_z)
      fft_run<T, N, E, true, true>(p2, sb, 1, j, twr, SyncWarp());
      __syncwarp();
      zcross_forward<T, N>(p0, p1, p2, sb, out, out + fs, out + 2 * fs, row + unit, uphys, ulayout, MZ, KIN, j, own,
                           twr);
      __syncwarp();  // every lane is done with the exchange buffer
    }
  }
}

// ------------------------------------------------------------------------------------------
// plane pass of small grids: inverse y, fused z and forward y of one x plane in shared memory
// ------------------------------------------------------------------------------------------
// The six fields' columns kz <= kc of one (box, x) plane fit one SM's shared memory for N <= 64
// (FP32 also 96): one block transforms them along y, takes the rows through the fused z pass and
// the three products back along y, so that neither the (6, N, N, Mzp) nor the (3, N, N, Mzp)
// intermediate goes through global memory and three launches become one.  Larger planes do not
// fit (128^2 in FP32: 270 KB) and take the separate passes.
// Row y of the plane holds its NC = 6 (kc + 1) values, columns (field, kz) contiguous; the z
// transforms of a row exchange inside the row, past the two products stored first.  The row pitch
// is NT mod 16 elements (FP32; mod 8 in FP64), so that the rows a half-warp (quarter-warp) works on
// start NT bank groups apart.  Along y a column of length N = R1 R2 takes two steps: R2 threads of
// radix R1 over y = j + R2 m, the twiddles W^(j k), then R1 threads of radix R2 over j; each step
// reads and writes the same places, so one block barrier separates them.
template <typename T, int N> struct PlaneCfg {
  static constexpr bool OK = N == 16 || N == 32 || N == 64 || (N == 96 && sizeof(T) == 4);
  static constexpr int M = OK ? N : 64;
  using Z = ZCfg<T, M>;
  static constexpr int KIN = Cfg<M>::KC + 1, NC = 6 * KIN;
  static constexpr int R1 = M == 96 ? 12 : (M == 16 ? 4 : 8), R2 = M / R1;
  static constexpr int MOD = sizeof(T) == 4 ? 16 : 8;
  static constexpr int LEAST = NC > 2 * KIN + Z::ZBUF ? NC : 2 * KIN + Z::ZBUF;
  static constexpr int PITCH = LEAST + ((Z::NT - LEAST) % MOD + MOD) % MOD;
  static constexpr int THREADS = M == 96 ? 384 : (M == 16 ? 128 : 256);
  static constexpr int TWZ = TwLane<T, M, Z::E>::ELEMS;
  static constexpr size_t SMEM = sizeof(cplx<T>) * ((size_t)M * PITCH + TWZ + M);
};

// W: (6, NO, My, Mzp) in (columns kz <= kc read), P: (3, NO, My, Mzp) out, NO = boxes x N planes
// MINB: blocks per SM asked of the compiler.  Many planes of FP32 64 run three per SM at 80 registers
// (16 boxes, five ensemble steps: 1.50 ms, 1.56 at 96 registers); a few run faster at 96 (one box:
// right-hand side 21.4 us, 26.2 at 80; four boxes: 621 and 626 us for five steps).
template <typename T, int N, int MINB>
__global__ void __launch_bounds__(PlaneCfg<T, N>::THREADS, MINB)
k_plane(const cplx<T>* __restrict__ W, cplx<T>* __restrict__ P, T* __restrict__ uphys, int ulayout, T s,
        const cplx<T>* __restrict__ tw, long long NO) {
  using C = PlaneCfg<T, N>;
  using Z = ZCfg<T, N>;
  constexpr int R1 = C::R1, R2 = C::R2, KIN = C::KIN, PITCH = C::PITCH, THREADS = C::THREADS, E = Z::E, NT = Z::NT;
  constexpr int MY = Cfg<N>::MY, MZ = Cfg<N>::MZP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* F = reinterpret_cast<cplx<T>*>(smem_raw);
  cplx<T>* twz = F + N * PITCH;
  cplx<T>* twy = twz + C::TWZ;
  const int tid = threadIdx.x;
  const long long o = blockIdx.x;
  for (int i = tid; i < N; i += THREADS) twy[i] = tw[i];
  TwLane<T, N, E>::fill(twz, tw, tid, THREADS);
  grid_dep();
  __syncthreads();
  // y inverse, first step: cube rows from global memory
  for (int t = tid; t < C::NC * R2; t += THREADS) {
    const int j = t / C::NC, col = t - j * C::NC, f = col / KIN, c = col - f * KIN;
    const cplx<T>* src = W + (f * NO + o) * (MY * MZ) + c;
    cplx<T> a[R1];
#pragma unroll
    for (int m = 0; m < R1; ++m) {
      const int r = crow(j + R2 * m, N, Cfg<N>::KC);
      a[m] = r < 0 ? czero<cplx<T>>() : src[r * MZ];
    }
    dft_any<T, R1, true>(a);
#pragma unroll
    for (int k = 0; k < R1; ++k)
      F[(k + R1 * j) * PITCH + col] = k ? cmul(a[k], twid<T, true>(twy, j * k)) : a[k];
  }
  __syncthreads();
  for (int t = tid; t < C::NC * R1; t += THREADS) {
    const int k = t / C::NC, col = t - k * C::NC;
    cplx<T> a[R2];
#pragma unroll
    for (int j = 0; j < R2; ++j) a[j] = F[(k + R1 * j) * PITCH + col];
    dft_any<T, R2, true>(a);
#pragma unroll
    for (int j = 0; j < R2; ++j) F[(k + R1 * j) * PITCH + col] = a[j];
  }
  __syncthreads();
  // z rows: NT lanes each, whole warps
  static_assert(N * NT % 32 == 0 && 32 % NT == 0, "whole rows per warp");
  for (int t = tid; t < N * NT; t += THREADS) {
    const int y = t / NT;
    int j = t % NT;
    __builtin_assume(j >= 0 && j < NT);
    cplx<T>* row = F + y * PITCH;
    cplx<T>* sb = row + 2 * KIN;
    TwLane<T, N, E> twr;
    twr.p = twz + j;
    cplx<T> p0[E], p1[E], p2[E];
    zload_pair<T, N, E>(p0, row, row + KIN, KIN, j, s);                // (u_x, u_y)
    zload_pair<T, N, E>(p1, row + 2 * KIN, row + 3 * KIN, KIN, j, s);  // (u_z, w_x)
    zload_pair<T, N, E>(p2, row + 4 * KIN, row + 5 * KIN, KIN, j, s);  // (w_y, w_z)
    __syncwarp();
    fft_run<T, N, E, true, true>(p0, sb, 1, j, twr, SyncWarp());
    __syncwarp();
    fft_run<T, N, E, true, true>(p1, sb, 1, j, twr, SyncWarp());
    __syncwarp();
    fft_run<T, N, E, true, true>(p2, sb, 1, j, twr, SyncWarp());
    __syncwarp();
    zcross_forward<T, N>(p0, p1, p2, sb, row, row + KIN, row + 2 * KIN, o * N + y, uphys, ulayout, KIN, KIN, j, true,
                         twr);
  }
  __syncthreads();
  // y forward of the three products
  constexpr int NP = 3 * KIN;
  for (int t = tid; t < NP * R2; t += THREADS) {
    const int j = t / NP, col = t - j * NP;
    cplx<T> a[R1];
#pragma unroll
    for (int m = 0; m < R1; ++m) a[m] = F[(j + R2 * m) * PITCH + col];
    dft_any<T, R1, false>(a);
#pragma unroll
    for (int k = 0; k < R1; ++k)
      F[(j + R2 * k) * PITCH + col] = k ? cmul(a[k], twid<T, false>(twy, j * k)) : a[k];
  }
  __syncthreads();
  for (int t = tid; t < 3 * MZ * R1; t += THREADS) {  // the padding columns are written too: whole sectors
    const int k = t / (3 * MZ), col = t - k * (3 * MZ), f = col / MZ, c = col - f * MZ;
    cplx<T> a[R2];
#pragma unroll
    for (int j = 0; j < R2; ++j) a[j] = c < KIN ? F[(j + R2 * k) * PITCH + f * KIN + c] : czero<cplx<T>>();
    dft_any<T, R2, false>(a);
    cplx<T>* dst = P + (f * NO + o) * (MY * MZ) + c;
#pragma unroll
    for (int j = 0; j < R2; ++j) {
      const int r = crow(k + R1 * j, N, Cfg<N>::KC);
      if (r >= 0) dst[r * MZ] = a[j];
    }
  }
}

// ------------------------------------------------------------------------------------------
// cube <-> reference layout, spectra, forcing, epilogue
// ------------------------------------------------------------------------------------------
template <typename T>
__global__ void k_to_cube(const cplx<T>* __restrict__ full, cplx<T>* __restrict__ cube, int N, int kc,
                          int My, int Mzp, long long total) {
  const int Nf = N / 2 + 1;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const long long per = (long long)My * My * Mzp;
    const int comp = (int)(e / per);
    long long r = e - comp * per;
    const int ix = (int)(r / ((long long)My * Mzp));
    r -= (long long)ix * My * Mzp;
    const int iy = (int)(r / Mzp);
    const int kz = (int)(r - (long long)iy * Mzp);
    const int kx = cfreq(ix, kc), ky = cfreq(iy, kc);
    const int k2 = kx * kx + ky * ky + kz * kz;
    cplx<T> v = czero<cplx<T>>();
    if (kz <= kc && k2 <= kc * kc + kc) {
      const int nx = kx < 0 ? kx + N : kx, ny = ky < 0 ? ky + N : ky;
      v = full[(long long)comp * N * N * Nf + ((long long)nx * N + ny) * Nf + kz];
    }
    cube[e] = v;
  }
}

template <typename T>
__global__ void k_from_cube(const cplx<T>* __restrict__ cube, cplx<T>* __restrict__ full, int N, int kc,
                            int My, int Mzp, long long total) {
  const int Nf = N / 2 + 1;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const long long per = (long long)N * N * Nf;
    const int comp = (int)(e / per);
    long long r = e - comp * per;
    const int nx = (int)(r / ((long long)N * Nf));
    r -= (long long)nx * N * Nf;
    const int ny = (int)(r / Nf);
    const int kz = (int)(r - (long long)ny * Nf);
    const int ix = crow(nx, N, kc), iy = crow(ny, N, kc);
    cplx<T> v = czero<cplx<T>>();
    if (ix >= 0 && iy >= 0 && kz <= kc)
      v = cube[(long long)comp * My * My * Mzp + ((long long)ix * My + iy) * Mzp + kz];
    full[e] = v;
  }
}

// End-of-step epilogue (F:596-620) on the cube: symmetrise kz = 0 (the irfft->rfft round trip),
// div-free projection, NaN and blow-up tests.  One thread per (kx, ky, kz) column element; the
// kz = 0 pair (k, -k) is handled by the lexicographically smaller member.
template <typename T>
__global__ void k_epilogue(cplx<T>* __restrict__ u, long long cs, int kc, int My, int Mzp,
                           T blowup, unsigned* status) {
  u += blockIdx.y * 3 * cs;  // box of a multi-box plan
  const long long total = (long long)My * My * Mzp;
  unsigned flags = 0;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int ix = (int)(e / ((long long)My * Mzp));
    const long long r = e - (long long)ix * My * Mzp;
    const int iy = (int)(r / Mzp);
    const int kz = (int)(r - (long long)iy * Mzp);
    const int kx = cfreq(ix, kc), ky = cfreq(iy, kc);
    cplx<T> v[3];
    if (kz == 0) {
      // partner -k
      const int jx = kx == 0 ? 0 : (-kx < 0 ? -kx + 2 * kc + 1 : -kx);
      const int jy = ky == 0 ? 0 : (-ky < 0 ? -ky + 2 * kc + 1 : -ky);
      const bool mine = (kx > 0) || (kx == 0 && ky >= 0);
      if (!mine) continue;
      const long long ep = ((long long)jx * My + jy) * Mzp;
      cplx<T> w[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        cplx<T> a = u[c * cs + e], b = u[c * cs + ep];
        v[c] = cmk(T(0.5) * (a.x + b.x), T(0.5) * (a.y - b.y));
        w[c] = cconj(v[c]);
      }
      // project both members with their own k
      for (int side = 0; side < 2; ++side) {
        cplx<T>* q = side ? w : v;
        const T qx = T(side ? -kx : kx), qy = T(side ? -ky : ky);
        const int k2 = kx * kx + ky * ky;
        if (k2 > 0 && k2 <= kc * kc + kc) {
          cplx<T> kd = cscale(cadd(cscale(q[0], qx), cscale(q[1], qy)), T(1) / T(k2));
          q[0] = csub(q[0], cscale(kd, qx));
          q[1] = csub(q[1], cscale(kd, qy));
        }
        if (k2 > kc * kc + kc) { q[0] = q[1] = q[2] = czero<cplx<T>>(); }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        u[c * cs + e] = v[c];
        if (ep != e) u[c * cs + ep] = w[c];
        if (!(isfinite(v[c].x) && isfinite(v[c].y))) flags |= LD_STATUS_NONFINITE;
        if (v[c].x > blowup || w[c].x > blowup) flags |= LD_STATUS_BLOWUP;
      }
      continue;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] = u[c * cs + e];
    const int k2 = kx * kx + ky * ky + kz * kz;
    if (kz <= kc && k2 <= kc * kc + kc) {
      const T qx = T(kx), qy = T(ky), qz = T(kz);
      cplx<T> kd = cscale(cadd(cadd(cscale(v[0], qx), cscale(v[1], qy)), cscale(v[2], qz)), T(1) / T(k2));
      v[0] = csub(v[0], cscale(kd, qx));
      v[1] = csub(v[1], cscale(kd, qy));
      v[2] = csub(v[2], cscale(kd, qz));
    } else {
      v[0] = v[1] = v[2] = czero<cplx<T>>();
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      u[c * cs + e] = v[c];
      if (!(isfinite(v[c].x) && isfinite(v[c].y))) flags |= LD_STATUS_NONFINITE;
      if (v[c].x > blowup) flags |= LD_STATUS_BLOWUP;
    }
  }
  if (flags) atomicOr(status, flags);
}

// The step epilogue on the kz = 0 plane only (k_epilogue's kz = 0 branch): for a state whose
// kz > 0 modes the final update stage has already projected and checked.
template <typename T>
__global__ void k_epilogue_plane0(cplx<T>* __restrict__ u, long long cs, int kc, int My, int Mzp, T blowup,
                                  unsigned* status) {
  grid_dep();
  u += blockIdx.y * 3 * cs;  // box of a multi-box plan
  const long long total = (long long)My * My;
  unsigned flags = 0;
  for (long long e2 = blockIdx.x * (long long)blockDim.x + threadIdx.x; e2 < total; e2 += (long long)gridDim.x * blockDim.x) {
    const int ix = (int)(e2 / My), iy = (int)(e2 - (long long)ix * My);
    const int kx = cfreq(ix, kc), ky = cfreq(iy, kc);
    const long long e = e2 * Mzp;
    const int jx = kx == 0 ? 0 : (-kx < 0 ? -kx + 2 * kc + 1 : -kx);
    const int jy = ky == 0 ? 0 : (-ky < 0 ? -ky + 2 * kc + 1 : -ky);
    const bool mine = (kx > 0) || (kx == 0 && ky >= 0);
    if (!mine) continue;
    const long long ep = ((long long)jx * My + jy) * Mzp;
    cplx<T> v[3], w[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      cplx<T> a = u[c * cs + e], b = u[c * cs + ep];
      v[c] = cmk(T(0.5) * (a.x + b.x), T(0.5) * (a.y - b.y));
      w[c] = cconj(v[c]);
    }
    for (int side = 0; side < 2; ++side) {
      cplx<T>* q = side ? w : v;
      const T qx = T(side ? -kx : kx), qy = T(side ? -ky : ky);
      const int k2 = kx * kx + ky * ky;
      if (k2 > 0 && k2 <= kc * kc + kc) {
        cplx<T> kd = cscale(cadd(cscale(q[0], qx), cscale(q[1], qy)), T(1) / T(k2));
        q[0] = csub(q[0], cscale(kd, qx));
        q[1] = csub(q[1], cscale(kd, qy));
      }
      if (k2 > kc * kc + kc) { q[0] = q[1] = q[2] = czero<cplx<T>>(); }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      u[c * cs + e] = v[c];
      if (ep != e) u[c * cs + ep] = w[c];
      if (!(isfinite(v[c].x) && isfinite(v[c].y))) flags |= LD_STATUS_NONFINITE;
      if (v[c].x > blowup || w[c].x > blowup) flags |= LD_STATUS_BLOWUP;
    }
  }
  if (flags) atomicOr(status, flags);
}

template <typename T>
__global__ void k_ifac(T* __restrict__ tab, int n, double nuh) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    tab[i] = T(exp(-nuh * double(i)));
}

// ------------------------------------------------------------------------------------------
// droplets
// ------------------------------------------------------------------------------------------
// Stencil along one axis: base index (periodic) and weights for offsets (lo .. lo+W-1).
template <typename T, int METHOD> struct AxisW;

template <typename T> struct AxisW<T, LD_INTERP_TRILINEAR> {
  static constexpr int W = 2, LO = 0;
  __device__ __forceinline__ static void get(double p, int N, double L, int& i0, T* w) {
    const double s = p * (double(N) / L);
    double fl = floor(s);
    const double t = s - fl;
    long long ii = (long long)fl % N;
    if (ii < 0) ii += N;
    i0 = int(ii);
    w[0] = T(1.0 - t);
    w[1] = T(t);
  }
};

template <typename T> struct AxisW<T, LD_INTERP_TRICUBIC> {
  static constexpr int W = 4, LO = -1;
  __device__ __forceinline__ static void get(double p, int N, double L, int& i0, T* w) {
    const double s = p * (double(N) / L);
    double fl = floor(s);
    const double t = s - fl;
    long long ii = (long long)fl % N;
    if (ii < 0) ii += N;
    i0 = int(ii);
    w[0] = T(-t * (t - 1.0) * (t - 2.0) / 6.0);
    w[1] = T((t + 1.0) * (t - 1.0) * (t - 2.0) / 2.0);
    w[2] = T(-(t + 1.0) * t * (t - 2.0) / 2.0);
    w[3] = T((t + 1.0) * t * (t - 1.0) / 6.0);
  }
};

// The reference's cosine kernel (P:9-16, P:441, P:456): offsets -1..2 around floor(pos/dx),
// weight (1 + cos((pos - X_j) pi / (2 dx))) / 4 with X_j on the periodic index.
template <typename T> struct AxisW<T, LD_INTERP_COSINE> {
  static constexpr int W = 4, LO = -1;
  __device__ __forceinline__ static void get(double p, int N, double L, int& i0, T* w) {
    const double dx = L / double(N);
    const double pm = p - L * floor(p / L);
    long long ii = (long long)floor(pm / dx);
    ii %= N;
    if (ii < 0) ii += N;
    i0 = int(ii);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      int jx = (i0 - 1 + a) % N;
      if (jx < 0) jx += N;
      const double Xj = double(jx) * dx;
      w[a] = T((1.0 + cos((pm - Xj) * (3.14159265358979323846 / (2.0 * dx)))) / 4.0);
    }
  }
};

// i in [-N, 2N) -> i mod N (stencil offsets around a cell index in [0, N); any N)
__device__ __forceinline__ int wrap_index(int i, int N) {
  i = i < 0 ? i + N : i;
  return i >= N ? i - N : i;
}

template <typename T, int METHOD>
__device__ __forceinline__ void gather_point(const T* __restrict__ f, int ncomp, long long fstride, int N,
                                             double L, double px, double py, double pz, T* out) {
  using A = AxisW<T, METHOD>;
  constexpr int W = A::W, LO = A::LO;
  int ix, iy, iz;
  T wx[W], wy[W], wz[W];
  A::get(px, N, L, ix, wx);
  A::get(py, N, L, iy, wy);
  A::get(pz, N, L, iz, wz);
  int jz[W];
#pragma unroll
  for (int c = 0; c < W; ++c) jz[c] = wrap_index(iz + LO + c, N);
  for (int c = 0; c < ncomp; ++c) out[c] = T(0);
#pragma unroll
  for (int a = 0; a < W; ++a) {
    const int jx = wrap_index(ix + LO + a, N);
#pragma unroll
    for (int b = 0; b < W; ++b) {
      const int jy = wrap_index(iy + LO + b, N);
      const long long base = ((long long)jx * N + jy) * N;
      const T wab = wx[a] * wy[b];
      for (int c = 0; c < ncomp; ++c) {
        const T* fc = f + c * fstride + base;
        T acc = T(0);
#pragma unroll
        for (int q = 0; q < W; ++q) acc += wz[q] * __ldg(fc + jz[q]);
        out[c] += wab * acc;
      }
    }
  }
}

template <typename T, int METHOD>
__global__ void k_gather(const T* __restrict__ f, int ncomp, int N, double L, const double* __restrict__ pos,
                         long long n, T* __restrict__ out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    T v[8];
    gather_point<T, METHOD>(f, ncomp, (long long)N * N * N, N, L, pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], v);
    for (int c = 0; c < ncomp; ++c) out[i * ncomp + c] = v[c];
  }
}

// Interpolation of an interleaved (N, N, N, 4) velocity: one 16/32-byte load per stencil point.
template <typename T, int METHOD>
__device__ __forceinline__ void gather_point4(const vec4<T>* __restrict__ f, int N, double L, double px, double py,
                                              double pz, T* out) {
  using A = AxisW<T, METHOD>;
  constexpr int W = A::W, LO = A::LO;
  int ix, iy, iz;
  T wx[W], wy[W], wz[W];
  A::get(px, N, L, ix, wx);
  A::get(py, N, L, iy, wy);
  A::get(pz, N, L, iz, wz);
  int jz[W];
#pragma unroll
  for (int c = 0; c < W; ++c) jz[c] = wrap_index(iz + LO + c, N);
  T o0 = 0, o1 = 0, o2 = 0;
#pragma unroll
  for (int a = 0; a < W; ++a) {
    const int jx = wrap_index(ix + LO + a, N);
#pragma unroll
    for (int b = 0; b < W; ++b) {
      const int jy = wrap_index(iy + LO + b, N);
      const vec4<T>* row = f + ((long long)jx * N + jy) * N;
      T s0 = 0, s1 = 0, s2 = 0;
#pragma unroll
      for (int q = 0; q < W; ++q) {
        const vec4<T> v = row[jz[q]];
        s0 += wz[q] * v.x;
        s1 += wz[q] * v.y;
        s2 += wz[q] * v.z;
      }
      const T wab = wx[a] * wy[b];
      o0 += wab * s0;
      o1 += wab * s1;
      o2 += wab * s2;
    }
  }
  out[0] = o0;
  out[1] = o1;
  out[2] = o2;
}

template <typename T, int METHOD>
__global__ void k_gather4(const vec4<T>* __restrict__ f, int N, double L, const double* __restrict__ pos, long long n,
                          T* __restrict__ out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    T v[3];
    gather_point4<T, METHOD>(f, N, L, pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], v);
    out[3 * i] = v[0];
    out[3 * i + 1] = v[1];
    out[3 * i + 2] = v[2];
  }
}

template <typename T, int METHOD, int STAGE>
__global__ void k_droplet_stage(const vec4<T>* __restrict__ u0, int N, double L, double* __restrict__ pos,
                                T* __restrict__ vel, const T* __restrict__ tau, T* __restrict__ a1,
                                long long n, double h, T g, const int* __restrict__ box = nullptr) {
  grid_dep();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    // the droplet's box of a multi-box plan: its field is box (N, N, N, 4) further on
    const vec4<T>* u = box ? u0 + (long long)box[i] * N * N * N : u0;
    const double px = pos[3 * i], py = pos[3 * i + 1], pz = pos[3 * i + 2];
    const T vx = vel[3 * i], vy = vel[3 * i + 1], vz = vel[3 * i + 2];
    const T it = T(1) / tau[i];
    T up[3];
    if (STAGE == 1) {
      gather_point4<T, METHOD>(u, N, L, px, py, pz, up);
      a1[3 * i] = (up[0] - vx) * it;
      a1[3 * i + 1] = (up[1] - vy) * it;
      a1[3 * i + 2] = (up[2] - vz) * it - g;
    } else {
      const T ax = a1[3 * i], ay = a1[3 * i + 1], az = a1[3 * i + 2];
      const T hh = T(h);
      const T sx = vx + hh * ax, sy = vy + hh * ay, sz = vz + hh * az;  // vs = v + h a1
      const double qx = px + h * double(vx), qy = py + h * double(vy), qz = pz + h * double(vz);
      gather_point4<T, METHOD>(u, N, L, qx, qy, qz, up);
      const T bx = (up[0] - sx) * it, by = (up[1] - sy) * it, bz = (up[2] - sz) * it - g;
      pos[3 * i] = px + 0.5 * h * (double(vx) + double(sx));
      pos[3 * i + 1] = py + 0.5 * h * (double(vy) + double(sy));
      pos[3 * i + 2] = pz + 0.5 * h * (double(vz) + double(sz));
      vel[3 * i] = vx + T(0.5) * hh * (ax + bx);
      vel[3 * i + 1] = vy + T(0.5) * hh * (ay + by);
      vel[3 * i + 2] = vz + T(0.5) * hh * (az + bz);
    }
  }
}

}  // namespace ld
