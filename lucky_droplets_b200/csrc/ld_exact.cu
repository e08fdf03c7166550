// Exact spectral (direct Fourier sum) velocity at arbitrary points, FP64.
//
//   u_c(x) = (1/N^3) sum_{kx,ky} sum_{kz=0}^{kc} w_kz Re( uk_c(kx,ky,kz) exp(i k.x) ),
//   w_0 = 1, w_kz = 2 (kz > 0),
// the continuous extension of the inverse real transform (at grid points it equals irfft, which
// also drops the imaginary part of the kz = 0 coefficients).  Only the modes of the spherical
// mask round(|k|) <= kc are summed: they are the only non-zero modes of a dealiased field.
//
// The sum over ky is a real matrix product on the FP64 tensor pipe.  With A = u(+ky) + u(-ky) and
// B = u(+ky) - u(-ky),
//   S(kx, kz; p) = sum_ky u exp(i ky y_p) = u(0) + sum_{ky > 0} A cos(ky y_p) + i B sin(ky y_p),
// so for every (c, kx, kz) the two rows (Re u0, Re A1, -Im B1, Re A2, ...) and (Im u0, Im A1,
// Re B1, ...) times the column (1, cos y, sin y, cos 2y, ...) of a point give Re S and Im S: two
// real multiply-adds per mode and component, half of a complex product and without a phase
// recurrence per mode.  k_exact_pack writes the rows once per call, in the order of the matrix
// fragments; k_exact_mma multiplies them with the columns of 16 points per warp and contracts
// S with exp(i kz z) and exp(i kx x) in the epilogues (a few multiply-adds per row and point).
#include "ld_internal.cuh"

namespace {

// Steps of four columns (ky terms) per staged chunk, 512 bytes each, and chunks in flight.  A chunk
// holds a whole item up to kc = 87, so that the block synchronises once per item: 6.25 ms for 1e4
// points at 256^3, against 6.48 with chunks of 32 and 6.89 with chunks of 16 steps.
constexpr int EX_CH = 44;
constexpr int EX_STAGES = 2;
constexpr size_t EX_RING = (size_t)EX_STAGES * EX_CH * 64 * sizeof(double);

// Steps of four columns that the rows (kx, kz = 8 t .. 8 t + 7) need: ky terms up to the edge of
// the sphere at kz = 8 t; 0 when the tile lies outside it.  (Integers below 2^24: sqrtf is exact
// enough for the floor.)
__device__ __forceinline__ int exact_steps(int ix, int t, int kc, int My) {
  const int kx = ix <= kc ? ix : ix - My;
  const int rem = kc * kc + kc - kx * kx - 64 * t * t;  // round(|k|) <= kc  <=>  k^2 <= kc^2 + kc
  if (rem < 0) return 0;
  return (2 * (int)sqrtf((float)rem) + 4) / 4;  // columns 1 + 2 ky_max, rounded up
}

// Rows in fragment order: item ((ix T + t) 3 + c), then step s of four columns, lane, (Re, Im):
// lane l holds kz = 8 t + l / 4 and column kappa = 4 s + l % 4 (0: 1, 2 j - 1: cos(j y), 2 j:
// sin(j y)).  The weight of kz > 0 is folded in (exact); modes outside the mask are zero.
template <typename T>
__global__ void k_exact_pack(const ld::cplx<T>* __restrict__ uk, long long cs, int kc, int My, int Mzp, int steps,
                             double2* __restrict__ rows) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const int s = e >> 5, l = e & 31;
  const int tc = blockIdx.y, t = tc / 3, c = tc - 3 * t, ix = blockIdx.z;
  if (s >= exact_steps(ix, t, kc, My)) return;
  const int kx = ix <= kc ? ix : ix - My;
  const int kz = 8 * t + (l >> 2), kap = 4 * s + (l & 3), j = (kap + 1) / 2;
  double2 v = make_double2(0.0, 0.0);
  if (kz <= kc && j <= kc && kx * kx + j * j + kz * kz <= kc * kc + kc) {
    const double w = kz ? 2.0 : 1.0;
    const ld::cplx<T>* u = uk + c * cs + (long long)ix * My * Mzp + kz;
    const ld::cplx<T> p = u[(long long)j * Mzp];
    if (j == 0) {
      v = make_double2(w * (double)p.x, w * (double)p.y);
    } else {
      const ld::cplx<T> m = u[(long long)(My - j) * Mzp];
      if (kap & 1) v = make_double2(w * ((double)p.x + (double)m.x), w * ((double)p.y + (double)m.y));
      else v = make_double2(-w * ((double)p.y - (double)m.y), w * ((double)p.x - (double)m.x));
    }
  }
  rows[((long long)(ix * gridDim.y + tc) * steps + s) * 32 + l] = v;
}

// c (16 x 8: eight Re rows, eight Im rows) += a (16 x 4) b (4 x 8)
__device__ __forceinline__ void mma_f64(double (&c)[4], double2 a, double b) {
  asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
               : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
               : "d"(a.x), "d"(a.y), "d"(b));
}

// Block = P points (16 per warp) x the kx planes ix = blockIdx.y, + gridDim.y, ...  The points'
// columns (cos, sin of every ky) stay in shared memory for the whole block; the rows stream
// through a ring of EX_STAGES chunks by 16-byte asynchronous copies, every warp using each chunk.
// Bound by the FP64 pipe: a warp's step is two 16 x 8 x 4 products (64 cycles of its share of the
// pipe) for eight shared-memory wavefronts.  1e4 points at 256^3, FP32 spectrum: 30.4 ms with a
// thread per point and a phase recurrence per mode (16 FP64 operations a mode), 6.25 ms here, 25 of
// the 36.7 TFLOP/s that the pipe gives these products, tiles' padding not counted.  P = 128 reuses each staged row for 128 points and
// still leaves room for the ring up to kc = 89; larger grids have columns of 64 points.
// Partial sums of the kx planes are added in block order afterwards (deterministic).
template <int P>
__global__ void __launch_bounds__(2 * P, 1)
k_exact_mma(const double2* __restrict__ rows, int kc, int My, int T, int steps, const double* __restrict__ pos,
            long long n, double* __restrict__ part) {
  constexpr int THREADS = 2 * P, NW = P / 16;
  extern __shared__ __align__(16) unsigned char ex_smem[];
  double2* ring = reinterpret_cast<double2*>(ex_smem);                 // [stage][step][lane] (Re, Im)
  double* cols = reinterpret_cast<double*>(ex_smem + EX_RING);         // [step][warp][lane][2 point octets]
  double* xs = cols + (size_t)steps * 4 * P;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long p0 = (long long)blockIdx.x * P;

  // the stream of chunks this block works through: (ix, t, c, step q)
  struct Walk {
    int ix, t, c, q, n4;
  };
  auto advance = [&](Walk& w) {
    w.q += EX_CH;
    if (w.q < w.n4) return;
    w.q = 0;
    if (++w.c < 3) return;
    w.c = 0;
    ++w.t;
    w.n4 = w.t < T ? exact_steps(w.ix, w.t, kc, My) : 0;
    if (w.n4 > 0) return;
    w.t = 0;
    w.ix += gridDim.y;
    w.n4 = w.ix < My ? exact_steps(w.ix, 0, kc, My) : 0;
  };
  auto fetch = [&](Walk& w, int stage) {
    if (w.ix < My) {
      const int m = (w.n4 - w.q < EX_CH ? w.n4 - w.q : EX_CH) * 32;
      const double2* src = rows + ((long long)((w.ix * T + w.t) * 3 + w.c) * steps + w.q) * 32;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(ring + stage * EX_CH * 32);
      for (int e = tid; e < m; e += THREADS)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * e), "l"(src + e) : "memory");
      advance(w);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  Walk ahead{(int)blockIdx.y, 0, 0, 0, exact_steps(blockIdx.y, 0, kc, My)};
#pragma unroll
  for (int s = 0; s < EX_STAGES - 1; ++s) fetch(ahead, s);

  // the block's columns
  for (int e = tid; e < P; e += THREADS) xs[e] = p0 + e < n ? pos[3 * (p0 + e)] : 0.0;
  for (int e = tid; e < 2 * steps * P; e += THREADS) {
    const int p = e % P, j = e / P;
    const double y = p0 + p < n ? pos[3 * (p0 + p) + 1] : 0.0;
    double sn = 0.0, cn = 0.0;
    if (j <= kc) sincos((double)j * y, &sn, &cn);
    auto slot = [&](int kap) -> double& {
      return cols[(((size_t)(kap >> 2) * NW + (p >> 4)) * 32 + ((p & 7) << 2) + (kap & 3)) * 2 + ((p >> 3) & 1)];
    };
    if (j > 0) slot(2 * j - 1) = cn;
    else slot(0) = 1.0;
    if (j > 0) slot(2 * j) = sn;
    if (j == 2 * steps - 1) slot(4 * steps - 1) = 0.0;
  }

  // this thread's accumulator columns: points 16 warp + 8 f + 2 (lane % 4) + e
  const int pl = 16 * warp + 2 * (lane & 3);
  double2 g0[4], gs[4], g[4], S[3][4];
  double u[3][4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const long long p = p0 + pl + 8 * (k >> 1) + (k & 1);
    const double z = p < n ? pos[3 * p + 2] : 0.0;
    sincos((double)(lane >> 2) * z, &g0[k].y, &g0[k].x);  // exp(i kz z) of the row's kz in tile 0
    sincos(8.0 * z, &gs[k].y, &gs[k].x);                  // from one tile to the next
#pragma unroll
    for (int c = 0; c < 3; ++c) u[c][k] = 0.0;
  }

  int it = 0;  // chunks done
  for (int ix = blockIdx.y; ix < My; ix += gridDim.y) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      g[k] = g0[k];
#pragma unroll
      for (int c = 0; c < 3; ++c) S[c][k] = make_double2(0.0, 0.0);
    }
    for (int t = 0; t < T; ++t) {
      const int n4 = exact_steps(ix, t, kc, My);
      if (n4 == 0) break;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        double acc[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};
        for (int q = 0; q < n4; q += EX_CH, ++it) {
          asm volatile("cp.async.wait_group %0;" ::"n"(EX_STAGES - 2) : "memory");
          __syncthreads();  // this chunk is in shared memory; the previous one has been used
          fetch(ahead, (it + EX_STAGES - 1) % EX_STAGES);
          const double2* a = ring + (it % EX_STAGES) * EX_CH * 32 + lane;
          const double2* b = reinterpret_cast<const double2*>(cols) + ((size_t)q * NW + warp) * 32 + lane;
          const int m = n4 - q < EX_CH ? n4 - q : EX_CH;
#pragma unroll 4
          for (int s = 0; s < m; ++s) {
            const double2 av = a[s * 32], bv = b[(size_t)s * NW * 32];
            mma_f64(acc[0], av, bv.x);
            mma_f64(acc[1], av, bv.y);
          }
        }
        // S(kx, kz; p) exp(i kz z): acc[f][e] = Re S, acc[f][2 + e] = Im S of point 2 f + e
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const double re = acc[k >> 1][k & 1], im = acc[k >> 1][2 + (k & 1)];
          S[c][k].x += re * g[k].x - im * g[k].y;
          S[c][k].y += re * g[k].y + im * g[k].x;
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const double gx = g[k].x * gs[k].x - g[k].y * gs[k].y;
        g[k].y = g[k].x * gs[k].y + g[k].y * gs[k].x;
        g[k].x = gx;
      }
    }
    const double kx = ix <= kc ? ix : ix - My;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      double sn, cn;
      sincos(kx * xs[pl + 8 * (k >> 1) + (k & 1)], &sn, &cn);
#pragma unroll
      for (int c = 0; c < 3; ++c) u[c][k] += S[c][k].x * cn - S[c][k].y * sn;  // Re(exp(i kx x) S)
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // the eight rows of a tile are spread over lane / 4
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
#pragma unroll
      for (int d = 4; d < 32; d <<= 1) u[c][k] += __shfl_xor_sync(0xffffffffu, u[c][k], d);
    }
  if (lane < 4) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const long long p = p0 + pl + 8 * (k >> 1) + (k & 1);
      if (p < n) {
#pragma unroll
        for (int c = 0; c < 3; ++c) part[((long long)blockIdx.y * n + p) * 3 + c] = u[c][k];
      }
    }
  }
}

// out = (1/N^3) sum over chunks, in chunk order
__global__ void k_exact_reduce(const double* __restrict__ part, int chunks, long long n, double scale,
                               double* __restrict__ out) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < 3 * n; e += (long long)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int c = 0; c < chunks; ++c) s += part[(long long)c * 3 * n + e];
    out[e] = s * scale;
  }
}

template <int P>
int launch_mma(const double2* rows, int kc, int My, int T, int steps, const double* pos, long long n, int chunks,
               double* part, cudaStream_t s) {
  const size_t smem = EX_RING + sizeof(double) * ((size_t)steps * 4 * P + P);
  auto k = k_exact_mma<P>;
  LD_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const dim3 grid((unsigned)((n + P - 1) / P), (unsigned)chunks);
  k<<<grid, 2 * P, smem, s>>>(rows, kc, My, T, steps, pos, n, part);
  LD_LAUNCH_CHECK();
  return LD_OK;
}

}  // namespace

extern "C" int ld_exact_sum(ld_plan* p, const void* uk, const double* pos, int64_t n, double* out, void* stream) {
  if (!p || !uk || !pos || !out || n < 0) return ld_fail(LD_ERR_ARG, "ld_exact_sum: bad arguments");
  if (n == 0) return LD_OK;
  cudaStream_t s = (cudaStream_t)stream;
  ProfScope ps(p, KID_EXACT, s);
  const int kc = p->kc, My = p->My, T = kc / 8 + 1, steps = (2 * kc + 4) / 4;
  // the rows and the partial sums live in the plan's transform workspace (free between steps): the
  // rows take 48 My T 8 * 4 steps bytes, less than the workspace's second half (48 N^2 Mzp and
  // more, with My and 4 steps below N); the partial sums get the rest, points in batches that fit
  const size_t row_bytes = sizeof(double2) * 32 * (size_t)My * T * 3 * steps;
  if (row_bytes >= p->work_bytes) return ld_fail(LD_ERR_CAPACITY, "ld_exact_sum: no workspace");
  double2* rows = (double2*)p->work;
  double* part = (double*)((char*)p->work + row_bytes);
  const long long cap = (long long)((p->work_bytes - row_bytes) / sizeof(double));
  const dim3 pg((unsigned)((steps * 32 + 127) / 128), (unsigned)(3 * T), (unsigned)My);
  if (p->prec == LD_F32) k_exact_pack<float><<<pg, 128, 0, s>>>((const float2*)uk, p->cube_elems(), kc, My, p->Mzp, steps, rows);
  else k_exact_pack<double><<<pg, 128, 0, s>>>((const double2*)uk, p->cube_elems(), kc, My, p->Mzp, steps, rows);
  LD_LAUNCH_CHECK();
  const double scale = 1.0 / ((double)p->N * p->N * p->N);
  const bool wide = EX_RING + sizeof(double) * ((size_t)steps * 4 * 128 + 128) <= 227 * 1024;
  const int P = wide ? 128 : 64;
  for (long long b0 = 0; b0 < n;) {
    long long nb = n - b0;
    if (3 * nb > cap) nb = cap / 3;
    if (nb > 65535LL * P) nb = 65535LL * P;
    if (nb < 1) return ld_fail(LD_ERR_CAPACITY, "ld_exact_sum: no workspace");
    // kx planes split over at least eight rounds of blocks (one block per SM), with the last
    // round as full as a few more blocks make it
    const long long tiles = (nb + P - 1) / P;
    const long long most = cap / (3 * nb) < My ? cap / (3 * nb) : My;
    long long lo = (148LL * 8 + tiles - 1) / tiles, chunks = 0;
    if (lo > most) lo = most;
    double best = 0.0;
    for (long long c = lo; c <= most && c < 2 * lo + 8; ++c) {
      const long long rounds = (tiles * c + 147) / 148;
      const double full = (double)(tiles * c) / (double)(148 * rounds);
      if (full > best + 0.005) { best = full; chunks = c; }
    }
    int rc = wide ? launch_mma<128>(rows, kc, My, T, steps, pos + 3 * b0, nb, (int)chunks, part, s)
                  : launch_mma<64>(rows, kc, My, T, steps, pos + 3 * b0, nb, (int)chunks, part, s);
    if (rc) return rc;
    long long rb = (3 * nb + 255) / 256;
    if (rb > 148LL * 16) rb = 148LL * 16;
    k_exact_reduce<<<(unsigned)rb, 256, 0, s>>>(part, (int)chunks, nb, scale, out + 3 * b0);
    LD_LAUNCH_CHECK();
    b0 += nb;
  }
  return LD_OK;
}
