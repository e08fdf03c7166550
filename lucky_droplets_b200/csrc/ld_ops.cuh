// Launch sequences for one (precision, N) instance.  Included by the ld_inst_*.cu units, each
// of which instantiates one OpsTable; compiling the twenty instances separately keeps the build
// parallel.
#pragma once
#include <cmath>
#include <type_traits>

#include "ld_internal.cuh"
#include "ld_kernels.cuh"

namespace ld_impl {

using namespace ld;

inline cudaStream_t S(void* s) { return reinterpret_cast<cudaStream_t>(s); }

template <class K> int set_smem(K kernel, size_t bytes) {
  if (bytes > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) { ld_set_last_error(e); return LD_ERR_CUDA; }
  }
  return LD_OK;
}

inline long long cdiv(long long a, long long b) { return (a + b - 1) / b; }

inline int grid1d(long long n, int threads) {
  long long b = cdiv(n, threads);
  if (b > 148LL * 32) b = 148LL * 32;
  if (b < 1) b = 1;
  return (int)b;
}

inline bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

template <typename T, int N> struct Ops {
  using C = cplx<T>;
  static constexpr int TB = Cfg<N>::TB;
  static constexpr size_t COL_SMEM = sizeof(C) * N * TB;
  using Z = ZCfg<T, N>;
  static constexpr size_t Z_SMEM = sizeof(C) * Z::UNITS1 * Z::ZBUF1;

  // whether the flow's passes may begin early: at most one x plane per SM (launch_dep)
  static bool early(const ld_plan* p) { return (long long)N * p->nbox <= kSMs; }
  // and those of a reference-layout transform of so many spectral elements
  static bool early_transform(long long elems) { return elems * (long long)sizeof(C) <= 300LL << 20; }

  template <bool INV, class Ld, class St>
  static int colpass(ld_plan* p, int kid, Ld ld, St st, int ncols, int nf, int nouter, const C* tw, cudaStream_t s,
                     bool dep) {
    ProfScope ps(p, kid, s);
    auto k = colfft_kernel<T, N, INV, Ld, St>();
    if (int rc = set_smem(k, COL_SMEM)) return rc;
    dim3 grid((unsigned)(cdiv(ncols, TB) * nf), (unsigned)nouter);
    LD_CUDA_CHECK(launch_dep(dep, k, grid, Cfg<N>::COL_THREADS, COL_SMEM, s, ld, st, ncols, nf, tw));
    return LD_OK;
  }

  // The same with two columns per thread (FP32, even row strides and columns, 16-byte aligned rows)
  static constexpr bool PAIRS = sizeof(T) == 4 && Col2<N>::OK;
  template <bool INV, class Ld, class St>
  static int colpass2(ld_plan* p, int kid, Ld ld, St st, int ncols, int nf, int nouter, const C* tw, cudaStream_t s) {
    ProfScope ps(p, kid, s);
    auto k = k_colfft2<N, INV, Ld, St>;
    if (int rc = set_smem(k, Col2<N>::SMEM)) return rc;
    dim3 grid((unsigned)(cdiv(ncols, TB) * nf), (unsigned)nouter);
    LD_CUDA_CHECK(launch_dep(early(p), k, grid, Col2<N>::THREADS, Col2<N>::SMEM, s, ld, st, ncols, nf, tw));
    return LD_OK;
  }
  template <bool INV, class St, bool IN_MAP, int RSC> static constexpr auto pipe_kernel() {
    if constexpr (PAIRS) return k_colfft_pipe2<N, INV, St, IN_MAP, RSC>;
    else return k_colfft_pipe<T, N, INV, St, IN_MAP, RSC>;
  }

  // Column pass over plain strided rows: the pipelined kernel where two staging buffers fit.
  static constexpr bool PIPE = 2 * COL_SMEM <= 72 * 1024;
  // IN_MAP: the input rows are compact cube rows; RS: their stride
  template <bool INV, bool IN_MAP, int RS, class St>
  static int colpass_rows(ld_plan* p, int kid, RowsIO<T> in, St st, int ncols, int nf, int nouter, const C* tw,
                          cudaStream_t s, int variant = -2) {
    const int choice = variant != -2 ? variant : p->tune_y[INV ? 0 : 1];
    if constexpr (!PIPE) {
      if constexpr (PAIRS) return colpass2<INV>(p, kid, LdRowsC<T, N, IN_MAP, RS>{in}, st, ncols, nf, nouter, tw, s);
      else return colpass<INV>(p, kid, LdRowsC<T, N, IN_MAP, RS>{in}, st, ncols, nf, nouter, tw, s, N <= 384);
    } else {
      // untuned plans: one-shot tiles for short columns (right-hand side at 128^3 FP64 96 us, 104 with the
      // pipelined pass; 16 boxes of it 1430 and 1480 us, 16 boxes of 96^3 758 and 830 us), except with two
      // columns per thread (FP32 58 -> 61 us).  Their grid has the outer index as its second dimension,
      // 65535 at most (682 boxes of 96^3); beyond it the pipelined pass, whose grid is linear, takes over.
      const bool one_shot = choice == 0 || (choice < 0 && N <= 128 && !PAIRS);
      if ((one_shot && nouter <= 65535) || cdiv(ncols, TB) * (long long)nf * nouter >= (1LL << 31)) {
        if constexpr (PAIRS) return colpass2<INV>(p, kid, LdRowsC<T, N, IN_MAP, RS>{in}, st, ncols, nf, nouter, tw, s);
        else return colpass<INV>(p, kid, LdRowsC<T, N, IN_MAP, RS>{in}, st, ncols, nf, nouter, tw, s, N <= 384);
      }
      ProfScope ps(p, kid, s);
      constexpr int threads = PAIRS ? Col2<N>::THREADS : Cfg<N>::COL_THREADS;
      constexpr size_t smem = 2 * COL_SMEM + (PAIRS ? sizeof(float4) * Col2<N>::Tw::ELEMS : 0);
      auto k = pipe_kernel<INV, St, IN_MAP, RS>();
      if (int rc = set_smem(k, smem)) return rc;
      static int occ = 0;
      if (occ == 0) {
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, threads, smem);
        if (e != cudaSuccess || occ < 1) occ = 1;
      }
      int dev = 0, sms = 148;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      const long long items = cdiv(ncols, TB) * (long long)nf * nouter;
      const int per_sm = choice > 0 && choice < occ ? choice : occ;
      const long long grid = items < (long long)sms * per_sm ? items : (long long)sms * per_sm;
      LD_CUDA_CHECK(launch_dep(early(p), k, dim3((unsigned)grid), threads, smem, s, in, st, ncols, nf, nouter, tw));
      return LD_OK;
    }
  }

  static RowsIO<T> io(const void* p, long long fs, long long os) { return RowsIO<T>{(C*)p, fs, os}; }
  using RS = RowStride<N>;

  static int z_c2r(ld_plan* p, const C* X, T* x, long long nrows, int ss, int Kin, T sc, long long xfs, long long Xfs,
                   int nf, const C* tw, cudaStream_t s, bool dep) {
    ProfScope ps(p, KID_ZC2R, s);
    auto k = k_z_c2r<T, N>;
    if (int rc = set_smem(k, Z_SMEM)) return rc;
    dim3 grid((unsigned)cdiv(nrows / 2, Z::UNITS1), (unsigned)nf);
    LD_CUDA_CHECK(launch_dep(dep, k, grid, Z::THREADS1, Z_SMEM, s, X, x, nrows, ss, Kin, sc, xfs, Xfs, tw));
    return LD_OK;
  }

  static int z_r2c(ld_plan* p, const T* x, C* X, long long nrows, int ss, int Kout, int Kval, long long xfs, long long Xfs,
                   int nf, const C* tw, cudaStream_t s, bool dep) {
    ProfScope ps(p, KID_ZR2C, s);
    auto k = k_z_r2c<T, N>;
    if (int rc = set_smem(k, Z_SMEM)) return rc;
    dim3 grid((unsigned)cdiv(nrows / 2, Z::UNITS1), (unsigned)nf);
    LD_CUDA_CHECK(launch_dep(dep, k, grid, Z::THREADS1, Z_SMEM, s, x, X, nrows, ss, Kout, Kval, xfs, Xfs, tw));
    return LD_OK;
  }

  // ---- reference-layout transforms --------------------------------------------------------
  static int rfft_full(ld_plan* p, const T* u, C* fu, int ncomp, cudaStream_t s) {
    const int Nf = p->Nf;
    const C* tw = (const C*)p->tw;
    const long long NN = (long long)N * N;
    const bool dep = early_transform(ncomp * NN * Nf);
    if (int rc = z_r2c(p, u, fu, NN, Nf, Nf, Nf, NN * N, NN * Nf, ncomp, tw, s, dep)) return rc;
    // y pass in place: columns kz (Nf), rows y, outer x
    auto yio = io(fu, NN * Nf, (long long)N * Nf);
    if (int rc = colpass<false>(p, KID_YFWD, LdRowsC<T, N, false, RS::YF>{yio}, StRowsC<T, N, false, RS::YF>{yio}, Nf, ncomp, N, tw, s, dep)) return rc;
    // x pass in place: columns (ky, kz) flat, rows x
    auto xio = io(fu, NN * Nf, 0);
    return colpass<false>(p, KID_XPASS, LdRowsC<T, N, false, RS::XF>{xio}, StRowsC<T, N, false, RS::XF>{xio}, N * Nf, ncomp, 1, tw, s, dep);
  }

  static int irfft_full(ld_plan* p, const C* fu, T* u, int ncomp, cudaStream_t s) {
    const int Nf = p->Nf;
    const C* tw = (const C*)p->tw;
    const long long NN = (long long)N * N;
    const long long per = NN * Nf;
    const int chunk = (int)(((long long)6 * NN * p->Mzp) / per);  // fields that fit in W2
    C* W = (C*)p->W2;
    for (int c0 = 0; c0 < ncomp; c0 += chunk) {
      const int nc = ncomp - c0 < chunk ? ncomp - c0 : chunk;
      const bool dep = early_transform(nc * per);
      auto xin = io(fu + c0 * per, per, 0);
      auto xout = io(W, per, 0);
      if (int rc = colpass<true>(p, KID_XPASS, LdRowsC<T, N, false, RS::XF>{xin}, StRowsC<T, N, false, RS::XF>{xout}, N * Nf, nc, 1, tw, s, dep)) return rc;
      auto yio = io(W, per, (long long)N * Nf);
      if (int rc = colpass<true>(p, KID_YINV, LdRowsC<T, N, false, RS::YF>{yio}, StRowsC<T, N, false, RS::YF>{yio}, Nf, nc, N, tw, s, dep)) return rc;
      const T sc = T(1.0 / (double(N) * N * N));
      if (int rc = z_c2r(p, W, u + (long long)c0 * NN * N, NN, Nf, Nf, sc, NN * N, per, nc, tw, s, dep)) return rc;
    }
    return LD_OK;
  }

  // ---- cube-layout (dealiased) transforms -----------------------------------------------------
  static int irfft_cube(ld_plan* p, const C* uk, T* u, int ncomp, cudaStream_t s) {
    const int kc = p->kc, My = p->My, Mzp = p->Mzp;
    const C* tw = (const C*)p->tw;
    const long long NN = (long long)N * N;
    const long long cs = p->cube_elems();
    C* W1 = (C*)p->W1;
    C* W2 = (C*)p->W2;
    const long long w1s = (long long)N * My * Mzp, w2s = NN * Mzp;
    for (int c0 = 0; c0 < ncomp; c0 += 6) {
      const int nc = ncomp - c0 < 6 ? ncomp - c0 : 6;
      auto xin = io(uk + c0 * cs, cs, 0);
      auto xout = io(W1, w1s, 0);
      if (int rc = colpass<true>(p, KID_XPASS, LdRowsC<T, N, true, RS::XC>{xin}, StRowsC<T, N, false, RS::XC>{xout}, My * Mzp, nc, 1, tw, s, true)) return rc;
      auto yin = io(W1, w1s, (long long)My * Mzp);
      auto yout = io(W2, w2s, (long long)N * Mzp);
      if (int rc = colpass<true>(p, KID_YINV, LdRowsC<T, N, true, RS::YC>{yin}, StRowsC<T, N, false, RS::YC>{yout}, Mzp, nc, N, tw, s, true)) return rc;
      const T sc = T(1.0 / (double(N) * N * N));
      if (int rc = z_c2r(p, W2, u + (long long)c0 * NN * N, NN, Mzp, kc + 1, sc, NN * N, w2s, nc, tw, s, true)) return rc;
    }
    return LD_OK;
  }

  static int rfft_cube(ld_plan* p, const T* u, C* uk, int ncomp, cudaStream_t s) {
    const int kc = p->kc, My = p->My, Mzp = p->Mzp;
    const C* tw = (const C*)p->tw;
    const long long NN = (long long)N * N;
    const long long cs = p->cube_elems();
    C* W1 = (C*)p->W1;
    C* W2 = (C*)p->W2;
    const long long w1s = (long long)N * My * Mzp, w2s = NN * Mzp;
    for (int c0 = 0; c0 < ncomp; c0 += 6) {
      const int nc = ncomp - c0 < 6 ? ncomp - c0 : 6;
      if (int rc = z_r2c(p, u + (long long)c0 * NN * N, W2, NN, Mzp, Mzp, kc + 1, NN * N, w2s, nc, tw, s, true)) return rc;
      auto yin = io(W2, w2s, (long long)N * Mzp);
      auto yout = io(W1, w1s, (long long)My * Mzp);
      if (int rc = colpass<false>(p, KID_YFWD, LdRowsC<T, N, false, RS::YC>{yin}, StRowsC<T, N, true, RS::YC>{yout}, Mzp, nc, N, tw, s, true)) return rc;
      auto xin = io(W1, w1s, 0);
      auto xout = io(uk + c0 * cs, cs, 0);
      if (int rc = colpass<false>(p, KID_XPASS, LdRowsC<T, N, false, RS::XC>{xin}, StCube<T, N>{xout}, My * Mzp, nc, 1, tw, s, true)) return rc;
    }
    return LD_OK;
  }

  // ---- forcing factors of the stage input y: shells kf_lo..kf_hi (none when nshell = 0) ------------
  static ShellArgs<T> forcing(ld_plan* p, const C* y, const ld_flow_params* prm) {
    ShellArgs<T> F;
    F.u = y; F.cs = p->cube_elems(); F.ubs = 3 * p->cube_elems();
    F.off = p->shell_off; F.idx = p->shell_idx; F.Mzp = p->Mzp;
    F.shell0 = prm->kf_lo;
    F.nshell = prm->kf_hi < prm->kf_lo || prm->f0 == 0.0 ? 0 : prm->kf_hi - prm->kf_lo + 1;
    F.norm0 = std::pow(2.0 * M_PI, 3) / std::pow((double)N, 6);
    F.f0 = prm->f0; F.as_factor = 1;
    F.out = p->factor; F.obs = p->Nf;
    return F;
  }

  // The integrating-factor table exp(-nu h k^2) for the current nu h, built on the stream when
  // nu h changes.  While the stream is being captured into a CUDA graph the table kernel is
  // recorded into the graph and the table is not marked built: the graph may never be replayed
  // (a discarded capture), so only a launch that runs marks it.
  static int ensure_ifac(ld_plan* p, double nuh, cudaStream_t s) {
    if (p->ifac_key == nuh) return LD_OK;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    LD_CUDA_CHECK(cudaStreamIsCapturing(s, &cap));
    ProfScope ps(p, KID_IFAC, s);
    k_ifac<T><<<grid1d(p->nifac, 256), 256, 0, s>>>((T*)p->ifac, p->nifac, nuh);
    LD_LAUNCH_CHECK();
    if (cap == cudaStreamCaptureStatusNone) p->ifac_key = nuh;
    return LD_OK;
  }

  // ---- pipelined fused z pass (rows inside a warp) -----------------------------------------------
  static int zcross_pipe(ld_plan* p, const C* W2, C* W1, T* uout, int ulayout, T sc, cudaStream_t s) {
    using ZP = ZPipe<T, N>;
    const long long NR = (long long)N * N * p->nbox;  // rows per field, all boxes
    auto k = k_z_cross_pipe<T, N>;
    if (int rc = set_smem(k, ZP::SMEM)) return rc;
    static int blocks_per_sm = -1;
    if (blocks_per_sm < 0) {
      int b = 0;
      cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k, ZP::WARPS * 32, ZP::SMEM);
      if (e != cudaSuccess) { ld_set_last_error(e); return LD_ERR_CUDA; }
      blocks_per_sm = b > 0 ? b : 1;
    }
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    long long grid = (long long)sms * blocks_per_sm;
    const long long need = cdiv(NR, (long long)ZP::WARPS * Z::R);
    if (grid > need) grid = need;
    LD_CUDA_CHECK(launch_dep(early(p), k, dim3((unsigned)grid), ZP::WARPS * 32, ZP::SMEM, s, W2, W1, uout, ulayout, sc,
                             (const C*)p->tw, p->status, p->wait_limit, p->wait_stall, NR));
    return LD_OK;
  }

  // ---- autotuner of the y passes: every launch variant timed on the plan's workspace ------------
  // (none where the right-hand side takes the plane pass: no y pass is launched)
  static int autotune(ld_plan* p, cudaStream_t s, double* ms) {
    if constexpr (PlaneCfg<T, N>::OK) {
      for (int v = 0; v < 8; ++v) ms[v] = -1.0;
      p->tune_y[0] = p->tune_y[1] = 0;
      LD_CUDA_CHECK(cudaStreamSynchronize(s));
      return LD_OK;
    } else {
      return autotune_y(p, s, ms);
    }
  }
  static int autotune_y(ld_plan* p, cudaStream_t s, double* ms) {
    const int My = p->My, Mzp = p->Mzp;
    const C* tw = (const C*)p->tw;
    C* W1 = (C*)p->W1;
    C* W2 = (C*)p->W2;
    const long long NN = (long long)N * N, w1s = (long long)N * My * Mzp, w2s = NN * Mzp;
    cudaEvent_t a, b;
    LD_CUDA_CHECK(cudaEventCreate(&a));
    LD_CUDA_CHECK(cudaEventCreate(&b));
    const int nv = PIPE ? 4 : 1;
    for (int pass = 0; pass < 2; ++pass) {
      double best = 1e30;
      int pick = -1;
      for (int v = 0; v < 4; ++v) {
        ms[4 * pass + v] = -1.0;
        if (v >= nv) continue;
        auto run = [&]() -> int {
          const int nb = p->nbox;
          if (pass == 0)
            return colpass_rows<true, true, RS::YC>(p, KID_YINV, io(W1, nb * w1s, (long long)My * Mzp),
                                            StRowsC<T, N, false, RS::YC>{io(W2, nb * w2s, (long long)N * Mzp)}, Mzp,
                                            6, nb * N, tw, s, v);
          return colpass_rows<false, false, RS::YC>(p, KID_YFWD, io(W1, nb * w2s, (long long)N * Mzp),
                                            StRowsC<T, N, true, RS::YC>{io(W2, nb * w1s, (long long)My * Mzp)}, Mzp,
                                            3, nb * N, tw, s, v);
        };
        if (int rc = run()) return rc;  // warm-up
        LD_CUDA_CHECK(cudaEventRecord(a, s));
        for (int r = 0; r < 5; ++r)
          if (int rc = run()) return rc;
        LD_CUDA_CHECK(cudaEventRecord(b, s));
        LD_CUDA_CHECK(cudaEventSynchronize(b));
        float t = 0.f;
        LD_CUDA_CHECK(cudaEventElapsedTime(&t, a, b));
        ms[4 * pass + v] = t / 5.0;
        if (t / 5.0 < best) { best = t / 5.0; pick = v; }
      }
      p->tune_y[pass] = PIPE ? pick : 0;
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    return LD_OK;
  }

  // ---- RHS pipeline: y (stage input) -> update epilogue ------------------------------------------
  template <int MODE>
  static int rhs(ld_plan* p, C* s0, C* s1, C* s2, T* uout, const ld_flow_params* prm, double visc,
                 cudaStream_t s, C* s3 = nullptr) {
    const int kc = p->kc, My = p->My, Mzp = p->Mzp;
    if (kc != Cfg<N>::KC || My != Cfg<N>::MY || Mzp != Cfg<N>::MZP)  // the kernels fix the cube by N
      return ld_fail(LD_ERR_UNSUPPORTED, "plan cube (%d, %d, %d) differs from N = %d's", kc, My, Mzp, N);
    const C* tw = (const C*)p->tw;
    const long long NN = (long long)N * N;
    const long long cs = p->cube_elems();
    C* W1 = (C*)p->W1;
    C* W2 = (C*)p->W2;
    const long long w1s = (long long)N * My * Mzp, w2s = NN * Mzp;
    const C* y = s1;  // stage input in every mode
    // boxes of a multi-box plan: each pass is one launch over all of them; the workspace holds
    // the box index next to x (fields (f, box, x, ...)), so that (box, x) is one outer index
    const int nb = p->nbox;
    if (nb > 1 && p->sm_vk) return ld_fail(LD_ERR_UNSUPPORTED, "slow-manifold output of a multi-box plan");
    // inverse x pass with the curl, 6 fields [u, w], and the forcing factors
    LdCurl<T, N> lc{y, cs, 3 * cs};
    auto xout = io(W1, nb * w1s, w1s);
    {
      ProfScope ps(p, KID_XINV, s);
      using St = StRowsC<T, N, false, RS::XC>;
      const ShellArgs<T> F = forcing(p, y, prm);
      const dim3 grid((unsigned)(cdiv(My * Mzp, TB) * 6 + F.nshell), (unsigned)nb);
      bool pairs = false;
      if constexpr (PAIRS) {
        pairs = aligned16(y);  // the state is the caller's buffer
        if (pairs) {
          auto k = k_xinv2<N, St>;
          if (int rc = set_smem(k, Col2<N>::SMEM)) return rc;
          LD_CUDA_CHECK(launch_dep(early(p), k, grid, Col2<N>::THREADS, Col2<N>::SMEM, s, lc, St{xout}, My * Mzp, tw, F));
        }
      }
      if (!pairs) {
        auto k = xinv_kernel<T, N, St>();
        if (int rc = set_smem(k, COL_SMEM)) return rc;
        LD_CUDA_CHECK(launch_dep(early(p), k, grid, Cfg<N>::COL_THREADS, COL_SMEM, s, lc, St{xout}, My * Mzp, tw, F));
      }
    }
    const T sc = T(1.0 / (double(N) * N * N));
    const int ulayout = (MODE == UPD_RHS) ? 0 : 1;  // the time steppers feed droplets: interleaved
    if constexpr (PlaneCfg<T, N>::OK) {
      // y inverse, fused z and y forward of one x plane per block (W1 -> W2 as (3, N, My, Mzp))
      using PC = PlaneCfg<T, N>;
      ProfScope ps(p, KID_ZCROSS, s);
      auto k = k_plane<T, N, 1>;
      if constexpr (N == 64 && sizeof(T) == 4) {
        if (nb * N >= 3 * kSMs) k = k_plane<T, N, 3>;
      }
      if (int rc = set_smem(k, PC::SMEM)) return rc;
      LD_CUDA_CHECK(launch_dep(early(p), k, dim3((unsigned)(nb * N)), PC::THREADS, PC::SMEM, s, W1, W2, uout, ulayout, sc, tw,
                               (long long)nb * N));
    } else {
      // inverse y pass
      auto yin = io(W1, nb * w1s, (long long)My * Mzp);
      auto yout = io(W2, nb * w2s, (long long)N * Mzp);
      if (int rc = colpass_rows<true, true, RS::YC>(p, KID_YINV, yin, StRowsC<T, N, false, RS::YC>{yout}, Mzp, 6, nb * N, tw, s))
        return rc;
      // fused z pass: u, w -> u x w  (W2 -> W1 as (3, N*N, Mzp))
      {
        ProfScope ps(p, KID_ZCROSS, s);
        if (int rc = zcross_pipe(p, W2, W1, uout, ulayout, sc, s)) return rc;
      }
      // forward y pass (W1 -> W2 as (3, N, My, Mzp))
      auto fyin = io(W1, nb * w2s, (long long)N * Mzp);
      auto fyout = io(W2, nb * w1s, (long long)My * Mzp);
      if (int rc = colpass_rows<false, false, RS::YC>(p, KID_YFWD, fyin, StRowsC<T, N, true, RS::YC>{fyout}, Mzp, 3, nb * N, tw, s))
        return rc;
    }
    // forward x pass + k-space update
    UpdArgs<T> A;
    A.nl = W2; A.nls = nb * w1s;
    A.nl_bs = w1s; A.cube_bs = 3 * cs; A.fac_bs = p->Nf;
    A.s0 = s0; A.s1 = s1; A.s2 = s2; A.s3 = s3; A.cs = cs;
    A.factor = p->factor; A.kf_lo = prm->kf_lo; A.kf_hi = (prm->f0 == 0.0) ? -1 : prm->kf_hi;
    A.ifac = (const T*)p->ifac;
    A.h = T(prm->dt); A.nu = T(prm->nu); A.visc = T(visc);
    A.kc = kc; A.My = My; A.Mzp = Mzp; A.status = p->status;
    A.vk = (C*)p->sm_vk; A.tps = T(p->sm_tps); A.vg = T(p->sm_tps * p->sm_g * (double)N * N * N);
    A.blowup = T(100.0 * (double)N * N * N);  // the blow-up threshold of the step epilogue (F:618)
    // the cube rows the update reads are staged in shared memory when that keeps 2 CTAs per SM
    const size_t pre_bytes = sizeof(C) * 3 * (size_t)(2 * kc + 1) * TB;
    const bool al = aligned16(MODE == UPD_RK2_2 ? s2 : s1);  // 16-byte copies from the caller's buffers
    A.prefetch = al && COL_SMEM + pre_bytes <= 112 * 1024 ? 1 : 0;
    const size_t smem = COL_SMEM + (A.prefetch ? pre_bytes : 0);
    ProfScope ps(p, KID_XFWD_UPD, s);
    auto k = k_xfwd_update<T, N, MODE>;
    if (int rc = set_smem(k, smem)) return rc;
    dim3 ugrid((unsigned)cdiv((long long)My * Mzp, TB), (unsigned)nb);
    LD_CUDA_CHECK(launch_dep(early(p), k, ugrid, Cfg<N>::COL_THREADS, smem, s, A, My * Mzp, tw));
    return LD_OK;
  }

  static int gather(ld_plan* p, const T* f, int ncomp, const double* pos, long long n, int method, T* out,
                    cudaStream_t s) {
    ProfScope ps(p, KID_GATHER, s);
    const int th = 256;
    const int g = grid1d(n, th);
    const double L = 2.0 * M_PI;
    if (method == LD_INTERP_TRILINEAR) k_gather<T, LD_INTERP_TRILINEAR><<<g, th, 0, s>>>(f, ncomp, N, L, pos, n, out);
    else if (method == LD_INTERP_TRICUBIC) k_gather<T, LD_INTERP_TRICUBIC><<<g, th, 0, s>>>(f, ncomp, N, L, pos, n, out);
    else k_gather<T, LD_INTERP_COSINE><<<g, th, 0, s>>>(f, ncomp, N, L, pos, n, out);
    LD_LAUNCH_CHECK();
    return LD_OK;
  }

  template <int M>
  static int dstage_m(ld_plan* p, int stage, const T* u, double* pos, T* vel, const T* tau, T* a1, long long n, double h,
                      double g, const int* box, cudaStream_t s) {
    ProfScope ps(p, stage == 1 ? KID_DROPLET1 : KID_DROPLET2, s);
    const int th = 256;
    const int gr = grid1d(n, th);
    const double L = 2.0 * M_PI;
    const vec4<T>* u4 = reinterpret_cast<const vec4<T>*>(u);
    auto k = stage == 1 ? k_droplet_stage<T, M, 1> : k_droplet_stage<T, M, 2>;
    LD_CUDA_CHECK(launch_dep(early_droplets(p, n, M != LD_INTERP_TRILINEAR), k, dim3(gr), th, 0, s, u4, N, L, pos, vel, tau, a1, n,
                             h, T(g), box));
    return LD_OK;
  }

  static int dstage(ld_plan* p, int stage, int method, const T* u, double* pos, T* vel, const T* tau, T* a1, long long n,
                    double h, double g, const int* box, cudaStream_t s) {
    if (method == LD_INTERP_TRILINEAR)
      return dstage_m<LD_INTERP_TRILINEAR>(p, stage, u, pos, vel, tau, a1, n, h, g, box, s);
    if (method == LD_INTERP_TRICUBIC)
      return dstage_m<LD_INTERP_TRICUBIC>(p, stage, u, pos, vel, tau, a1, n, h, g, box, s);
    return dstage_m<LD_INTERP_COSINE>(p, stage, u, pos, vel, tau, a1, n, h, g, box, s);
  }
};


// ---- type-erased wrappers ------------------------------------------------------------------
template <typename T, int N> struct Table {
  using O = Ops<T, N>;
  using C = ld::cplx<T>;
  static int rfft_full(ld_plan* p, const void* u, void* fu, int nc, cudaStream_t s) {
    return O::rfft_full(p, (const T*)u, (C*)fu, nc, s);
  }
  static int irfft_full(ld_plan* p, const void* fu, void* u, int nc, cudaStream_t s) {
    return O::irfft_full(p, (const C*)fu, (T*)u, nc, s);
  }
  static int irfft_cube(ld_plan* p, const void* uk, void* u, int nc, cudaStream_t s) {
    return O::irfft_cube(p, (const C*)uk, (T*)u, nc, s);
  }
  static int rfft_cube(ld_plan* p, const void* u, void* uk, int nc, cudaStream_t s) {
    return O::rfft_cube(p, (const T*)u, (C*)uk, nc, s);
  }
  static int to_cube(ld_plan* p, const void* full, void* cube, int nc, cudaStream_t s) {
    ProfScope ps(p, KID_CONVERT, s);
    const long long total = p->cube_elems() * nc;
    ld::k_to_cube<T><<<grid1d(total, 256), 256, 0, s>>>((const C*)full, (C*)cube, p->N, p->kc, p->My, p->Mzp, total);
    LD_LAUNCH_CHECK();
    return LD_OK;
  }
  static int from_cube(ld_plan* p, const void* cube, void* full, int nc, cudaStream_t s) {
    ProfScope ps(p, KID_CONVERT, s);
    const long long total = (long long)p->N * p->N * p->Nf * nc;
    ld::k_from_cube<T><<<grid1d(total, 256), 256, 0, s>>>((const C*)cube, (C*)full, p->N, p->kc, p->My, p->Mzp, total);
    LD_LAUNCH_CHECK();
    return LD_OK;
  }
  static int shell_spectrum(ld_plan* p, const void* uk, double* ek, cudaStream_t s) {
    ProfScope ps(p, KID_SHELL, s);
    ld::ShellArgs<T> A;
    A.u = (const C*)uk; A.cs = p->cube_elems(); A.ubs = 0;
    A.off = p->shell_off; A.idx = p->shell_idx; A.Mzp = p->Mzp;
    A.shell0 = 0; A.nshell = p->Nf;
    A.norm0 = std::pow(2.0 * M_PI, 3) / std::pow((double)N, 6);
    A.f0 = 0.0; A.as_factor = 0;
    A.out = ek; A.obs = 0;
    LD_CUDA_CHECK(launch_dep(true, ld::k_shell_sum<T>, dim3((unsigned)p->Nf), 256, 0, s, A));
    return LD_OK;
  }
  static int autotune(ld_plan* p, cudaStream_t s, double* ms) { return O::autotune(p, s, ms); }
  static int prepare(ld_plan* p, const ld_flow_params* prm, cudaStream_t s) {
    return O::ensure_ifac(p, prm->nu * prm->dt, s);
  }
  static int rhs(ld_plan* p, int mode, void* s0, void* s1, void* s2, void* s3, void* uout,
                 const ld_flow_params* prm, double visc, cudaStream_t s) {
    C *a = (C*)s0, *b = (C*)s1, *c = (C*)s2, *d = (C*)s3;
    if (mode == ld::UPD_RK2_1 || mode == ld::UPD_RK2_2)
      if (int rc = O::ensure_ifac(p, prm->nu * prm->dt, s)) return rc;
    switch (mode) {
      case ld::UPD_RHS: return O::template rhs<ld::UPD_RHS>(p, a, b, c, (T*)uout, prm, visc, s, d);
      case ld::UPD_RK2_1: return O::template rhs<ld::UPD_RK2_1>(p, a, b, c, (T*)uout, prm, visc, s, d);
      case ld::UPD_RK2_2: return O::template rhs<ld::UPD_RK2_2>(p, a, b, c, (T*)uout, prm, visc, s, d);
      case ld::UPD_RK4_1: return O::template rhs<ld::UPD_RK4_1>(p, a, b, c, (T*)uout, prm, visc, s, d);
      case ld::UPD_RK4_2: return O::template rhs<ld::UPD_RK4_2>(p, a, b, c, (T*)uout, prm, visc, s, d);
      case ld::UPD_RK4_3: return O::template rhs<ld::UPD_RK4_3>(p, a, b, c, (T*)uout, prm, visc, s, d);
      case ld::UPD_RK4_4: return O::template rhs<ld::UPD_RK4_4>(p, a, b, c, (T*)uout, prm, visc, s, d);
      default: return ld_fail(LD_ERR_ARG, "bad update mode %d", mode);
    }
  }
  static int epilogue(ld_plan* p, void* uk, cudaStream_t s) {
    ProfScope ps(p, KID_EPILOGUE, s);
    const long long total = p->cube_elems();
    const double blow = 100.0 * (double)N * N * N;
    dim3 grid((unsigned)grid1d(total, 256), (unsigned)p->nbox);
    ld::k_epilogue<T><<<grid, 256, 0, s>>>((C*)uk, total, p->kc, p->My, p->Mzp, T(blow), p->status);
    LD_LAUNCH_CHECK();
    return LD_OK;
  }  static int epilogue0(ld_plan* p, void* uk, cudaStream_t s) {
    ProfScope ps(p, KID_EPILOGUE, s);
    const double blow = 100.0 * (double)N * N * N;
    const long long plane = (long long)p->My * p->My;
    dim3 grid((unsigned)grid1d(plane, 256), (unsigned)p->nbox);
    LD_CUDA_CHECK(launch_dep(O::early(p), ld::k_epilogue_plane0<T>, grid, 256, 0, s, (C*)uk, p->cube_elems(), p->kc, p->My, p->Mzp,
                             T(blow), p->status));
    return LD_OK;
  }

  static int gather(ld_plan* p, const void* f, int nc, const double* pos, long long n, int method, void* out,
                    cudaStream_t s) {
    return O::gather(p, (const T*)f, nc, pos, n, method, (T*)out, s);
  }
  static int dstage(ld_plan* p, int stage, int method, const void* u, double* pos, void* vel, const void* tau,
                    void* a1, long long n, double h, double g, const int* box, cudaStream_t s) {
    return O::dstage(p, stage, method, (const T*)u, pos, (T*)vel, (const T*)tau, (T*)a1, n, h, g, box, s);
  }
  static const OpsTable* get() {
    static const OpsTable t = {rfft_full, irfft_full, irfft_cube, rfft_cube, to_cube, from_cube,
                               shell_spectrum, rhs, epilogue, epilogue0, gather, dstage, autotune, prepare};
    return &t;
  }
};

}  // namespace ld_impl

#define LD_DEFINE_TABLE(P, TT, N) \
  const OpsTable* ops_table_##P##_##N() { return ld_impl::Table<TT, N>::get(); }
