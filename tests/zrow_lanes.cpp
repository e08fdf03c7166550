// One warp of the one-shot z kernels (k_z_c2r, k_z_r2c) on the host, its lanes as coroutines: each
// runs alone from one barrier to the next, in rising or in falling order.  Nothing but the barriers
// orders the lanes, so a value that one lane changes while another still needs it comes out wrong.
// Prints, per precision, length and order, the largest error of both transforms against a direct sum.
#include <cuda_runtime.h>
#include <ucontext.h>

#include <cmath>
#include <complex>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <functional>
#include <random>
#include <type_traits>
#include <vector>

namespace {
struct Dim { unsigned x, y, z; };
Dim threadIdx{}, blockIdx{}, blockDim{32, 1, 1}, gridDim{1, 1, 1};
ucontext_t lanes[32], host;
bool done[32];
int running;
double mailbox[32];
std::function<void()> body;

void barrier() { swapcontext(&lanes[running], &host); }
void __syncwarp(unsigned = 0) { barrier(); }
void __syncthreads() { barrier(); }
template <typename V> V __shfl_sync(unsigned, V v, int src) {
  mailbox[running] = v;
  barrier();
  const V r = (V)mailbox[src & 31];
  barrier();
  return r;
}
template <typename V> V __shfl_down_sync(unsigned, V v, int) { return v; }
template <typename V> V __ldg(const V* p) { return *p; }
float __uint_as_float(unsigned u) { float f; std::memcpy(&f, &u, 4); return f; }
unsigned atomicOr(unsigned* p, unsigned v) { return *p |= v; }
int __all_sync(unsigned, int v) { return v; }
size_t __cvta_generic_to_shared(const void* p) { return (size_t)p; }
float2 __fadd2_rn(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
float2 __fmul2_rn(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
float2 __ffma2_rn(float2 a, float2 b, float2 c) { return make_float2(std::fma(a.x, b.x, c.x), std::fma(a.y, b.y, c.y)); }

void entry() {
  body();
  done[running] = true;
}

// all 32 lanes from barrier to barrier until they return
void warp(bool rising, std::function<void()> f) {
  static std::vector<char> stacks(32 << 20);
  body = std::move(f);
  for (int l = 0; l < 32; ++l) {
    getcontext(&lanes[l]);
    lanes[l].uc_stack.ss_sp = stacks.data() + ((size_t)l << 20);
    lanes[l].uc_stack.ss_size = 1 << 20;
    lanes[l].uc_link = &host;
    makecontext(&lanes[l], entry, 0);
    done[l] = false;
  }
  for (bool any = true; any;) {
    any = false;
    for (int i = 0; i < 32; ++i) {
      running = rising ? i : 31 - i;
      if (done[running]) continue;
      any = true;
      threadIdx.x = (unsigned)running;
      swapcontext(&host, &lanes[running]);
    }
  }
}
}  // namespace

#define __builtin_assume(x)
#define __launch_bounds__(...)
#define asm  // no inline PTX on the host: asm volatile(...) leaves nothing
#define volatile(...)
#include "ld_kernels.cuh"
#undef asm
#undef volatile

namespace ld {
alignas(16) unsigned char smem_raw[1 << 18];
}

template <typename T, int N> void check(const char* prec, bool rising) {
  using namespace ld;
  using C = cplx<T>;
  using Z = ZCfg<T, N>;
  constexpr int ROWS = 2 * (32 / (N / Z::E1)), K = N / 2 + 1;  // rows of the warp
  std::mt19937 rng(N);
  std::normal_distribution<double> gauss;
  std::vector<T> x(ROWS * N), back(ROWS * N);
  std::vector<C> X(ROWS * K), tw(N);
  for (auto& v : x) v = (T)gauss(rng);
  const double w = -2.0 * M_PI / N;
  for (int p = 0; p < N; ++p) tw[p] = cmk((T)std::cos(w * p), (T)std::sin(w * p));
  auto r2c = [&] { k_z_r2c<T, N>(x.data(), X.data(), ROWS, K, K, K, 0, 0, tw.data()); };
  auto c2r = [&] { k_z_c2r<T, N>(X.data(), back.data(), ROWS, K, K, T(1.0 / N), 0, 0, tw.data()); };
  warp(rising, r2c);
  double worst = 0.0;
  for (int r = 0; r < ROWS; ++r)
    for (int k = 0; k < K; ++k) {
      std::complex<double> s = 0.0;
      for (int n = 0; n < N; ++n) s += (double)x[r * N + n] * std::polar(1.0, w * (n * k % N));
      worst = std::fmax(worst, std::abs(s - std::complex<double>(X[r * K + k].x, X[r * K + k].y)) / std::sqrt((double)N));
    }
  warp(rising, c2r);
  for (int e = 0; e < ROWS * N; ++e) worst = std::fmax(worst, std::fabs((double)back[e] - (double)x[e]));
  std::printf("%s %d %d %.3e\n", prec, N, (int)rising, worst);
}

template <int... N> void all(std::integer_sequence<int, N...>) {
  for (bool rising : {true, false})
    (..., (check<float, N>("f32", rising), check<double, N>("f64", rising)));
}

int main() { all(std::integer_sequence<int, 16, 32, 64, 96, 128, 192, 256, 360, 384, 512>()); }
