// bx_diag.cu -- FP64 FMA throughput probe (include/boxzy_diag.h).
#include <cuda_runtime.h>

#include "../../include/boxzy_diag.h"
#include "bx_math.cuh"

namespace {
constexpr int kChains = 8;
constexpr int kIters = 2048;

__global__ void __launch_bounds__(256) k_dfma(double* out, double seed) {
  double a[kChains];
  const double b = 1.0 + 1e-9 * threadIdx.x, c = 1e-12 * blockIdx.x;
#pragma unroll
  for (int k = 0; k < kChains; ++k) a[k] = seed + k;
  for (int it = 0; it < kIters; ++it) {
#pragma unroll
    for (int k = 0; k < kChains; ++k) a[k] = fma(a[k], b, c);
  }
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < kChains; ++k) s += a[k];
  if (s == 1234.5678) out[0] = s;  // keeps the chains live
}
}  // namespace

namespace {
// splitmix64 stream -> doubles with random mantissa and exponent in [-e, e]
__device__ __forceinline__ unsigned long long mix(unsigned long long z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ double rnd(unsigned long long z, int erange, bool sign) {
  const unsigned long long mant = z & 0xfffffffffffffull;
  const int ex = (int)((z >> 52) % (2 * erange + 1)) - erange;
  unsigned long long bits = mant | ((unsigned long long)(ex + 1023) << 52);
  if (sign && ((z >> 63) & 1)) bits |= 1ull << 63;
  return __longlong_as_double((long long)bits);
}
__global__ void k_divcheck(unsigned long long n, unsigned long long seed, int erange,
                           unsigned long long* bad, double* example) {
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += stride) {
    const unsigned long long z1 = mix(seed ^ (2 * i)), z2 = mix(seed ^ (2 * i + 1));
    const double d = rnd(z1, erange, false);
    double a = rnd(z2, erange, true);
    if ((i & 7) == 0) a = d * (double)(long long)(z2 % 1000003ull);  // exact multiples
    if ((i & 15) == 1) a = __longlong_as_double(__double_as_longlong(d) + (long long)(z2 % 5) - 2);
    if ((i & 31) == 2) a = ((z2 >> 7) & 1) ? -0.0 : 0.0;  // signed zeros
    const bx::SharedDiv div(d);
    const double q = div(a), q2 = bx::cdiv(a, d, 1.0 / d), ref = a / d;
    const bool ok1 = __double_as_longlong(q) == __double_as_longlong(ref) || (q == 0.0 && ref == 0.0);
    // cdiv serves grid constants, which bx_create keeps inside [2^-450, 2^450]
    const bool in_window = d >= 0x1p-450 && d <= 0x1p+450;
    bool ok4 = true;
    if (bx::den_fast_ok(d))
      ok4 = __double_as_longlong(bx::rcp_fast(d)) == __double_as_longlong(1.0 / d);
    const bool ok2 = !in_window || __double_as_longlong(q2) == __double_as_longlong(ref) ||
                     (q2 == 0.0 && ref == 0.0);
    // the HLL form: every bit of the IEEE quotient, the sign of a zero included,
    // wherever quot_fast_ok admits the numerator and d lies in the window
    bool ok3 = true;
    if (bx::den_fast_ok(d) && bx::quot_fast_ok(a)) {
      const double q3 = bx::quot_fast(a, d, bx::rcp_fast(d));
      ok3 = __double_as_longlong(q3) == __double_as_longlong(ref);
    }
    if (!(ok1 && ok2 && ok3 && ok4)) {
      if (atomicAdd(bad, 1ull) == 0) { example[0] = a; example[1] = d; }
    }
  }
}

// sqrt_fast against the IEEE square root: the n given arguments, then `nrandom`
// random ones with exponents in [-e, e]
__global__ void k_rootcheck(const double* q, unsigned long long n, unsigned long long nrandom,
                            unsigned long long seed, int erange, unsigned long long* bad,
                            double* example) {
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
       i < n + nrandom; i += stride) {
    const double x = i < n ? q[i] : rnd(mix(seed ^ i), erange, false);
    if (__double_as_longlong(bx::sqrt_fast(x)) != __double_as_longlong(sqrt(x)))
      if (atomicAdd(bad, 1ull) == 0) example[0] = x;
  }
}
}  // namespace

extern "C" int bx_check_root(const double* q, unsigned long long n, unsigned long long nrandom,
                             unsigned long long seed, int exp_range,
                             unsigned long long* mismatches, double* example) {
  if ((n && !q) || exp_range < 0 || exp_range > 900) return 1;
  double* d = nullptr;
  unsigned long long* bad = nullptr;
  const size_t bytes = n * sizeof(double);
  if (cudaMalloc(&d, bytes + sizeof(double)) != cudaSuccess) return 5;
  if (cudaMalloc(&bad, sizeof(*bad)) != cudaSuccess) { cudaFree(d); return 5; }
  cudaMemset(bad, 0, sizeof(*bad));
  cudaMemset(d + n, 0, sizeof(double));
  if (n) cudaMemcpy(d, q, bytes, cudaMemcpyHostToDevice);
  k_rootcheck<<<1184, 256>>>(d, n, nrandom, seed, exp_range, bad, d + n);
  unsigned long long h = 0;
  double hx = 0.0;
  cudaMemcpy(&h, bad, sizeof(h), cudaMemcpyDeviceToHost);
  cudaMemcpy(&hx, d + n, sizeof(hx), cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(bad);
  if (mismatches) *mismatches = h;
  if (example) *example = hx;
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

namespace {
__global__ void k_logcheck(unsigned long long n, unsigned long long seed, double low, double step,
                           int steps, unsigned long long* bad, double* example) {
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += stride) {
    const unsigned long long z = mix(seed ^ i);
    // a step's edge (down to two below the table), off by 2^-1 .. 2^-53 of itself or not at all
    const double edge = exp10(low + ((double)(z % (unsigned)(steps + 3)) - 2.0) * step);
    const double off = (z >> 40 & 63) > 53 ? 0.0 : ldexp((z >> 39 & 1) ? 1.0 : -1.0, -(int)(z >> 40 & 63));
    const double x = edge + edge * off;
    if (bx::log_steps(x, low, step) != (int)((log10(x) - low) / step))
      if (atomicAdd(bad, 1ull) == 0) example[0] = x;
  }
}
}  // namespace

extern "C" int bx_check_log_steps(unsigned long long n, unsigned long long seed, double low,
                                  double step, int steps, unsigned long long* mismatches,
                                  double* example) {
  if (steps < 1 || !(step > 0.0)) return 1;
  unsigned long long* bad = nullptr;
  double* ex = nullptr;
  if (cudaMalloc(&bad, sizeof(*bad)) != cudaSuccess) return 5;
  if (cudaMalloc(&ex, sizeof(double)) != cudaSuccess) { cudaFree(bad); return 5; }
  cudaMemset(bad, 0, sizeof(*bad));
  cudaMemset(ex, 0, sizeof(double));
  k_logcheck<<<1184, 256>>>(n, seed, low, step, steps, bad, ex);
  unsigned long long h = 0;
  double hx = 0.0;
  cudaMemcpy(&h, bad, sizeof(h), cudaMemcpyDeviceToHost);
  cudaMemcpy(&hx, ex, sizeof(hx), cudaMemcpyDeviceToHost);
  cudaFree(bad);
  cudaFree(ex);
  if (mismatches) *mismatches = h;
  if (example) *example = hx;
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

extern "C" int bx_check_shared_division(unsigned long long n, unsigned long long seed,
                                         int exp_range, unsigned long long* mismatches,
                                         double* example_a, double* example_d) {
  unsigned long long* bad = nullptr;
  double* ex = nullptr;
  if (cudaMalloc(&bad, sizeof(unsigned long long)) != cudaSuccess) return 5;
  if (cudaMalloc(&ex, 2 * sizeof(double)) != cudaSuccess) { cudaFree(bad); return 5; }
  cudaMemset(bad, 0, sizeof(unsigned long long));
  cudaMemset(ex, 0, 2 * sizeof(double));
  k_divcheck<<<1184, 256>>>(n, seed, exp_range, bad, ex);
  unsigned long long h = 0;
  double hx[2] = {0, 0};
  cudaMemcpy(&h, bad, sizeof(h), cudaMemcpyDeviceToHost);
  cudaMemcpy(hx, ex, sizeof(hx), cudaMemcpyDeviceToHost);
  cudaFree(bad);
  cudaFree(ex);
  if (mismatches) *mismatches = h;
  if (example_a) *example_a = hx[0];
  if (example_d) *example_d = hx[1];
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

extern "C" int bx_fp64_peak(double* tflops, double* ms_out) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 2;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  double* out = nullptr;
  if (cudaMalloc(&out, sizeof(double)) != cudaSuccess) return 5;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  const int blocks = sms * 8, threads = 256;
  for (int w = 0; w < 3; ++w) k_dfma<<<blocks, threads>>>(out, 1.0);
  float best = 1e30f;
  for (int r = 0; r < 5; ++r) {
    cudaEventRecord(e0);
    k_dfma<<<blocks, threads>>>(out, 1.0);
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (ms < best) best = ms;
  }
  const double flops = 2.0 * kChains * (double)kIters * blocks * threads;
  if (tflops) *tflops = flops / (best * 1e-3) / 1e12;
  if (ms_out) *ms_out = best;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
