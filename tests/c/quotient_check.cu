// Compares quot_rn (fp64.cuh) with the division operator bit for bit, and the
// approximate reciprocal behind it with its stated bound.  Prints one line per
// family: name, pairs, differences.
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <vector>

#include "fp64.cuh"

using namespace ddcsvd;

__device__ uint64_t mix(uint64_t x) {  // splitmix64's output function
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}

__device__ void compare(double a, double x, unsigned long long* diff) {
  const double q = quot_rn(a, x), w = a / x;
  if (__double_as_longlong(q) != __double_as_longlong(w) && !(isnan(q) && isnan(w))) atomicAdd(diff, 1ull);
}

__global__ void pairs_kernel(const double* a, const double* x, size_t n, unsigned long long* diff) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    compare(a[i], x[i], diff);
}

// random significands; exponents within 2^+-`span` of 1, signs both
__global__ void random_kernel(size_t n, int span, uint64_t seed, unsigned long long* diff) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint64_t r = mix(seed + 3 * i), s = mix(seed + 3 * i + 1), e = mix(seed + 3 * i + 2);
    const uint64_t ea = 1023 - span + (e & 0xffff) % (2 * span + 1), ex = 1023 - span + ((e >> 16) & 0xffff) % (2 * span + 1);
    compare(__longlong_as_double((long long)((r & 0x800fffffffffffffull) | ea << 52)),
            __longlong_as_double((long long)((s & 0x800fffffffffffffull) | ex << 52)), diff);
  }
}

// every high part of a significand, lowest and highest low part: |1 - x r| of the seed
__global__ void seed_kernel(unsigned long long* worst) {
  const unsigned h = blockIdx.x * blockDim.x + threadIdx.x;  // 2^20
  for (int k = 0; k < 2; k++) {
    const double x = __hiloint2double((int)(0x3ff00000u | h), k ? -1 : 0);
    const double e = fabs(fma(-x, rcp_approx(x), 1.0));
    atomicMax(worst, (unsigned long long)__double_as_longlong(e));
  }
}

static uint64_t rng_state = 12345;
static uint64_t rnd() {
  uint64_t x = rng_state += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}
static int failed = 0;

struct Pairs {
  std::vector<double> a, x;
  void add(double p, double q) {
    a.push_back(p);
    x.push_back(q);
  }
  void run(const char* name) {
    double *da, *dx;
    unsigned long long *dd, d = 0;
    cudaMalloc(&da, a.size() * 8);
    cudaMalloc(&dx, a.size() * 8);
    cudaMalloc(&dd, 8);
    cudaMemcpy(da, a.data(), a.size() * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(dx, x.data(), a.size() * 8, cudaMemcpyHostToDevice);
    cudaMemset(dd, 0, 8);
    pairs_kernel<<<512, 256>>>(da, dx, a.size(), dd);
    if (cudaMemcpy(&d, dd, 8, cudaMemcpyDeviceToHost) != cudaSuccess) failed = 1;
    printf("%s %zu %llu\n", name, a.size(), d);
    cudaFree(da);
    cudaFree(dx);
    cudaFree(dd);
  }
};

int main() {
  const uint64_t one = 1ull << 52;
  {  // divisors with significands next to all ones (and next to 1), simple and random numerators
    Pairs p;
    for (uint64_t k = 0; k < 4096; k++)
      for (int side = 0; side < 2; side++) {
        const double x = ldexp((double)(side ? 2 * one - 1 - k : one + k), -52);
        for (int e = -3; e <= 3; e++) p.add(ldexp(1.0, e), x);
        for (int t = 0; t < 16; t++) p.add(ldexp((double)(one | (rnd() >> 12)), -52), x);
        for (int t = 0; t < 8; t++) p.add(ldexp((double)(2 * one - 1 - (rnd() & 4095)), -52), x);
      }
    p.run("near_ones");
  }
  for (int top = 0; top < 2; top++) {  // quotients next to the midpoint of two doubles, for any divisor and for large ones
    Pairs p;
    while (p.a.size() < 400000) {
      const uint64_t X = (top ? 2 * one - 1 - (rnd() & ((1ull << (rnd() % 40)) - 1)) : one | (rnd() >> 12)) | 1;
      uint64_t inv = X;  // X^-1 mod 2^64
      for (int k = 0; k < 6; k++) inv *= 2 - X * inv;
      const int64_t t = (int64_t)(2 * (rnd() % 8) + 1) * ((rnd() & 1) ? 1 : -1);
      // an odd M of 54 bits with M X = t mod 2^53: (M X - t) / 2^53 over X is M / 2^53 but for t
      const uint64_t M = ((uint64_t)t * inv & (2 * one - 1)) | 2 * one;
      const __int128 A = ((__int128)M * X - t) >> 53;
      if (A >= 2 * one && (A & 1)) continue;
      p.add(ldexp((double)(uint64_t)A, (int)(rnd() % 41) - 20), ldexp((double)X, (int)(rnd() % 41) - 20));
    }
    p.run(top ? "midpoints_large_divisors" : "midpoints");
  }
  {  // the ends of mid_range and beyond; zeros, subnormals, infinities, NaN
    Pairs p;
    std::vector<double> v = {0.0, -0.0, 5e-324, 2.2250738585072014e-308, 1.7976931348623157e308, INFINITY, -INFINITY, NAN};
    for (int e : {-1022, -1000, -512, -502, -501, -500, -499, -498, -1, 0, 1, 498, 499, 500, 501, 502, 512, 1000, 1023})
      for (int k = 0; k < 40; k++) v.push_back(ldexp((double)(k < 2 ? one + k : k < 4 ? 2 * one - k + 1 : one | (rnd() >> 12)), e - 52));
    for (double a : v)
      for (double x : v) {
        p.add(a, x);
        p.add(-a, x);
      }
    p.run("range_ends");
  }
  unsigned long long *dd, d = 0;
  cudaMalloc(&dd, 8);
  for (int span : {0, 20, 498}) {
    cudaMemset(dd, 0, 8);
    random_kernel<<<2048, 256>>>(1ull << 26, span, 1000 + span, dd);
    if (cudaMemcpy(&d, dd, 8, cudaMemcpyDeviceToHost) != cudaSuccess) failed = 1;
    printf("random_%d %llu %llu\n", span, 1ull << 26, d);
  }
  cudaMemset(dd, 0, 8);
  seed_kernel<<<4096, 256>>>(dd);
  if (cudaMemcpy(&d, dd, 8, cudaMemcpyDeviceToHost) != cudaSuccess) failed = 1;
  double worst;
  memcpy(&worst, &d, 8);
  printf("seed_log2 %.3f 0\n", log2(worst));
  printf("%s\n", failed ? "cuda_error 0 1" : "done 0 0");
  return failed;
}
