// Errors of householder_fast and of the sums behind it (common.cuh) against
// FP64: prints the largest relative errors, in units of 2^-24 (of 2^-46 for the
// sums).
#include <math.h>
#include <stdint.h>
#include <stdio.h>

#include "common.cuh"

using namespace ddcsvd;

__device__ uint64_t mix(uint64_t x) {  // splitmix64's output function
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}
__device__ float value(uint64_t r, int ex) {
  return __uint_as_float(((unsigned)r & 0x807fffffu) | (unsigned)(127 + ex) << 23);
}
__device__ void worst(double* w, double e) {
  atomicMax(reinterpret_cast<unsigned long long*>(w), (unsigned long long)__double_as_longlong(e));
}

// x0 2^-k to 2^k of the tail's norm, both over 2^+-`span`
__global__ void reflectors(unsigned n, int span, double* w) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint64_t a = mix(3ull * i), b = mix(3ull * i + 1), c = mix(3ull * i + 2);
    const int ex = (int)(c % (2 * span + 1)) - span, rel = (int)((c >> 20) % 25) - 12;
    const float x0 = value(a, ex), h = fabsf(value(b, max(-110, min(110, 2 * (ex + rel)))));
    const FF t2{h, ldexpf((float)(int)(b >> 32), -31) * h * 0x1p-25f};
    const double x = x0, nn = sqrt((double)t2.hi + t2.lo + x * x), sg = x < 0 ? -1.0 : 1.0;
    float al, ta, sc;
    householder_fast(x0, t2, &al, &ta, &sc);
    worst(w, fabs(al / (-sg * nn) - 1));
    worst(w + 1, fabs(ta / ((nn + fabs(x)) / nn) - 1));
    worst(w + 2, fabs(sc / (sg / (fabs(x) + nn)) - 1));
  }
}

// a warp's sum of 32 R squares of values over a range of magnitudes
template <int R>
__global__ void sums(unsigned n, double* w) {
  const int lane = threadIdx.x & 31;
  for (unsigned i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
    FF v{0.f, 0.f};
    double d = 0.0;  // squares of FP32 values are exact in FP64
    for (int q = 0; q < R; q++) {
      const uint64_t r = mix(((uint64_t)i * 32 + lane) * R + q);
      const float x = value(r, (int)((r >> 40) % 17) - 8);
      v = ff_acc(v, ff_square(x));
      d += (double)x * x;
    }
    v = ff_lanes<32>(v);
    d = warp_sum(d);
    if (lane == 0) worst(w, fabs(((double)v.hi + v.lo) / d - 1));
  }
}

__global__ void zeros(float* out) { householder_fast(0.f, FF{0.f, 0.f}, out, out + 1, out + 2); }

int main() {
  double *w, h[8];
  cudaMalloc(&w, sizeof h);
  cudaMemset(w, 0, sizeof h);
  reflectors<<<1024, 256>>>(1u << 25, 8, w);
  reflectors<<<1024, 256>>>(1u << 25, 40, w);
  sums<2><<<1024, 256>>>(1u << 18, w + 3);
  sums<24><<<1024, 256>>>(1u << 16, w + 3);
  zeros<<<1, 1>>>(reinterpret_cast<float*>(w + 4));
  if (cudaMemcpy(h, w, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  const float* z = reinterpret_cast<const float*>(h + 4);
  printf("alpha %.4f\ntau %.4f\nscale %.4f\nsum %.4f\nzero %.1f\n", h[0] * 0x1p24, h[1] * 0x1p24, h[2] * 0x1p24,
         h[3] * 0x1p46, fabs(z[0]) + fabs(z[1]) + fabs(z[2]));
  return 0;
}
