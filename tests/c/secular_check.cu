// Secular roots of the short form (dc.cu, sec_root without kBits) at several
// scales of the problem against the same roots at scale 1 with every rounding
// kept.  Prints per scale (as a power of two) the largest relative difference of
// sigma^2 in units of 2^-53, of the short form and of the plain one.
#include <math.h>
#include <stdint.h>
#include <stdio.h>

#include <algorithm>
#include <vector>

#include "dc.cu"

namespace ddcsvd {

__global__ void roots_kernel(int q, int nprob, double scale, const double* d1, const double* z1, const double* zz1,
                             double* d, double* z, float2* df, float* zf, double* worst, bool plain) {
  const int lane = threadIdx.x & 31, prob = blockIdx.x;
  const double* dp = d1 + (size_t)prob * q;
  const double* zp = z1 + (size_t)prob * q;
  double* ds = d + (size_t)prob * q;
  double* zs = z + (size_t)prob * q;
  float2* dfs = df + (size_t)prob * 2 * q;
  float* zfs = zf + (size_t)prob * 2 * q;
  auto copies = [&](const double* dd, const double* zd, float2* f, float* g) {
    for (int j = threadIdx.x; j < q; j += blockDim.x) {
      const float h = (float)dd[j];
      f[j] = make_float2(h, (float)(dd[j] - (double)h));
      g[j] = (float)zd[j];
    }
  };
  for (int j = threadIdx.x; j < q; j += blockDim.x) {
    ds[j] = dp[j] * scale;
    zs[j] = zp[j] * scale;
  }
  __syncthreads();
  copies(dp, zp, dfs, zfs);
  copies(ds, zs, dfs + q, zfs + q);
  __syncthreads();
  const LaneGroup<32> g = make_group<32>(32, lane);
  for (int i = threadIdx.x >> 5; i < q; i += blockDim.x >> 5) {
    int o, os;
    double t, ts;
    const bool ok = sec_root<true, 32>(q, dp, zp, dfs, zfs, zz1[prob], i, g, 80, &o, &t);
    const double zzs = zz1[prob] * scale * scale;
    const bool oks = plain ? sec_root<true, 32>(q, ds, zs, dfs + q, zfs + q, zzs, i, g, 80, &os, &ts)
                           : sec_root<false, 32>(q, ds, zs, dfs + q, zfs + q, zzs, i, g, 80, &os, &ts);
    if (lane == 0) {
      const double want = fma(dp[o], dp[o], t);
      // sigma^2 - d_os^2 of both, so that no cancellation hides an error of tau
      const double tw = (os == o) ? t : t + (dp[o] - dp[os]) * (dp[o] + dp[os]);
      const double e = (ok && oks) ? fabs(ts / (scale * scale) - tw) / want : 1e300;
      atomicMax(reinterpret_cast<unsigned long long*>(worst), (unsigned long long)__double_as_longlong(e));
    }
  }
}

}  // namespace ddcsvd

using namespace ddcsvd;

static uint64_t state = 7;
static double uni() {
  uint64_t x = state += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return (double)((x ^ (x >> 31)) >> 11) * 0x1p-53;
}

int main() {
  const int q = 48, nprob = 4000;
  std::vector<double> d(q * nprob), z(q * nprob), zz(nprob);
  for (int p = 0; p < nprob; p++) {
    double* a = &d[(size_t)p * q];
    for (int j = 0; j < q; j++)
      a[j] = (p % 4 == 0) ? uni() + j : (p % 4 == 1) ? pow(10.0, 4.0 * uni() - 4.0) : (p % 4 == 2) ? 1.0 + 1e-3 * uni() : pow(10.0, 6.0 * uni() - 6.0);
    a[0] = 0.0;
    std::sort(a, a + q);
    double s = 0.0;
    for (int j = 0; j < q; j++) {
      // (the last kind: roots so near to their poles that tau leaves FP32's range)
      const double v = (uni() < 0.2 ? (p % 4 == 3 ? 1e-15 : 1e-3) : 1.0) * (2.0 * uni() - 1.0) * a[q - 1];
      z[(size_t)p * q + j] = v;
      s += v * v;
    }
    zz[p] = s;
  }
  double *dd, *dz, *dzz, *d2, *z2, *w;
  float2* df;
  float* zf;
  const size_t n = (size_t)q * nprob;
  cudaMalloc(&dd, 8 * n);
  cudaMalloc(&dz, 8 * n);
  cudaMalloc(&dzz, 8 * nprob);
  cudaMalloc(&d2, 8 * n);
  cudaMalloc(&z2, 8 * n);
  cudaMalloc(&df, 16 * n);
  cudaMalloc(&zf, 8 * n);
  cudaMalloc(&w, 8);
  cudaMemcpy(dd, d.data(), 8 * n, cudaMemcpyHostToDevice);
  cudaMemcpy(dz, z.data(), 8 * n, cudaMemcpyHostToDevice);
  cudaMemcpy(dzz, zz.data(), 8 * nprob, cudaMemcpyHostToDevice);
  for (int e : {0, -30, -45, -50, -55, -58, -60, -70, 30, 55, 60, 62, 63, 64, 70}) {
    double h[2];
    for (int plain = 0; plain < 2; plain++) {
      cudaMemset(w, 0, 8);
      roots_kernel<<<nprob, 128>>>(q, nprob, ldexp(1.0, e), dd, dz, dzz, d2, z2, df, zf, w, plain);
      if (cudaMemcpy(h + plain, w, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    }
    printf("%d %.2f %.2f\n", e, h[0] * 0x1p53, h[1] * 0x1p53);
  }
  return 0;
}
