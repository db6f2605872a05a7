// adjoint.cu -- reverse-mode derivative of the thin SVD A = U diag(s) V^T
// (m >= n, k = n) for a batch of equally sized problems, FP64 or FP32.
//
//   J = U^T gU,  K = V^T gV                                (k x k)
//   F_ij = 1 / (s_j^2 - s_i^2) for i != j, 0 on the diagonal
//   M = diag(gs) + (F o (J - J^T)) S + S (F o (K - K^T)) - J S^-1
//   gA = (U M + gU S^-1) V^T
// which equals U [diag(gs) + (F o (J - J^T)) S + S (F o (K - K^T))] V^T
// + (I - U U^T) gU S^-1 V^T.  (The reference has no derivative; this is the
// standard SVD adjoint.)  Any of gU, gs, gV may be null (zero).
//
// FP32 problems whose matrices fit one CTA's shared memory take one launch
// (adjoint_fused_kernel).  Otherwise four: J and K together, an elementwise kernel
// for M, then P = U M + gU S^-1 and gA = P V^T, all batched products of any
// strides.  FP32 products run on the FP32 pipe; FP64 ones on the tensor cores, on
// digits (ozgemm_kernel), because GB300's FP64 pipe is 1/64 of FP32's.
#include <cudaTypedefs.h>

#include <cuda_fp16.h>

#include "ctx_cache.hpp"
#include "fp64.cuh"
#include "internal.hpp"

namespace ddcsvd {

__device__ __forceinline__ float adj_quot(float a, float x) { return a / x; }
__device__ __forceinline__ double adj_quot(double a, double x) { return quot_rn(a, x); }
// a / x with rx = 1 / x at hand: the quotient and one correction by its remainder
// (the product alone is up to an ulp worse than a division)
__device__ __forceinline__ float adj_quot(float a, float x, float) { return a / x; }
__device__ __forceinline__ double adj_quot(double a, double x, double rx) {
  if (!(mid_range(a) && mid_range(rx))) return a / x;
  const double q = a * rx;
  return fma(fma(-x, q, a), rx, q);
}

// A matrix of every problem: element (r, c) of problem b at p + b*b_ + r*r_ + c*c_.
template <typename T>
struct BMat {
  const T* p;
  long long r, c, b;
};

// C[b] (M x N, column-major, ldc) = A[b] B[b] + X[b] diag(s[b])^-1 (X.p may be null).
template <typename T>
struct BGemm {
  int M, N, K;
  BMat<T> A, B, X;
  const T* s;
  long long sb;
  T* C;
  int ldc;
  long long cb;
};

// 64 x 64 tiles, 256 threads with 4 x 4 outputs each (rows ty + 16 a, columns
// tx + 16 c), K in slabs of 16.  Tile loads walk the operand's unit-stride index
// fastest, so either layout of A and B (the adjoint reads U, V transposed and
// not) is read in coalesced segments.  blockIdx.z: problem, first of g0, then of
// g1.
constexpr int kBgTile = 64, kBgK = 16;

template <typename T>
__device__ __forceinline__ void bgemm_load(T (*dst)[kBgTile + 1], const T* __restrict__ src, long long s_mn,
                                           long long s_k, int mn0, int MN, int k0, int K) {
  // dst[kk][i] = element (mn0 + i, k0 + kk); the index with stride 1 varies fastest across threads
  const bool k_fast = (s_k == 1 && s_mn != 1);
  for (int idx = threadIdx.x; idx < kBgTile * kBgK; idx += blockDim.x) {
    int i, kk;
    if (k_fast) { kk = idx % kBgK; i = idx / kBgK; }
    else { i = idx % kBgTile; kk = idx / kBgTile; }
    const int r = mn0 + i, k = k0 + kk;
    dst[kk][i] = (r < MN && k < K) ? src[r * s_mn + k * s_k] : T(0);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) bgemm_kernel(BGemm<T> g0, BGemm<T> g1, int batch) {
  __shared__ T At[kBgK][kBgTile + 1];
  __shared__ T Bt[kBgK][kBgTile + 1];
  const bool first = (int)blockIdx.z < batch;
  const BGemm<T> g = first ? g0 : g1;
  const int b = first ? blockIdx.z : blockIdx.z - batch;
  const int r0 = blockIdx.x * kBgTile, c0 = blockIdx.y * kBgTile;
  if (r0 >= g.M || c0 >= g.N) return;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const T* Ab = g.A.p + b * g.A.b;
  const T* Bb = g.B.p + b * g.B.b;
  T acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int c = 0; c < 4; c++) acc[a][c] = T(0);
  for (int k0 = 0; k0 < g.K; k0 += kBgK) {
    bgemm_load<T>(At, Ab, g.A.r, g.A.c, r0, g.M, k0, g.K);
    bgemm_load<T>(Bt, Bb, g.B.c, g.B.r, c0, g.N, k0, g.K);
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kBgK; kk++) {
      T x[4], y[4];
#pragma unroll
      for (int a = 0; a < 4; a++) {
        x[a] = At[kk][ty + 16 * a];
        y[a] = Bt[kk][tx + 16 * a];
      }
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[a][c] += x[a] * y[c];
    }
    __syncthreads();
  }
  T* Cb = g.C + b * g.cb;
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const int r = r0 + ty + 16 * a, cc = c0 + tx + 16 * c;
      if (r < g.M && cc < g.N) {
        T v = acc[a][c];
        if (g.X.p) v += adj_quot(g.X.p[b * g.X.b + r * g.X.r + cc * g.X.c], g.s[b * g.sb + cc]);
        Cb[r + (size_t)cc * g.ldc] = v;
      }
    }
}

// ---------------------------------------------------------------- FP64 products on the tensor cores
// The Ozaki scheme (Ozaki, Ogita, Oishi, Rump, "Error-free transformations of
// matrix multiplication", Numer. Algorithms 59, 2012; on FP16 tensor cores:
// Mukunoki, Ozaki, Ogita, Imamura, ISC 2020): every row of A and column of B is
// scaled by a power of two and rounded to a 62-bit integer, the integer written
// in eight signed base-256 digits, and each pair of digit matrices multiplied in
// FP16 with FP32 accumulation.  Digits are at most 128 in magnitude (the first
// 64), so a sum of up to eight pairs over K = 128 stays below 2^24 and every
// accumulation is exact; the 36 pairs of weight 256^14 .. 256^7 are kept and put
// together in 64-bit integers.
//
// What is lost, the pairs below and the bits beyond 62, is relative to the
// largest entries of the row and of the column: about 2^-59 sqrt(K) of their
// product.  An FP64 sum keeps the bits of each of its products, however small
// beside those entries, so the digits stand in for it only where they are as
// good: the first digits' magnitudes are multiplied too, and an element whose
// sum of |a| |b| falls below 2^-11 sqrt(K) of the product of the largest entries
// (where the loss reaches four roundings of that sum) is formed as an FP64 sum
// after all -- by its warp, or by the CTA where a tile has more than a few of them
// or holds Inf or NaN.  (Seven digits of 54 bits without that test lost the
// columns of an unevenly scaled problem: A = X diag(scale) with V near the
// identity, 8 decades, 3e-9 of a column instead of 5e-16.)  Against extended
// precision the worst column of the adjoint is 0.3 to 1 times as far off as with
// FP64 sums, for even and graded values, V or U near the identity, and each
// gradient alone.
//
// The FP64 pipe bounded the direct form (0.98 ms for the four products of 256 x
// (128 x 64), 0.85 ms at cuBLAS's DGEMM rate); this one is bound by the tensor
// pipe and the digit extraction (integer instructions).
//
// 64 x 32 tile per CTA, eight warps of 16 x 16, two CTAs per SM (one extracts
// digits while the other multiplies), K in slabs of 32 through two stages.
constexpr int kOzThreads = 256;
constexpr int kOzM = 64, kOzN = 32, kOzK = 32;           // tile, slab
constexpr int kOzD = 8, kOzS = 8;                        // digits, diagonals
constexpr int kOzChunk = 128;                            // K per exact accumulation
constexpr int kOzStage = kOzD * (kOzM + kOzN) * kOzK;    // halves per stage: A's digits, then B's
constexpr int kOzSmem = 2 * kOzStage * (int)sizeof(__half);
constexpr int kOzFew = 64;                               // elements of a tile that warps sum in FP64 one by one

// Place of the eight halves k .. k + 7 of a staged row: rows are 64 bytes, their
// 16-byte parts exchanged so that eight rows of ldmatrix meet distinct banks.
__device__ __forceinline__ int oz_at(int row, int k) { return row * kOzK + ((((k >> 3) ^ (row >> 1)) & 3) << 3); }

// One operand of the tile: R rows (of A, or columns of B) by K.
struct OzOp {
  const double* p;  // problem's matrix at the tile's first row
  long long s_r, s_k;
  int rows;  // valid rows
  int K;
  bool k_fast;  // K has the unit stride
};
// Unit u of an R x 32 slab: eight consecutive k of one row (a 16-byte store per
// digit); consecutive threads walk the operand's unit stride.
template <int R>
__device__ __forceinline__ void oz_place(const OzOp& o, int u, int& r, int& k) {
  if (o.k_fast) {
    r = u >> 2;
    k = 8 * (u & 3);
  } else {
    r = u % R;
    k = 8 * (u / R);
  }
}
template <int R>
__device__ __forceinline__ void oz_load(const OzOp& o, int k0, int u, double (&v)[8]) {
  int r, k;
  oz_place<R>(o, u, r, k);
  k += k0;
  const double* q = o.p + r * o.s_r + k * o.s_k;
#pragma unroll
  for (int h = 0; h < 8; h++) v[h] = (r < o.rows && k + h < o.K) ? q[h * o.s_k] : 0.0;
}
template <int R>
__device__ __forceinline__ bool oz_max(const OzOp& o, int* e) {  // exponents of the largest entries; any non-finite?
  bool bad = false;
  for (int u = threadIdx.x; u < 4 * R; u += kOzThreads) {
    int ex = 1, r, k;
    oz_place<R>(o, u, r, k);
#pragma unroll 2
    for (int k0 = 0; k0 < o.K; k0 += kOzK) {
      double v[8];
      oz_load<R>(o, k0, u, v);
#pragma unroll
      for (int h = 0; h < 8; h++) ex = max(ex, (__double2hiint(v[h]) >> 20) & 0x7ff);
    }
    atomicMax(&e[r], ex);
    bad = bad || ex == 0x7ff;
  }
  return bad;
}
// v 2^(62 - e) rounded to an integer, where |v| < 2^e, plus 128 in each byte:
// byte t is then digit t + 128
__device__ __forceinline__ unsigned long long oz_digits(double v, int e) {
  const long long b = __double_as_longlong(v);
  const int ex = (int)((b >> 52) & 0x7ff);
  unsigned long long m = (unsigned long long)b & 0xfffffffffffffull;
  if (ex) m |= 0x10000000000000ull;
  const int sh = (ex ? ex : 1) - 1075 + 62 - e;  // at most 9
  unsigned long long x;
  if (sh >= 0) x = m << sh;
  else if (sh > -64) x = (m + (1ull << (-sh - 1))) >> -sh;
  else x = 0;
  return (b < 0 ? 0ull - x : x) + 0x8080808080808080ull;
}
// digits of one slab into a stage: digit d (0 = most significant) of row r at
// dst + oz_at(d R + r, k)
template <int R>
__device__ __forceinline__ void oz_stage(const OzOp& o, const int* e, int k0, __half* dst) {
  for (int u = threadIdx.x; u < 4 * R; u += kOzThreads) {
    double v[8];
    oz_load<R>(o, k0, u, v);
    int r, k;
    oz_place<R>(o, u, r, k);
    const int er = e[r];
    unsigned long long y[8];
#pragma unroll
    for (int h = 0; h < 8; h++) y[h] = oz_digits(v[h], er);
    __half* q = dst + oz_at(r, k);
#pragma unroll
    for (int d = 0; d < kOzD; d++) {
      const int t = kOzD - 1 - d;  // byte
      const unsigned by = t & 3;
      unsigned w[4];
#pragma unroll
      for (int h = 0; h < 4; h++) {
        const unsigned w0 = t < 4 ? (unsigned)y[2 * h] : (unsigned)(y[2 * h] >> 32);
        const unsigned w1 = t < 4 ? (unsigned)y[2 * h + 1] : (unsigned)(y[2 * h + 1] >> 32);
        // halves 1024 + (digit + 128) from the bytes, minus 1152
        const unsigned x = (__byte_perm(w0, w1, by | (4 + by) << 8) & 0x00ff00ffu) | 0x64006400u;
        const __half2 hv = __hsub2(*reinterpret_cast<const __half2*>(&x), __half2half2(__ushort_as_half(0x6480)));
        w[h] = *reinterpret_cast<const unsigned*>(&hv);
      }
      *reinterpret_cast<uint4*>(q + d * R * kOzK) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}
__device__ __forceinline__ void ldsm4(unsigned (&r)[4], const __half* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((unsigned)__cvta_generic_to_shared(p))
               : "memory");
}
__device__ __forceinline__ void mma16816(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// the same on magnitudes, FP16 sums (infinite beyond its range)
__device__ __forceinline__ void mma16816_abs(unsigned (&c)[2], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  constexpr unsigned m = 0x7fff7fffu;
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f16.f16.f16.f16 {%0, %1}, {%2, %3, %4, %5}, {%6, %7}, {%0, %1};"
      : "+r"(c[0]), "+r"(c[1])
      : "r"(a[0] & m), "r"(a[1] & m), "r"(a[2] & m), "r"(a[3] & m), "r"(b0 & m), "r"(b1 & m));
}

// The tile's eight elements of a thread as FP64 sums, k ascending; `sm` holds a
// slab of both operands.
__device__ __forceinline__ void oz_plain(const OzOp& A, const OzOp& B, double* sm, int lr, int lc, double (&run)[8]) {
  double(*sa)[kOzM + 1] = reinterpret_cast<double(*)[kOzM + 1]>(sm);
  double(*sb)[kOzN + 1] = reinterpret_cast<double(*)[kOzN + 1]>(sm + kOzK * (kOzM + 1));
  static_assert(kOzThreads == 4 * kOzM, "a unit of A per thread");
  const int t = threadIdx.x;
#pragma unroll
  for (int x = 0; x < 8; x++) run[x] = 0.0;
  for (int k0 = 0; k0 < A.K; k0 += kOzK) {
    double v[8];
    int r, k;
    __syncthreads();
    oz_load<kOzM>(A, k0, t, v);
    oz_place<kOzM>(A, t, r, k);
#pragma unroll
    for (int h = 0; h < 8; h++) sa[k + h][r] = v[h];
    if (t < 4 * kOzN) {
      oz_load<kOzN>(B, k0, t, v);
      oz_place<kOzN>(B, t, r, k);
#pragma unroll
      for (int h = 0; h < 8; h++) sb[k + h][r] = v[h];
    }
    __syncthreads();
    for (k = 0; k < min(kOzK, A.K - k0); k++)
#pragma unroll
      for (int x = 0; x < 8; x++)
        run[x] = fma(sa[k][lr + 8 * ((x >> 1) & 1)], sb[k][lc + 8 * (x >> 2) + (x & 1)], run[x]);
  }
}

__global__ void __launch_bounds__(kOzThreads, 2) ozgemm_kernel(BGemm<double> g0, BGemm<double> g1, int batch) {
  extern __shared__ __align__(16) __half ozm[];  // [stage][A digits, B digits]
  __shared__ int s_ea[kOzM], s_eb[kOzN];         // exponent bound of each row of A / column of B
  __shared__ double s_rs[kOzN];                  // 1 / s of each column
  __shared__ int s_bad, s_weak;
  const bool first = (int)blockIdx.z < batch;
  const BGemm<double>& g = first ? g0 : g1;
  const int b = first ? blockIdx.z : blockIdx.z - batch;
  const int r0 = blockIdx.x * kOzM, c0 = blockIdx.y * kOzN;
  if (r0 >= g.M || c0 >= g.N) return;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const OzOp A{g.A.p + b * g.A.b + r0 * g.A.r, g.A.r, g.A.c, min(kOzM, g.M - r0), g.K, g.A.c == 1};
  const OzOp B{g.B.p + b * g.B.b + c0 * g.B.c, g.B.c, g.B.r, min(kOzN, g.N - c0), g.K, g.B.r == 1};
  // ---- exponent of the largest entry of each row / column
  if (t < kOzM) s_ea[t] = 1;
  if (t < kOzN) s_eb[t] = 1;
  if (t == 0) s_bad = s_weak = 0;
  __syncthreads();
  const bool bada = oz_max<kOzM>(A, s_ea), badb = oz_max<kOzN>(B, s_eb);
  if (bada || badb) s_bad = 1;
  if (g.X.p && t < B.rows) s_rs[t] = adj_quot(1.0, g.s[b * g.sb + c0 + t]);
  __syncthreads();
  bool plain = s_bad != 0;
  if (t < kOzM) s_ea[t] -= 1022;  // |v| < 2^(exponent - 1022)
  if (t < kOzN) s_eb[t] -= 1022;
  __syncthreads();
  const int wm = (wid & 3) * 16, wn = (wid >> 2) * 16;  // the warp's part of the tile
  // value x of the lane: row (lane >> 2) + 8 ((x >> 1) & 1), column 8 (x >> 2) + 2 (lane & 3) + (x & 1)
  const int lr = wm + (lane >> 2), lc = wn + 2 * (lane & 3);
  double run[8];
#pragma unroll
  for (int x = 0; x < 8; x++) run[x] = 0.0;
  unsigned weak = 0;  // elements left to FP64 sums
  if (!plain) {
    auto stage = [&](int s, int op) { return ozm + (size_t)s * kOzStage + op * kOzD * kOzM * kOzK; };
    oz_stage<kOzM>(A, s_ea, 0, stage(0, 0));
    oz_stage<kOzN>(B, s_eb, 0, stage(0, 1));
    float acc[kOzS][2][4];
    unsigned mag[2][2] = {{0u, 0u}, {0u, 0u}};  // sums of the first digits' |a| |b|
#pragma unroll
    for (int s = 0; s < kOzS; s++)
#pragma unroll
      for (int x = 0; x < 8; x++) acc[s][x >> 2][x & 3] = 0.f;
    int buf = 0;
    for (int k0 = 0; k0 < g.K; k0 += kOzK, buf ^= 1) {
      const bool more = k0 + kOzK < g.K;
      __syncthreads();  // stage `buf` written; the other one's readers are done
#pragma unroll
      for (int kk = 0; kk < kOzK; kk += 16) {
        const __half* sa = stage(buf, 0) + oz_at(wm + (lane & 15), kk + 8 * (lane >> 4));
        const __half* sb = stage(buf, 1) + oz_at(wn + (lane & 7) + 8 * (lane >> 4), kk + 8 * ((lane >> 3) & 1));
        unsigned bf[kOzD][4];
#pragma unroll
        for (int j = 0; j < kOzD; j++) ldsm4(bf[j], sb + j * kOzN * kOzK);
#pragma unroll
        for (int i = 0; i < kOzD; i++) {
          unsigned af[4];
          ldsm4(af, sa + i * kOzM * kOzK);
          if (i == 0) {
            mma16816_abs(mag[0], af, bf[0][0], bf[0][1]);
            mma16816_abs(mag[1], af, bf[0][2], bf[0][3]);
          }
#pragma unroll
          for (int j = 0; j < kOzD; j++) {
            if (i + j >= kOzS) continue;
            mma16816(acc[i + j][0], af, bf[j][0], bf[j][1]);
            mma16816(acc[i + j][1], af, bf[j][2], bf[j][3]);
          }
        }
      }
      if (more) {
        oz_stage<kOzM>(A, s_ea, k0 + kOzK, stage(buf ^ 1, 0));
        oz_stage<kOzN>(B, s_eb, k0 + kOzK, stage(buf ^ 1, 1));
      }
      if (!more || (k0 + kOzK) % kOzChunk == 0) {
        // the exact sums of this chunk, weights 2^112 .. 2^88 and 2^80 .. 2^56; each
        // half is below 2^49, so an integer added to the bits of 1.5 2^52 is its double
#pragma unroll
        for (int x = 0; x < 8; x++) {
          double w[2];
#pragma unroll
          for (int h = 0; h < 2; h++) {
            long long q = 0;
#pragma unroll
            for (int s = 4 * h; s < 4 * h + 4; s++) {
              float& f = acc[s][x >> 2][x & 3];
              q = q * 256 + __float2int_rn(f);
              f = 0.f;
            }
            w[h] = __longlong_as_double(0x4338000000000000ll + q) - 6755399441055744.0;
          }
          const double v = fma(w[0], 4294967296.0, w[1]);
          run[x] = k0 < kOzChunk ? v : run[x] + v;
        }
      }
    }
    // 2^-11 sqrt(K) of the largest product, 64 x 64 of the first digits (a row or
    // column of zeros or subnormals is exact)
    const float least = 2.f * sqrtf((float)g.K);
#pragma unroll
    for (int x = 0; x < 8; x++) {
      const int r = lr + 8 * ((x >> 1) & 1), c = lc + 8 * (x >> 2) + (x & 1);
      const unsigned h = mag[x >> 2][(x >> 1) & 1] >> (16 * (x & 1));
      const bool strong = __half2float(__ushort_as_half((unsigned short)h)) >= least || s_ea[r] == 1 - 1022 ||
                          s_eb[c] == 1 - 1022 || r >= A.rows || c >= B.rows;
      weak |= strong ? 0u : 1u << x;
    }
    if (weak) atomicAdd(&s_weak, __popc(weak));
    __syncthreads();
    plain = s_weak > kOzFew;
  }
  if (plain) {
    oz_plain(A, B, reinterpret_cast<double*>(ozm), lr, lc, run);
  } else if (s_weak) {
#pragma unroll
    for (int x = 0; x < 8; x++)
      for (unsigned w = __ballot_sync(0xffffffffu, (weak >> x) & 1u); w; w &= w - 1) {
        const int src = __ffs(w) - 1;  // the warp forms lane src's element
        const int r = wm + (src >> 2) + 8 * ((x >> 1) & 1), c = wn + 2 * (src & 3) + 8 * (x >> 2) + (x & 1);
        double v = 0.0;
        for (int k = lane; k < g.K; k += 32) v = fma(A.p[r * A.s_r + k * A.s_k], B.p[c * B.s_r + k * B.s_k], v);
        v = warp_sum(v);
        if (lane == src) run[x] = v;
      }
  }
  double* Cb = g.C + b * g.cb;
#pragma unroll
  for (int x = 0; x < 8; x++) {
    const int r = lr + 8 * ((x >> 1) & 1), c = lc + 8 * (x >> 2) + (x & 1);
    if (r < A.rows && c < B.rows) {
      double v = run[x];
      if (!plain && !((weak >> x) & 1u)) {  // v 2^(e_r + e_c - 68), in the exponent field where both ends are normal
        const int sh = s_ea[r] + s_eb[c] - 68, ex = (__double2hiint(v) >> 20) & 0x7ff;
        if (ex != 0 && ex + sh > 0 && ex + sh < 0x7ff)
          v = __hiloint2double(__double2hiint(v) + (sh << 20), __double2loint(v));
        else
          v = scalbn(v, sh);
      }
      if (g.X.p) {
        const double xv = g.X.p[b * g.X.b + (r0 + r) * g.X.r + (c0 + c) * g.X.c];
        v += adj_quot(xv, g.s[b * g.sb + c0 + c], s_rs[c]);
      }
      Cb[(r0 + r) + (size_t)(c0 + c) * g.ldc] = v;
    }
  }
}

// M (k x k per problem) from J, K, s, gs.  The pair (i, j), (j, i) shares
// F_ij (J_ij - J_ji) and F_ij (K_ij - K_ji), which do not change under exchange.
// Columns a and k - 1 - a of the upper triangle hold k + 1 entries together, so
// the pairs fill a rectangle and no lane idles through an FP64 instruction.
constexpr int kCoreCols = 512;

template <typename T>
__global__ void __launch_bounds__(256) adjoint_core_kernel(int k, const T* __restrict__ J, const T* __restrict__ Kv,
                                                           const T* __restrict__ s, const T* __restrict__ gs, T* Mo) {
  const int b = blockIdx.y;
  const T* Jb = J ? J + (size_t)b * k * k : nullptr;
  const T* Kb = Kv ? Kv + (size_t)b * k * k : nullptr;
  const T* sb = s + (size_t)b * k;
  T* Mb = Mo + (size_t)b * k * k;
  // 1 / s of every column once per CTA (columns beyond the table divide)
  __shared__ T s_rs[kCoreCols];
  for (int c = threadIdx.x; c < min(k, kCoreCols); c += blockDim.x) s_rs[c] = adj_quot(T(1), sb[c]);
  __syncthreads();
  auto over = [&](T x, int c) {  // x / s_c
    return c < kCoreCols ? adj_quot(x, sb[c], s_rs[c]) : adj_quot(x, sb[c]);
  };
  const int half = (k + 1) / 2;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < half * (k + 1); idx += gridDim.x * blockDim.x) {
    const int a = idx / (k + 1), c = idx % (k + 1);
    const int i = c <= a ? c : c - a - 1, j = c <= a ? a : k - 1 - a;
    if (c > a && 2 * a + 1 == k) continue;  // odd k: the middle column once
    const T si = sb[i], sj = sb[j];
    const int ij = i + j * k, ji = j + i * k;
    if (i == j) {
      T v = gs ? gs[(size_t)b * k + i] : T(0);
      if (Jb) v -= over(Jb[ij], j);
      Mb[ij] = v;
      continue;
    }
    const T f = adj_quot(T(1), (sj - si) * (sj + si));
    T vij = T(0), vji = T(0);
    if (Jb) {
      const T x = Jb[ij], y = Jb[ji], fj = f * (x - y);
      vij += fj * sj - over(x, j);
      vji += fj * si - over(y, i);
    }
    if (Kb) {
      const T fk = f * (Kb[ij] - Kb[ji]);
      vij += si * fk;
      vji += sj * fk;
    }
    Mb[ij] = vij;
    Mb[ji] = vji;
  }
}

static int bgemm(ddcsvd_context* ctx, int batch, const BGemm<float>& g0, const BGemm<float>* g1) {
  const int M = std::max(g0.M, g1 ? g1->M : 0), N = std::max(g0.N, g1 ? g1->N : 0);
  dim3 grid(ceil_div(M, kBgTile), ceil_div(N, kBgTile), batch * (g1 ? 2 : 1));
  bgemm_kernel<float><<<grid, 256, 0, ctx->stream>>>(g0, g1 ? *g1 : g0, batch);
  count_launch();
  DDC_CUDA_TRY(cudaGetLastError());
  return DDCSVD_OK;
}
static int bgemm(ddcsvd_context* ctx, int batch, const BGemm<double>& g0, const BGemm<double>* g1) {
  const int M = std::max(g0.M, g1 ? g1->M : 0), N = std::max(g0.N, g1 ? g1->N : 0);
  dim3 grid(ceil_div(M, kOzM), ceil_div(N, kOzN), batch * (g1 ? 2 : 1));
  DDC_CUDA_TRY(cudaFuncSetAttribute((const void*)ozgemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kOzSmem));
  ozgemm_kernel<<<grid, kOzThreads, kOzSmem, ctx->stream>>>(g0, g1 ? *g1 : g0, batch);
  count_launch();
  DDC_CUDA_TRY(cudaGetLastError());
  return DDCSVD_OK;
}

// ---------------------------------------------------------------- FP32, one CTA per problem
// Small FP32 problems are bound by the launches and by each product's load
// latency per slab, not by arithmetic (300 x (97 x 41): three products of ~21 us
// for 5 us worth of FMAs), so a CTA keeps its whole problem in shared memory and
// forms J, K, M, P and gA there: one round trip to memory in and one out, 71 -> 41
// us of kernels with cold caches (bound by shared-memory reads), the call 111 ->
// 78 us.  Rows of every matrix are an odd number of floats apart, so
// walks along rows and along columns both spread over the banks.
constexpr int kFusedThreadsMax = 512;
static size_t fused_floats(int m, int n) {
  const size_t ld = (size_t)(n | 1);
  return 2 * m * ld + 4 * n * ld + n;
}

// 512 threads where the m x n products have a tile for each: shared memory holds one
// or two such problems per SM, and 8 warps each leave its latency open (call on 400 x
// (128 x 64) 172 -> 135 us, 1500 x (200 x 60) 748 -> 580, 20 x (150 x 80) 122 -> 100).
// Smaller problems fill the SM with CTAs of 256 (1500 x (64 x 32) 101 us, 122 with 512).
static int fused_threads(int m, int n) { return ceil_div(m, 4) * ceil_div(n, 4) >= 512 ? 512 : 256; }

// out(i, j) for i < MI, j < NJ in 4 x 4 register tiles: sum over q < K of a(i, q) b(q, j)
template <typename FA, typename FB, typename FO>
__device__ __forceinline__ void fused_product(int MI, int NJ, int K, int t0, int nt, FA a, FB b, FO out) {
  const int TI = (MI + 3) >> 2, TJ = (NJ + 3) >> 2;
  for (int t = t0; t < TI * TJ; t += nt) {
    const int ti = t % TI, tj = t / TI;
    int ri[4], cj[4];
#pragma unroll
    for (int x = 0; x < 4; x++) {
      ri[x] = min(ti + TI * x, MI - 1);
      cj[x] = min(tj + TJ * x, NJ - 1);
    }
    float acc[4][4];
#pragma unroll
    for (int x = 0; x < 16; x++) acc[x >> 2][x & 3] = 0.f;
#pragma unroll 4
    for (int q = 0; q < K; q++) {
      float u[4], v[4];
#pragma unroll
      for (int x = 0; x < 4; x++) {
        u[x] = a(ri[x], q);
        v[x] = b(q, cj[x]);
      }
#pragma unroll
      for (int x = 0; x < 16; x++) acc[x >> 2][x & 3] += u[x >> 2] * v[x & 3];
    }
#pragma unroll
    for (int x = 0; x < 16; x++) {
      const int i = ti + TI * (x >> 2), j = tj + TJ * (x & 3);
      if (i < MI && j < NJ) out(i, j, acc[x >> 2][x & 3]);
    }
  }
}

__global__ void __launch_bounds__(kFusedThreadsMax) adjoint_fused_kernel(int m, int n, BMat<float> U, const float* S,
                                                                      BMat<float> V, BMat<float> gU, const float* gS,
                                                                      BMat<float> gV, float* gA) {
  extern __shared__ __align__(16) float fsm[];
  const int t = threadIdx.x, nt = blockDim.x, ld = n | 1;
  const long long b = blockIdx.x;
  float* sU = fsm;
  float* sP = sU + m * ld;  // gU, then P
  float* sV = sP + m * ld;
  float* sW = sV + n * ld;  // gV
  float* sJ = sW + n * ld;  // J, then M
  float* sK = sJ + n * ld;
  float* ss = sK + n * ld;
  auto load = [&](float* dst, const BMat<float>& x, int rows) {
    if (!x.p) return;
    const float* p = x.p + b * x.b;
    const bool rfast = x.r == 1 && x.c != 1;
    for (int idx = t; idx < rows * n; idx += nt) {
      const int r = rfast ? idx % rows : idx / n, c = rfast ? idx / rows : idx % n;
      dst[r * ld + c] = p[r * x.r + c * x.c];
    }
  };
  load(sU, U, m);
  load(sP, gU, m);
  load(sV, V, n);
  load(sW, gV, n);
  for (int c = t; c < n; c += nt) ss[c] = S[b * n + c];
  __syncthreads();
  // J = U^T gU on one half of the threads, K = V^T gV on the other
  const int h = nt / 64 * 32;
  if (t < h) {
    if (gU.p)
      fused_product(n, n, m, t, h, [&](int i, int q) { return sU[q * ld + i]; },
                    [&](int q, int j) { return sP[q * ld + j]; }, [&](int i, int j, float v) { sJ[i * ld + j] = v; });
  } else if (gV.p) {
    fused_product(n, n, n, t - h, nt - h, [&](int i, int q) { return sV[q * ld + i]; },
                  [&](int q, int j) { return sW[q * ld + j]; }, [&](int i, int j, float v) { sK[i * ld + j] = v; });
  }
  __syncthreads();
  for (int idx = t; idx < n * n; idx += nt) {  // M in place of J, a pair at a time
    const int i = idx / n, j = idx % n;
    if (i > j) continue;
    const float si = ss[i], sj = ss[j];
    if (i == j) {
      float v = gS ? gS[b * n + i] : 0.f;
      if (gU.p) v -= sJ[i * ld + i] / sj;
      sJ[i * ld + i] = v;
      continue;
    }
    const float f = 1.f / ((sj - si) * (sj + si));
    float vij = 0.f, vji = 0.f;
    if (gU.p) {
      const float x = sJ[i * ld + j], y = sJ[j * ld + i], fj = f * (x - y);
      vij += fj * sj - x / sj;
      vji += fj * si - y / si;
    }
    if (gV.p) {
      const float fk = f * (sK[i * ld + j] - sK[j * ld + i]);
      vij += si * fk;
      vji += sj * fk;
    }
    sJ[i * ld + j] = vij;
    sJ[j * ld + i] = vji;
  }
  __syncthreads();
  fused_product(m, n, n, t, nt, [&](int i, int q) { return sU[i * ld + q]; },
                [&](int q, int j) { return sJ[q * ld + j]; },
                [&](int i, int j, float v) { sP[i * ld + j] = gU.p ? v + sP[i * ld + j] / ss[j] : v; });
  __syncthreads();
  float* out = gA + b * m * n;
  fused_product(m, n, n, t, nt, [&](int i, int q) { return sP[i * ld + q]; },
                [&](int q, int j) { return sV[j * ld + q]; },
                [&](int i, int j, float v) { out[i + (size_t)j * m] = v; });
}

// The launches of one adjoint on intermediates J, Kv, Mm (k x k per problem)
// and P (m x k per problem).  Launch grids carry the batch in gridDim.z /
// gridDim.y (at most 65535, two products in one launch), so larger batches go
// in chunks.  Inputs by strides (column-major for the C entry points).
constexpr int kBatchChunk = 32767;

template <typename T>
static int adjoint_enqueue(ddcsvd_context* h, int batch, int m, int n, BMat<T> U, const T* S, BMat<T> V, BMat<T> gU,
                           const T* gS, BMat<T> gV, T* gA, T* J, T* Kv, T* Mm, T* P) {
  const int k = n;
  const long long sP = (long long)m * k, sK = (long long)k * k, sA = (long long)m * n;
  auto tr = [](BMat<T> x) { return BMat<T>{x.p, x.c, x.r, x.b}; };
  const BMat<T> none{nullptr, 0, 0, 0};
  for (int b0 = 0; b0 < batch; b0 += kBatchChunk) {
    const int nb = std::min(kBatchChunk, batch - b0);
    auto at = [&](BMat<T> x) { return BMat<T>{x.p ? x.p + b0 * x.b : nullptr, x.r, x.c, x.b}; };
    const BMat<T> Ub = at(U), Vb = at(V), gUb = at(gU), gVb = at(gV);
    const T* Sb = S + b0 * (long long)k;
    T* Jb = J + b0 * sK;
    T* Kb = Kv + b0 * sK;
    T* Mb = Mm + b0 * sK;
    T* Pb = P + b0 * sP;
    // J = U^T gU, K = V^T gV
    const BGemm<T> gj{k, k, m, tr(Ub), gUb, none, nullptr, 0, Jb, k, sK};
    const BGemm<T> gk{k, k, n, tr(Vb), gVb, none, nullptr, 0, Kb, k, sK};
    if (gUb.p && gVb.p) DDC_TRY(bgemm(h, nb, gj, &gk));
    else if (gUb.p) DDC_TRY(bgemm(h, nb, gj, nullptr));
    else if (gVb.p) DDC_TRY(bgemm(h, nb, gk, nullptr));
    dim3 g2(std::max(1, std::min(64, ceil_div((k + 1) / 2 * (k + 1), 256))), nb);
    adjoint_core_kernel<T><<<g2, 256, 0, h->stream>>>(k, gUb.p ? Jb : nullptr, gVb.p ? Kb : nullptr, Sb,
                                                      gS ? gS + b0 * (long long)k : nullptr, Mb);
    count_launch();
    DDC_CUDA_TRY(cudaGetLastError());
    // P = U M + gU S^-1
    const BGemm<T> gp{m, k, k, Ub, BMat<T>{Mb, 1, k, sK}, gUb, Sb, k, Pb, m, sP};
    DDC_TRY(bgemm(h, nb, gp, nullptr));
    // gA = P V^T
    const BGemm<T> ga{m, n, k, BMat<T>{Pb, 1, m, sP}, tr(Vb), none, nullptr, 0, gA + b0 * sA, m, sA};
    DDC_TRY(bgemm(h, nb, ga, nullptr));
  }
  return DDCSVD_OK;
}

template <typename T>
static int svd_backward(ddcsvd_context* h, int batch, int m, int n, BMat<T> U, const T* S, BMat<T> V, BMat<T> gU,
                        const T* gS, BMat<T> gV, T* gA) {
  if (!h || batch <= 0 || m <= 0 || n <= 0 || m < n || !U.p || !S || !V.p || !gA) return DDCSVD_ERR_ARG;
  std::lock_guard<std::mutex> g(h->mu);
  DDC_CUDA_TRY(cudaSetDevice(h->device));
  const int k = n;
  const size_t kk = (size_t)k * k * batch, mk = (size_t)m * k * batch;
  Arena plan;
  plan.take<T>(kk);
  plan.take<T>(kk);
  plan.take<T>(kk);
  plan.take<T>(mk);
  DDC_TRY(ensure_workspace(h, plan.off + 4096));
  Arena a;
  a.plan = false;
  a.base = (char*)h->ws;
  T* J = a.take<T>(kk);
  T* Kv = a.take<T>(kk);
  T* Mm = a.take<T>(kk);
  T* P = a.take<T>(mk);
  DDC_TRY(reset_status(h));
  DDC_TRY(adjoint_enqueue<T>(h, batch, m, n, U, S, V, gU, gS, gV, gA, J, Kv, Mm, P));
  return check_status(h, "svd_backward");
}
// FP32 problems whose six matrices fit one CTA's shared memory: one launch
static int svd_backward_f32(ddcsvd_context* h, int batch, int m, int n, BMat<float> U, const float* S, BMat<float> V,
                            BMat<float> gU, const float* gS, BMat<float> gV, float* gA) {
  if (!h || batch <= 0 || m <= 0 || n <= 0 || m < n || !U.p || !S || !V.p || !gA) return DDCSVD_ERR_ARG;
  const size_t bytes = fused_floats(m, n) * sizeof(float);
  if (bytes > h->smem_optin - 1024) return svd_backward<float>(h, batch, m, n, U, S, V, gU, gS, gV, gA);
  std::lock_guard<std::mutex> g(h->mu);
  DDC_CUDA_TRY(cudaSetDevice(h->device));
  DDC_TRY(reset_status(h));
  DDC_TRY(allow_smem(h, (const void*)adjoint_fused_kernel));
  adjoint_fused_kernel<<<batch, fused_threads(m, n), bytes, h->stream>>>(m, n, U, S, V, gU, gS, gV, gA);
  count_launch();
  DDC_CUDA_TRY(cudaGetLastError());
  return check_status(h, "svd_backward");
}
// column-major matrices of `rows` rows, one after another
template <typename T>
static BMat<T> colmajor(const T* p, int rows, int cols) {
  return BMat<T>{p, 1, rows, (long long)rows * cols};
}

// ---------------------------------------------------------------- allocation-free variant
// Some callers cannot allocate device memory at the moment they need the
// adjoint: code running inside another framework's memory pool or a
// pre-planned fixed memory budget, a real-time loop that must not reach the
// driver's allocator (cudaMalloc can synchronise the device and fail under
// fragmentation), or a context in which only caller-owned buffers may be
// touched.  For them the FP64 adjoint has a variant whose intermediates live
// in a fixed-size array compiled into this library instead of the handle's
// workspace; it needs no handle either.
constexpr size_t kNoAllocScratchBytes = (size_t)16 << 20;  // 16 MiB, held by every GPU that loads the library
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// The array's host-side name is only a stand-in: its device address is
// looked up (cudaGetSymbolAddress, with the caller's context current) the
// first time a context calls, and kept per context id.
using CtxGetCurrentFn = PFN_cuCtxGetCurrent_v4000;
using CtxGetIdFn = PFN_cuCtxGetId_v12000;
static CtxValueCache<64> g_noalloc_addr;

static int driver_fn(const char* name, void** fn) {
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPointByVersion(name, fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess || !*fn) {
    cudaGetLastError();
    set_last_error("driver entry point %s unavailable", name);
    return DDCSVD_ERR_CUDA;
  }
  return DDCSVD_OK;
}

static int lookup_scratch(void** p) {
  const cudaError_t e = cudaGetSymbolAddress(p, g_noalloc_scratch);
  if (e != cudaSuccess || !*p) {
    cudaGetLastError();
    set_last_error("cudaGetSymbolAddress of the adjoint scratch failed: %s", cudaGetErrorString(e));
    return DDCSVD_ERR_CUDA;
  }
  return DDCSVD_OK;
}

static int noalloc_scratch_address(char** out) {
  static CtxGetCurrentFn get_current = nullptr;
  static CtxGetIdFn get_id = nullptr;
  if (!get_current) DDC_TRY(driver_fn("cuCtxGetCurrent", reinterpret_cast<void**>(&get_current)));
  if (!get_id) DDC_TRY(driver_fn("cuCtxGetId", reinterpret_cast<void**>(&get_id)));
  CUcontext c = nullptr;
  if (get_current(&c) != CUDA_SUCCESS) {
    set_last_error("cuCtxGetCurrent failed");
    return DDCSVD_ERR_CUDA;
  }
  if (!c) {
    // no context current on this thread yet: the runtime's lookup makes the
    // current device's primary context current
    void* p = nullptr;
    DDC_TRY(lookup_scratch(&p));
    if (get_current(&c) != CUDA_SUCCESS || !c) {
      set_last_error("no CUDA context is current");
      return DDCSVD_ERR_CUDA;
    }
  }
  unsigned long long id = 0;
  if (get_id(c, &id) != CUDA_SUCCESS) {
    set_last_error("cuCtxGetId failed");
    return DDCSVD_ERR_CUDA;
  }
  void* p = nullptr;
  DDC_TRY(g_noalloc_addr.get(id, &p, lookup_scratch));
  *out = static_cast<char*>(p);
  return DDCSVD_OK;
}

// Bytes of scratch one call takes: J, K and M (k x k per problem) and
// P (m x k per problem), each region rounded up to 256 bytes.
static size_t noalloc_bytes(int batch, int m, int n) {
  const size_t kk = 8 * (size_t)n * n * batch, mk = 8 * (size_t)m * n * batch;
  return 3 * (size_t)round_up((long long)kk, 256) + (size_t)round_up((long long)mk, 256);
}

static int svd_backward_f64_noalloc(cudaStream_t stream, int batch, int m, int n, const double* U, const double* S,
                                    const double* V, const double* gU, const double* gS, const double* gV,
                                    double* gA) {
  if (batch <= 0 || m <= 0 || n <= 0 || m < n || !U || !S || !V || !gA) return DDCSVD_ERR_ARG;
  const size_t need = noalloc_bytes(batch, m, n);
  if (need > kNoAllocScratchBytes) {
    set_last_error("allocation-free adjoint needs %zu bytes of scratch; its fixed limit is %zu bytes "
                   "(3 r(8 batch n^2) + r(8 batch m n), r = round up to 256): split the batch",
                   need, kNoAllocScratchBytes);
    return DDCSVD_ERR_ARG;
  }
  char* base = nullptr;
  DDC_TRY(noalloc_scratch_address(&base));
  int dev = 0;
  DDC_CUDA_TRY(cudaGetDevice(&dev));
  const int k = n;
  const size_t kk = (size_t)k * k * batch, mk = (size_t)m * k * batch;
  Arena a;
  a.plan = false;
  a.base = base;
  double* J = a.take<double>(kk);
  double* Kv = a.take<double>(kk);
  double* Mm = a.take<double>(kk);
  double* P = a.take<double>(mk);
  ddcsvd_context ctx;  // stream only: nothing here allocates
  ctx.device = dev;
  ctx.stream = stream;
  // The array keeps the previous call's contents; J, K, M and P are fully
  // overwritten before they are read, so nothing needs clearing.  The call
  // only enqueues: kernels of the same stream run in order, and a caller
  // reads gA after synchronising the stream.
  DDC_TRY(adjoint_enqueue<double>(&ctx, batch, m, n, colmajor(U, m, n), S, colmajor(V, n, n), colmajor(gU, m, n), gS,
                                  colmajor(gV, n, n), gA, J, Kv, Mm, P));
  return DDCSVD_OK;
}
}  // namespace ddcsvd

using namespace ddcsvd;

extern "C" int ddcsvd_svd_backward_f64_noalloc(void* stream, int batch, int m, int n, const double* dU,
                                               const double* dS, const double* dV, const double* gU,
                                               const double* gS, const double* gV, double* gA) {
  return svd_backward_f64_noalloc(static_cast<cudaStream_t>(stream), batch, m, n, dU, dS, dV, gU, gS, gV, gA);
}

extern "C" int ddcsvd_svd_backward_f64_device(ddcsvd_handle_t h, int batch, int m, int n, const double* dU,
                                              const double* dS, const double* dV, const double* gU,
                                              const double* gS, const double* gV, double* gA) {
  return svd_backward<double>(h, batch, m, n, colmajor(dU, m, n), dS, colmajor(dV, n, n), colmajor(gU, m, n), gS,
                              colmajor(gV, n, n), gA);
}

extern "C" int ddcsvd_svd_backward_f32_device(ddcsvd_handle_t h, int batch, int m, int n, const float* dU,
                                              const float* dS, const float* dV, const float* gU, const float* gS,
                                              const float* gV, float* gA) {
  return svd_backward_f32(h, batch, m, n, colmajor(dU, m, n), dS, colmajor(dV, n, n), colmajor(gU, m, n), gS,
                          colmajor(gV, n, n), gA);
}

template <typename T>
static BMat<T> strided(const T* p, const long long* st) {
  return BMat<T>{p, st[0], st[1], st[2]};
}

extern "C" int ddcsvd_svd_backward_f64_strided(ddcsvd_handle_t h, int batch, int m, int n, const double* dU,
                                               const double* dS, const double* dV, const double* gU,
                                               const double* gS, const double* gV, const long long* strides,
                                               double* gA) {
  if (!strides) return DDCSVD_ERR_ARG;
  return svd_backward<double>(h, batch, m, n, strided(dU, strides), dS, strided(dV, strides + 3),
                              strided(gU, strides + 6), gS, strided(gV, strides + 9), gA);
}

extern "C" int ddcsvd_svd_backward_f32_strided(ddcsvd_handle_t h, int batch, int m, int n, const float* dU,
                                               const float* dS, const float* dV, const float* gU, const float* gS,
                                               const float* gV, const long long* strides, float* gA) {
  if (!strides) return DDCSVD_ERR_ARG;
  return svd_backward_f32(h, batch, m, n, strided(dU, strides), dS, strided(dV, strides + 3),
                          strided(gU, strides + 6), gS, strided(gV, strides + 9), gA);
}
