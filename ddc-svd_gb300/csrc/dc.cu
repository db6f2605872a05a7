// dc.cu -- stage 2: double divide-and-conquer singular values (FP64).
//
// Replaces GetSingularValues_Parallel / DivideAndConquer_Parallel
// (Calculations-Parallel.c:706-874).  The recursion tree is the reference's:
// an N x (N+1) upper bidiagonal node splits at K = N/2 into a K x (K+1) and an
// (N-K-1) x (N-K) child (:731-750); leaves have N <= 2 (:722-726).  A merge
// forms z from the children's last/first right-vector rows and the rotation
// (r0, c0, s0) of their null vectors (:769-782), solves the secular equation
// for the new singular values (:48-348) and, unless it is the root,
// recomputes z-hat (Gu-Eisenstat) and the first/last rows of the merged right
// vectors for its parent (:351-588), then normalises them with phi/psi
// (:807-845).
//
// GB300 layout: one cooperative persistent kernel walks the tree bottom-up,
// one depth at a time, with five bounded grid barriers per depth:
//   P1  leaves (thread each) and merge set-up (CTA per node): parallel merge
//       of the children's sorted values, deflation, compaction;
//   P2  secular roots, one warp per root, lanes split the O(N) sums;
//   P3  z-hat, one warp per component, lanes split the O(N) product;
//   P4  merged first/last rows, one warp per root;
//   P5  merge of roots and deflated values into ascending order, row
//       normalisation (CTA per node).
// Nodes of one depth own disjoint slot ranges, so every per-node array is
// indexed by slot and lives in one N-element buffer; outputs ping-pong
// between two buffers by depth parity.
//
// Deliberate differences from the reference (shared with the FP64 oracle):
// roots are iterated to full FP64 accuracy with a two-pole rational model
// (middle way) inside a bisection bracket, differences d_j^2 - sigma_i^2 are
// formed from the nearer pole without cancellation, z-hat uses products
// instead of logs, sign(z-hat_j) = sign(z_j), tiny z_j and equal d_j deflate,
// and every iteration is capped.
#include <algorithm>
#include <vector>

#include <cooperative_groups.h>

#include "fp64.cuh"
#include "internal.hpp"

namespace cg = cooperative_groups;

namespace ddcsvd {

constexpr int kDcThreads = 512;

struct DcParams {
  int N, nnodes, maxdepth, P;
  int terms;  // terms per lane that the depths' lane groups were sized for
  int maxit;  // FP64 iterations per secular root (the handle's limit, 80 by default)
  const int* nd_r0;
  const int* nd_nn;
  const int* nd_slot;
  const int* nd_K;
  const int* nd_c1;
  const int* nd_c2;
  const int* depth_start;  // [maxdepth + 2]
  const int* depth_merge;  // merge-node ids sorted by depth then slot
  const int* dm_start;     // [maxdepth + 2] ranges into depth_merge
  const int* dgroup;       // [maxdepth + 2] lanes per root at each depth (1..32)
  const double* b1;
  const double* b2;
  double* sig[2];
  double* F[2];
  double* L[2];
  double *ds, *zs, *hfs, *hls;
  double *dq, *zq, *fq, *lq;
  float2* dqf;       // dq as a pair of floats (hi + lo), for the FP32 phase of the root solver
  float* zqf;        // FP32 copy of zq
  double *dd, *fd, *ld;  // deflated entries (ascending d)
  double *tau, *dor, *zh, *rS, *rF, *rL;  // root i: sigma^2 = dor^2 + tau, dor its origin pole
  int* defl;
  int* nq;
  double *zz, *phi, *psi;
  GridBarrier* bar;
  DevStatus* st;
};

// Two versions of the stage's arithmetic.  kBits = true keeps every FP64
// rounding of the plain formulas (division operator, hypot, sqrt, a fixed
// order of sums): the twisted vectors' signs follow from a twist index that
// rounding decides among the large components, so one last-bit change of a
// sigma may flip its vectors.  The entry points that hand back what a stored
// bidiagonal or batch gave before run with it.  kBits = false (single SVDs,
// whose FP32 reduction rounds by the launch knobs anyway) spends fewer FP64
// instructions on results of the same accuracy.
template <bool kBits>
__device__ __forceinline__ double quotient(double a, double x) {
  return kBits ? quot_rn(a, x) : quot(a, x);
}

// p = m 2^e with |m| in [1, 2): keeps the mantissa, adds e to ex (zero,
// subnormal and non-finite values stay as they are)
__device__ __forceinline__ double take_exponent(double p, int& ex) {
  const int hi = __double2hiint(p);
  const int e = (hi >> 20) & 0x7ff;
  if (e == 0 || e == 0x7ff) return p;
  ex += e - 1023;
  return __hiloint2double((hi & 0x800fffff) | 0x3ff00000, __double2loint(p));
}

// ---------------------------------------------------------------- leaves
__device__ void dc_leaf(int nn, const double* b1, const double* b2, double* sig, double* fr,
                        double* lr, double* phi, double* psi) {
  if (nn == 1) {
    double s = hypot(b1[0], b2[0]);
    sig[0] = s;
    if (s > 0.0) {
      fr[0] = b1[0] / s; lr[0] = b2[0] / s; *phi = b2[0] / s; *psi = -b1[0] / s;
    } else {
      fr[0] = 1.0; lr[0] = 0.0; *phi = 0.0; *psi = 1.0;
    }
    return;
  }
  const double x1 = b1[0], x2 = b2[0], x3 = b1[1], x4 = b2[1];
  const double a = x1 * x1 + x2 * x2, e = x3 * x3 + x4 * x4, c = x2 * x3;
  const double det = x1 * x1 * x3 * x3 + x1 * x1 * x4 * x4 + x2 * x2 * x4 * x4;
  const double rad = hypot(0.5 * (a - e), c);
  const double lmax = 0.5 * (a + e) + rad;
  const double lmin = (lmax > 0.0) ? det / lmax : 0.0;
  const double lam[2] = {lmin, lmax};
  for (int k = 0; k < 2; k++) {
    sig[k] = sqrt(lam[k]);
    double u1a = c, u2a = lam[k] - a, u1b = lam[k] - e, u2b = c;
    double na = hypot(u1a, u2a), nb = hypot(u1b, u2b), u1, u2;
    if (na >= nb && na > 0.0) { u1 = u1a / na; u2 = u2a / na; }
    else if (nb > 0.0) { u1 = u1b / nb; u2 = u2b / nb; }
    else { u1 = (k == 0) ? 0.0 : 1.0; u2 = (k == 0) ? 1.0 : 0.0; }
    double v1 = x1 * u1, v2 = x2 * u1 + x3 * u2, v3 = x4 * u2;
    double nv = sqrt(v1 * v1 + v2 * v2 + v3 * v3);
    if (nv > 0.0) { fr[k] = v1 / nv; lr[k] = v3 / nv; }
    else { fr[k] = (k == 0) ? 1.0 : 0.0; lr[k] = 0.0; }
  }
  double n1 = x2 * x4, n2 = -x1 * x4, n3 = x1 * x3;
  double nn3 = sqrt(n1 * n1 + n2 * n2 + n3 * n3);
  if (nn3 > 0.0) { *phi = n1 / nn3; *psi = n3 / nn3; }
  else { *phi = 0.0; *psi = 1.0; }
}

// ---------------------------------------------------------------- block helpers
// Exclusive scan of per-thread counts; returns this thread's offset, total in *tot.
__device__ int block_exscan(int v, int* sh, int* tot) {
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5, nw = blockDim.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) sh[wid] = x;
  __syncthreads();
  if (t == 0) {
    int acc = 0;
    for (int w = 0; w < nw; w++) { int s = sh[w]; sh[w] = acc; acc += s; }
    sh[nw] = acc;
  }
  __syncthreads();
  int r = sh[wid] + x - v;
  *tot = sh[nw];
  __syncthreads();
  return r;
}

__device__ __forceinline__ long long warp_max_ll(long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__device__ long long block_max_ll(long long v, double* sh) {
  long long* shl = reinterpret_cast<long long*>(sh);
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5, nw = blockDim.x >> 5;
  v = warp_max_ll(v);
  __syncthreads();
  if (lane == 0) shl[wid] = v;
  __syncthreads();
  long long r = 0;
  for (int w = 0; w < nw; w++) r = max(r, shl[w]);
  __syncthreads();
  return r;
}

// (kOrdered: the warps' parts are added in order)
template <bool kOrdered>
__device__ double block_sumd(double v, double* sh) {
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5, nw = blockDim.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  if (t < 32) {  // one warp: every warp adding them would queue at the FP64 pipe
    double r = 0.0;
    if (kOrdered) {
      if (t == 0)
        for (int w = 0; w < nw; w++) r += sh[w];
    } else {
      r = warp_sum(t < nw ? sh[t] : 0.0);
    }
    __syncwarp();
    if (t == 0) sh[0] = r;
  }
  __syncthreads();
  const double r = sh[0];
  __syncthreads();
  return r;
}

// 1 / sqrt(a + a1^2) and 1 / sqrt(b + b1^2), or 1 where that is not positive,
// in lanes 0 and 1 of one warp (one pass of the FP64 pipe for both)
__device__ __forceinline__ double lane_inv_norm(double a, double a1, double b, double b1, int lane) {
  const double v = (lane == 0) ? a : b, w = (lane == 0) ? a1 : b1;
  const double n2 = v + w * w;
  return (n2 > 0.0) ? rsqrt(n2) : 1.0;
}
// sqrt(a + a1^2) and sqrt(b + b1^2) likewise
__device__ __forceinline__ double lane_norm(double a, double a1, double b, double b1, int lane) {
  const double v = (lane == 0) ? a : b, w = (lane == 0) ? a1 : b1;
  return sqrt(v + w * w);
}

// Both sums over the warp.
__device__ __forceinline__ void warp_sum2(double& a, double& b) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
}

// Cooperation policies for the per-node phases: a whole CTA for large nodes,
// one warp for nodes of at most kWarpNode entries (a batch forest has
// thousands of those per depth; a CTA each would mostly wait at barriers).
constexpr int kWarpNode = 64;
struct CtaGroup {
  int* shi;
  double* shd;
  __device__ int rank() const { return threadIdx.x; }
  __device__ int size() const { return blockDim.x; }
  __device__ void sync() const { __syncthreads(); }
  __device__ long long maxbits(long long v) const { return block_max_ll(v, shd); }
  template <bool kOrdered>
  __device__ double sum(double v) const { return block_sumd<kOrdered>(v, shd); }
  __device__ int exscan(int v, int* tot) const { return block_exscan(v, shi, tot); }
  __device__ int any(int v) const { return __syncthreads_or(v); }
  // lane_inv_norm / lane_norm of the two sums, taken by one warp and shared
  // (every warp computing them would queue at the FP64 pipe); kInv adds the
  // warps' parts in a tree, else in order
  template <bool kInv>
  __device__ void norms(double* a, double a1, double* b, double b1) const {
    const int t = threadIdx.x, lane = t & 31, nw = blockDim.x >> 5;
    warp_sum2(*a, *b);
    __syncthreads();
    if (lane == 0) {
      shd[t >> 5] = *a;
      shd[20 + (t >> 5)] = *b;
    }
    __syncthreads();
    if (t < 32) {
      double v = 0.0;
      if (kInv) {
        if ((lane >> 1) < nw) v = shd[20 * (lane & 1) + (lane >> 1)];
#pragma unroll
        for (int o = 16; o > 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      } else if (lane < 2) {
        for (int w = 0; w < nw; w++) v += shd[20 * lane + w];
      }
      const double r = kInv ? lane_inv_norm(v, a1, v, b1, lane) : lane_norm(v, a1, v, b1, lane);
      __syncwarp();
      if (lane < 2) shd[lane] = r;
    }
    __syncthreads();
    *a = shd[0];
    *b = shd[1];
  }
};
struct WarpGroup {
  __device__ int rank() const { return threadIdx.x & 31; }
  __device__ int size() const { return 32; }
  __device__ void sync() const { __syncwarp(); }
  __device__ long long maxbits(long long v) const { return warp_max_ll(v); }
  template <bool kOrdered>
  __device__ double sum(double v) const { return warp_sum(v); }
  __device__ int exscan(int v, int* tot) const {
    const int lane = threadIdx.x & 31;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    *tot = __shfl_sync(0xffffffffu, x, 31);
    return x - v;
  }
  __device__ int any(int v) const { return __any_sync(0xffffffffu, v); }
  template <bool kInv>
  __device__ void norms(double* a, double a1, double* b, double b1) const {
    const int lane = threadIdx.x & 31;
    warp_sum2(*a, *b);
    const double r = kInv ? lane_inv_norm(*a, a1, *b, b1, lane) : lane_norm(*a, a1, *b, b1, lane);
    *a = __shfl_sync(0xffffffffu, r, 0);
    *b = __shfl_sync(0xffffffffu, r, 1);
  }
};

// number of a[0..n) < v (strict) or <= v, all values non-negative
__device__ __forceinline__ int count_lt(const double* a, int n, double v) {
  const long long vb = bits(v);
  int lo = 0, hi = n;
  while (lo < hi) { int mid = (lo + hi) >> 1; if (bits(a[mid]) < vb) lo = mid + 1; else hi = mid; }
  return lo;
}
__device__ __forceinline__ int count_le(const double* a, int n, double v) {
  const long long vb = bits(v);
  int lo = 0, hi = n;
  while (lo < hi) { int mid = (lo + hi) >> 1; if (bits(a[mid]) <= vb) lo = mid + 1; else hi = mid; }
  return lo;
}

// ---------------------------------------------------------------- P1 merge set-up
template <bool kBits, class Grp>
__device__ void dc_setup_node(const DcParams& p, int node, int par, const Grp& grp) {
  const int t = grp.rank(), nt = grp.size();
  const int nn = p.nd_nn[node], slot = p.nd_slot[node], K = p.nd_K[node], r0 = p.nd_r0[node];
  const int c1 = p.nd_c1[node], c2 = p.nd_c2[node];
  const int n1 = K, n2 = nn - K - 1;
  const int cp = par ^ 1;
  const double* s1 = p.sig[cp] + slot + 1;
  const double* f1 = p.F[cp] + slot + 1;
  const double* l1 = p.L[cp] + slot + 1;
  const double* s2 = p.sig[cp] + slot + K + 1;
  const double* f2 = p.F[cp] + slot + K + 1;
  const double* l2 = p.L[cp] + slot + K + 1;
  const double bk1 = p.b1[r0 + K], bk2 = p.b2[r0 + K];
  double* ds = p.ds + slot;
  double* zs = p.zs + slot;
  double* hfs = p.hfs + slot;
  double* hls = p.hls + slot;
  // parallel merge of [0] ++ child1 ++ child2 by value (ties: entry 0, then child1)
  long long zb = 0;  // max |z|, as bits
  for (int k = t; k < max(n1, n2); k += nt) {  // one of each child at a time: their loads and searches overlap
    const bool h1 = k < n1, h2 = k < n2;
    double va = 0.0, la = 0.0, fa = 0.0, vb = 0.0, fb = 0.0, lb = 0.0;
    if (h1) { va = s1[k]; la = l1[k]; fa = f1[k]; }
    if (h2) { vb = s2[k]; fb = f2[k]; lb = l2[k]; }
    const int pa = 1 + k + (h1 ? count_lt(s2, n2, va) : 0);
    const int pb = 1 + k + (h2 ? count_le(s1, n1, vb) : 0);
    const double za = bk1 * la, zc = bk2 * fb;
    if (h1) { ds[pa] = va; zs[pa] = za; hfs[pa] = fa; hls[pa] = 0.0; }
    if (h2) { ds[pb] = vb; zs[pb] = zc; hfs[pb] = 0.0; hls[pb] = lb; }
    zb = max(zb, max(max_bits(za), max_bits(zc)));
  }
  if (t < 32) {  // one warp: each further one would queue at the FP64 pipe for the same values
    // r = hypot(x, y), (c0, s0) = (x, y) / r  (Calculations-Parallel.c:769-771)
    const double phi1 = p.phi[c1], psi1 = p.psi[c1], phi2 = p.phi[c2], psi2 = p.psi[c2];
    const double rx = bk1 * psi1, ry = bk2 * phi2;
    const double r2 = fma(rx, rx, ry * ry);
    double r, c0, s0;
    if (!kBits && bits(r2) > bits(1e-280) && bits(r2) < bits(1e280)) {
      const double ri = rsqrt(r2);
      r = r2 * ri;
      c0 = rx * ri;
      s0 = ry * ri;
    } else {
      r = hypot(rx, ry);
      c0 = (r > 0.0) ? quot_rn(rx, r) : 1.0;
      s0 = (r > 0.0) ? quot_rn(ry, r) : 0.0;
    }
    zb = max(zb, max_bits(r));
    if (t == 0) {
      ds[0] = 0.0; zs[0] = r; hfs[0] = c0 * phi1; hls[0] = s0 * psi2;
      p.phi[node] = -s0 * phi1;  // Calculations-Parallel.c:807-808 (normalised in P5)
      p.psi[node] = c0 * psi2;
    }
  }
  // the children's values ascend, so the largest d is one of their last
  zb = max(grp.maxbits(zb), max(n1 > 0 ? max_bits(s1[n1 - 1]) : 0ll, n2 > 0 ? max_bits(s2[n2 - 1]) : 0ll));
  const double tol = 8.0 * DBL_EPSILON * __longlong_as_double(zb);
  const long long tolb = bits(tol);
  grp.sync();
  // deflation 1: negligible z
  const int per = ceil_div(nn, nt);
  const int lo = min(nn, t * per), hi = min(nn, lo + per);
  int cnt = 0;
  for (int k = lo; k < hi; k++) {
    int dfl = abs_bits(zs[k]) <= tolb;
    p.defl[slot + k] = dfl;
    cnt += !dfl;
  }
  int tot;
  int off = grp.exscan(cnt, &tot);
  // positions of non-deflated entries -> compacted arrays (tentative)
  for (int k = lo; k < hi; k++)
    if (!p.defl[slot + k]) { p.dq[slot + off] = ds[k]; off++; }
  grp.sync();
  // deflation 2 needed?  (adjacent non-deflated values within tol)
  int close = 0;
  for (int k = 1 + t; k < tot; k += nt)
    if (bits(p.dq[slot + k] - p.dq[slot + k - 1]) <= tolb) close = 1;
  const int need2 = grp.any(close);
  if (need2 && t == 0) {
    int prev = -1;
    for (int k = 0; k < nn; k++) {
      if (p.defl[slot + k]) continue;
      if (prev >= 0 && ds[k] - ds[prev] <= tol) {
        double rr = hypot(zs[prev], zs[k]);
        double c = zs[k] / rr, s = zs[prev] / rr;
        zs[k] = rr; zs[prev] = 0.0; p.defl[slot + prev] = 1;
        double fa = hfs[prev], fb = hfs[k], la = hls[prev], lb = hls[k];
        hfs[prev] = c * fa - s * fb; hfs[k] = s * fa + c * fb;
        hls[prev] = c * la - s * lb; hls[k] = s * la + c * lb;
      }
      prev = k;
    }
  }
  grp.sync();
  // final compaction: non-deflated -> dq/zq/fq/lq, deflated -> dd/fd/ld
  cnt = 0;
  for (int k = lo; k < hi; k++) cnt += !p.defl[slot + k];
  off = grp.exscan(cnt, &tot);
  int doff = lo - off;  // deflated entries before this thread's range
  double zzl = 0.0;
  for (int k = lo; k < hi; k++) {
    if (!p.defl[slot + k]) {
      p.dq[slot + off] = ds[k]; p.zq[slot + off] = zs[k];
      const float dh = (float)ds[k];
      p.dqf[slot + off] = make_float2(dh, (float)(ds[k] - (double)dh));
      p.zqf[slot + off] = (float)zs[k];
      p.fq[slot + off] = hfs[k]; p.lq[slot + off] = hls[k];
      zzl += zs[k] * zs[k];
      off++;
    } else {
      p.dd[slot + doff] = ds[k]; p.fd[slot + doff] = hfs[k]; p.ld[slot + doff] = hls[k];
      doff++;
    }
  }
  const double zz = grp.template sum<kBits>(zzl);
  if (t == 0) {
    p.nq[node] = tot;
    p.zz[node] = zz;
  }
}

// ---------------------------------------------------------------- lane groups
// The per-root phases run one group of G lanes (G = 1, 2, ..., 32, chosen per
// depth from its largest node) per root: small nodes of a batch forest would
// otherwise leave most of a warp idle and pay five shuffle rounds per sum.
// kG fixes the group's size at compile time: a whole warp (32) reduces in five
// rounds with a constant mask, several sums to a round.  With the size and mask
// read at run time and one loop per sum, the four sums of one FP32 evaluation
// took most of its 2900 cycles (48 to 128 poles).  kG = 0: any size up to 16.
//
// kG = -V: any size, each lane with the terms of V lanes of a group V times as
// large, V partial sums apart and then added in the order that group's reduction
// has: the same bits.  V times as many roots share a warp's instructions for what
// is done once per root (75 FP64 instructions a step, against 11 a term), which is
// what a forest of many trees wants; a single tree has lanes to spare.
template <int kG>
struct LaneGroup {
  int G;          // lanes per group
  int lg;         // lane within the group
  unsigned mask;  // lanes of this group within the warp
  static constexpr int kV = kG < 0 ? -kG : 1;
  __device__ __forceinline__ int size() const { return kG > 0 ? kG : G; }
};
template <int kG>
__device__ __forceinline__ LaneGroup<kG> make_group(int G, int lane) {
  LaneGroup<kG> g;
  g.G = kG > 0 ? kG : G;
  g.lg = lane & (g.size() - 1);
  g.mask = (kG == 32) ? 0xffffffffu : (((1u << G) - 1u) << (lane & ~(G - 1)));
  return g;
}
// every v becomes its sum over the group (the same order of additions for each kG)
template <int kG, typename... T>
__device__ __forceinline__ void gsum(const LaneGroup<kG>& g, T&... v) {
  if constexpr (kG == 32) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ((v += __shfl_xor_sync(0xffffffffu, v, o)), ...);
  } else {
    for (int o = g.G >> 1; o > 0; o >>= 1) ((v += __shfl_xor_sync(g.mask, v, o)), ...);
  }
}
// acc: the group's sums of body over the terms 0 .. q - 1
template <int kG, int N, typename T, class F>
__device__ __forceinline__ void group_sums(const LaneGroup<kG>& g, int q, T (&acc)[N], F body) {
  constexpr int V = LaneGroup<kG>::kV;
  static_assert(N == 3 || N == 4, "");
#pragma unroll
  for (int u = 0; u < N; u++) acc[u] = T(0);
  if constexpr (V == 1) {
    for (int j = g.lg; j < q; j += g.size()) body(j, acc);
  } else {
    T part[V][N];
#pragma unroll
    for (int k = 0; k < V; k++)
#pragma unroll
      for (int u = 0; u < N; u++) part[k][u] = T(0);
    for (int j = g.lg; j < q; j += V * g.size())
#pragma unroll
      for (int k = 0; k < V; k++)
        if (k == 0 || j + k * g.size() < q) body(j + k * g.size(), part[k]);
#pragma unroll
    for (int h = V / 2; h > 0; h /= 2)
#pragma unroll
      for (int k = 0; k < h; k++)
#pragma unroll
        for (int u = 0; u < N; u++) part[k][u] += part[k + h][u];
#pragma unroll
    for (int u = 0; u < N; u++) acc[u] = part[0][u];
  }
  if constexpr (N == 4) gsum(g, acc[0], acc[1], acc[2], acc[3]);
  else gsum(g, acc[0], acc[1], acc[2]);
}
// the product of v and the sum of e over the group
template <int kG>
__device__ __forceinline__ void gprod(const LaneGroup<kG>& g, double& v, int& e) {
  if constexpr (kG == 32) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      v *= __shfl_xor_sync(0xffffffffu, v, o);
      e += __shfl_xor_sync(0xffffffffu, e, o);
    }
  } else {
    for (int o = g.G >> 1; o > 0; o >>= 1) {
      v *= __shfl_xor_sync(g.mask, v, o);
      e += __shfl_xor_sync(g.mask, e, o);
    }
  }
}

// ---------------------------------------------------------------- secular roots
template <int kG>
__device__ __forceinline__ void sec_eval(int q, const double* d, const double* z, double dorg,
                                         double tau, int split, const LaneGroup<kG>& g, double& f, double& psi,
                                         double& dpsi, double& phi, double& dphi) {
  double acc[4];
  group_sums(g, q, acc, [&](int j, double (&a)[4]) {
    const double dj = d[j];
    const double del = (dj - dorg) * (dj + dorg) - tau;
    const double tt = quot_rn(z[j], del);
    // (the side's sums by selects: a branch here sent most warps down both sides)
    const bool le = j <= split;
    const double v = (le ? a[0] : a[2]) + z[j] * tt, dv = (le ? a[1] : a[3]) + tt * tt;
    a[0] = le ? v : a[0];
    a[1] = le ? dv : a[1];
    a[2] = le ? a[2] : v;
    a[3] = le ? a[3] : dv;
  });
  psi = acc[0]; dpsi = acc[1]; phi = acc[2]; dphi = acc[3];
  f = 1.0 + psi + phi;
}

// FP32 reciprocal to an ulp or so (range ends flush to 0 or infinity)
__device__ __forceinline__ float rcp32(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// d_j - d_o from the float pairs: the heads' difference is exact when they are
// close, so it keeps FP32's relative accuracy down to gaps of 2^-24 |d| (from
// the heads alone, a gap of |d| / 1000 had only 14 good bits, and the FP64
// phase then needed a second evaluation for most roots)
__device__ __forceinline__ float pair_diff(float2 a, float2 b) { return (a.x - b.x) + (a.y - b.y); }

// FP32 twin of sec_eval on the float copies of d and z (kBits: the heads and
// the division operator only).
template <bool kBits, int kG>
__device__ __forceinline__ void sec_eval32(int q, const float2* d, const float* z, float2 dorg, float tau, int split,
                                           const LaneGroup<kG>& g, float& f, float& psi, float& dpsi, float& phi,
                                           float& dphi) {
  float acc[4];
  group_sums(g, q, acc, [&](int j, float (&a)[4]) {
    const float2 dj = d[j];
    const float zj = z[j];
    const float del = (kBits ? dj.x - dorg.x : pair_diff(dj, dorg)) * (dj.x + dorg.x) - tau;
    const float tt = kBits ? zj / del : zj * rcp32(del);
    if (j <= split) { a[0] += zj * tt; a[1] += tt * tt; }
    else { a[2] += zj * tt; a[3] += tt * tt; }
  });
  psi = acc[0]; dpsi = acc[1]; phi = acc[2]; dphi = acc[3];
  f = 1.f + psi + phi;
}

// One FP64 evaluation for the third-order step: f, f' = sum (z / del)^2, and
// in FP32 the second-derivative sum g2 = sum (z / del)^2 (tau / del), which
// only forms the correction term.  Nine FP64 instructions per pole.
template <int kG>
__device__ __forceinline__ void sec_eval_newton(int q, const double* d, const double* z, double dorg, double tau,
                                                const LaneGroup<kG>& g, double& f, double& fp, float& g2) {
  const float t32 = (float)tau;
  double s = 0.0, sp = 0.0;
  float sg = 0.f;
  for (int j = g.lg; j < q; j += g.size()) {
    const double dj = d[j], zj = z[j];
    const double del = fma(dj - dorg, dj + dorg, -tau);
    const double r = rcp_approx(del);
    const double e = fma(-del, r, 1.0);
    const double y = fma(e, e, e);
    const double t = zj * r;
    const double tt = fma(t, y, t);
    s = fma(zj, tt, s);
    sp = fma(tt, tt, sp);
    const float tf = (float)tt;
    sg += tf * tf * ((float)r * t32);
  }
  gsum(g, s, sp, sg);
  f = 1.0 + s;
  fp = sp;
  g2 = sg;
}

// One safeguarded step of the root iteration (two-pole rational model for an
// interior root, one pole for the last root), shared by the FP32 and FP64
// phases.  Returns true when converged.
// (without kBits the FP32 steps use approximate quotients and roots: the test of
// f decides when to stop, so a step need not be rounded correctly)
__device__ __forceinline__ float sqrt32(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
template <bool kBits>
__device__ __forceinline__ float step_quot(float a, float x) { return kBits ? a / x : a * rcp32(x); }
template <bool kBits>
__device__ __forceinline__ double step_quot(double a, double x) { return quot_rn(a, x); }
template <bool kBits>
__device__ __forceinline__ float step_sqrt(float x) { return kBits ? sqrtf(x) : sqrt32(x); }
template <bool kBits>
__device__ __forceinline__ double step_sqrt(double x) { return sqrt(x); }

// |a| <= b for b >= 0, a < 0 and the larger magnitude; in FP64 by the bits (a
// comparison takes the FP64 pipe as long as a product)
__device__ __forceinline__ bool abs_le(float a, float b) { return fabsf(a) <= b; }
__device__ __forceinline__ bool abs_le(double a, double b) {
  return abs_bits(a) <= bits(b) && bits(b) <= 0x7ff0000000000000ll;  // (false for a NaN)
}
__device__ __forceinline__ bool negative(float a) { return a < 0.f; }
__device__ __forceinline__ bool negative(double a) { return bits(a) < 0 && abs_bits(a) > 0; }
__device__ __forceinline__ float max_abs(float a, float b) { return fmaxf(fabsf(a), fabsf(b)); }
__device__ __forceinline__ double max_abs(double a, double b) {
  return __longlong_as_double(max(abs_bits(a), abs_bits(b)));
}

template <bool kBits, typename T>
__device__ __forceinline__ bool sec_step(bool last, T f, T psi, T dpsi, T phi, T dphi, T da0, T db0, T eps,
                                         T& lo, T& hi, T& tau, bool& halved) {
  const T err = last ? T(8) * (T(1) + fabs(psi)) + fabs(tau) * dpsi
                     : T(8) * (T(1) + fabs(psi) + fabs(phi)) + fabs(tau) * (dpsi + dphi);
  if (abs_le(f, eps * err)) return true;
  if (negative(f)) lo = tau; else hi = tau;
  if (abs_le(hi - lo, T(4) * eps * max_abs(lo, hi))) return true;
  T tn;
  if (last) {
    const T da = -tau;
    const T s1 = da * da * dpsi;
    const T c = f - step_quot<kBits>(s1, da);
    tn = (c != T(0)) ? tau + da + step_quot<kBits>(s1, c) : T(0.5) * (lo + hi);
  } else {
    const T da = da0 - tau, db = db0 - tau;
    const T s1 = da * da * dpsi, s2 = db * db * dphi;
    const T c = f - step_quot<kBits>(s1, da) - step_quot<kBits>(s2, db);
    const T aq = c, bq = c * (da + db) + s1 + s2, cq = da * db * f;
    const T disc = step_sqrt<kBits>(fabs(bq * bq - T(4) * aq * cq));
    // the smaller root of the model's quadratic, one quotient for its three forms
    const bool low = !(bq > T(0));
    T num = low ? bq - disc : T(2) * cq, den = low ? T(2) * aq : bq + disc;
    if (aq == T(0)) {
      num = cq;
      den = bq;
    }
    tn = tau + step_quot<kBits>(num, den);
  }
  halved = !(tn > lo && tn < hi);
  if (halved) tn = T(0.5) * (lo + hi);
  tau = tn;
  return false;
}

#ifdef DDCSVD_PHASE_TRACE
__device__ unsigned g_dc_iters[64 * 84];  // [depth][FP64 iterations 0..80, 81: FP32 phase gave up early]
#endif

// 1 and the poles other than o at tau = 0: c in c - z_o^2 / tau, the equation
// a root much nearer to its pole than any other pole solves
template <int kG>
__device__ __forceinline__ float sec_rest32(int q, const float2* d, const float* z, int o, const LaneGroup<kG>& g) {
  const float2 dorg = d[o];
  float s = 0.f;
  for (int j = g.lg; j < q; j += g.size()) {
    const float2 dj = d[j];
    const float t = z[j] * z[j] * rcp32(pair_diff(dj, dorg) * (dj.x + dorg.x));
    if (j != o) s += t;
  }
  gsum(g, s);
  return 1.f + s;
}

// f at the midpoint of (d_i, d_i+1) on the float pairs, with a bound on its
// error: del_j = (d_j - d_o)(d_j + d_o) - tau carries a relative error of a few
// eps32 on the product and on tau, plus 2^-47 of |d| in each difference (the
// pairs' own rounding; tau comes from such a difference too); term j is off by
// its size times that over |del_j| (plus a few roundings), and the sum by
// q eps32 of the total.  A term whose del_j may change sign, or lies near the
// FP32 subnormal range (where the copies lose relative precision), makes the
// bound infinite.
template <int kG>
__device__ __forceinline__ void sec_mid32(int q, const float2* d, const float* z, float2 dorg, float tau,
                                          const LaneGroup<kG>& g, float& f, float& err) {
  constexpr float e32 = FLT_EPSILON;
  float acc[3];
  group_sums(g, q, acc, [&](int j, float (&a)[3]) {
    const float2 dj = d[j];
    const float ad = fabsf(dj.x) + fabsf(dorg.x);
    const float dif = pair_diff(dj, dorg);
    const float del = dif * (dj.x + dorg.x) - tau;
    const float ir = rcp32(del);
    const float tt = z[j] * z[j] * ir;
    const float ed = 4.f * e32 * (fabsf(dif) * ad + fabsf(tau)) + 0x1p-44f * ad * ad;
    const float at = fabsf(tt), adel = fabsf(del);
    a[0] += tt;
    a[1] += at;
    a[2] += (ed < 0.5f * adel && adel >= 0x1p-100f && adel <= 0x1p100f) ? at * (2.5f * ed * fabsf(ir) + 6.f * e32)
                                                                       : INFINITY;
  });
  const float s = acc[0], sa = acc[1], ea = acc[2];
  f = 1.f + s;
  err = ea + (float)(q + 2) * e32 * (1.f + sa);
}

// Root i of the node's secular equation; returns its origin pole (local index)
// and tau = sigma^2 - d_o^2.
// Phase 1 iterates in FP32 to about single precision.  Phase 2 evaluates f and
// f' once in FP64 at that point and takes the step x = -u (1 + g u), u = f/f',
// g = sum z^2/del^3 / f' (Chebyshev's method, third order): with |u / tau| near
// 1e-6 what is left is below FP64 resolution, so no second evaluation is
// needed to confirm it.  The estimate of the third-order rest decides; a root
// it does not clear (clustered poles, range trouble) goes through the
// safeguarded FP64 iteration from there.  The corrected step counts as two
// iterations against the caller's cap.
// kBits iterates both phases with the two-pole model alone.
template <bool kBits, int kG>
__device__ bool sec_root(int q, const double* d, const double* z, const float2* df, const float* zf, double zz,
                         int i, const LaneGroup<kG>& g, int maxit, int* origin, double* tau_out, int* iters = nullptr) {
  double f, psi, dpsi, phi, dphi;
  const bool last = (i == q - 1);
  const int split = last ? q - 1 : i;
  int o;
  float dd32 = 0.f, f32 = 0.f;
  bool sure = false;
  double dd = 0.0;
  if (!last) {
    // origin = nearer pole, from the sign of f at the midpoint: from the float
    // copies when f clears twice its error bound, else in FP64 (an FP32 sign
    // taken without the bound picked the wrong half on close poles of a
    // batch forest, and the root then lies outside the bracket)
    const float2 a = df[i], b = df[i + 1];
    dd32 = pair_diff(b, a) * (b.x + a.x);
    float e32;
    sec_mid32(q, df, zf, a, 0.5f * dd32, g, f32, e32);
    sure = fabsf(f32) > 2.f * e32 && fabsf(f32) < INFINITY;
    if (kBits || !sure) dd = (d[i + 1] - d[i]) * (d[i + 1] + d[i]);
    if (sure) {
      o = (f32 >= 0.f) ? i : i + 1;
    } else {
      sec_eval(q, d, z, d[i], 0.5 * dd, i, g, f, psi, dpsi, phi, dphi);
      o = (f >= 0.0) ? i : i + 1;
    }
  } else {
    o = q - 1;
  }
  *origin = o;
  const double dorg = d[o];
  const float2 od = df[o];
  const bool left = (o == i);  // tau > 0
  // ---- phase 1: FP32
  float lo32, hi32, t32, da32, db32;
  if (kBits) {
    const double hd = last ? 0.5 * zz : 0.5 * dd;
    lo32 = left ? 0.f : (float)-hd;
    hi32 = last ? (float)zz : left ? (float)hd : 0.f;
    t32 = left ? (float)hd : (float)-hd;
    da32 = (last || left) ? 0.f : (float)((d[i] - dorg) * (d[i] + dorg));
    db32 = (last || !left) ? 0.f : (float)((d[i + 1] - dorg) * (d[i + 1] + dorg));
  } else {
    lo32 = left ? 0.f : -0.5f * dd32;
    hi32 = last ? (float)zz : left ? 0.5f * dd32 : 0.f;
    t32 = last ? 0.5f * hi32 : left ? hi32 : lo32;
    da32 = (last || left) ? 0.f : -dd32;
    db32 = (last || !left) ? 0.f : dd32;
    // Start from the root of c + (the two poles next to the interval), c what the
    // other poles and 1 add up to where f is known already (the midpoint; half
    // the bracket for the last root).  A root that a small z leaves at 1e-20 of
    // the gap from its pole starts there; from the midpoint the bracket was
    // halved up to 40 times, and the warps with such a root held up the barrier
    // by three times the common root's time.
    if (last) {
      float e32;
      const int far = max(i - 1, 0);
      const float gap = (q > 1) ? pair_diff(od, df[far]) * (od.x + df[far].x) : 1.f;
      const float wn = zf[i] * zf[i], wf = (q > 1) ? zf[far] * zf[far] : 0.f;
      sec_mid32(q, df, zf, od, t32, g, f32, e32);
      const float c = f32 + wf * rcp32(gap + t32) + wn * rcp32(t32);
      const float b = c * gap - wf - wn, r = sqrt32(b * b + 4.f * c * wn * gap);
      const float t = (b > 0.f) ? 2.f * wn * gap * rcp32(b + r) : (r - b) * rcp32(2.f * c);
      if (c > 0.f && t > lo32 && t < hi32) t32 = t;
    } else if (sure) {
      const float zi = zf[i] * zf[i], zj = zf[i + 1] * zf[i + 1];
      const float wn = left ? zi : zj, wf = left ? zj : zi;
      const float c = f32 + 2.f * (zi - zj) * rcp32(dd32), cs = (left ? c : -c) * dd32;
      const float b = cs + wn + wf, h = cs - wn + wf, r = sqrt32(h * h + 4.f * wn * wf);
      const float t = (b > 0.f) ? 2.f * wn * dd32 * rcp32(b + r) : (b - r) * dd32 * rcp32(2.f * cs);
      const float ts = left ? t : -t;
      if (ts > lo32 && ts < hi32) t32 = ts;
    }
  }
  bool fine = false, tried = false, halved;
  for (int it = 0; it < 40; it++) {
    float f3, ps3, dps3, ph3, dph3;
    sec_eval32<kBits>(q, df, zf, od, t32, split, g, f3, ps3, dps3, ph3, dph3);
    if (!(fabsf(f3) < INFINITY) || !(dps3 < INFINITY) || !(dph3 < INFINITY)) break;
    if (sec_step<kBits, float>(last, f3, ps3, dps3, ph3, dph3, da32, db32, 4.f * FLT_EPSILON, lo32, hi32, t32,
                               halved)) {
      if (!kBits) {
        const float tn = t32 - f3 / (dps3 + dph3);  // the evaluation's own Newton step is free
        if (tn > lo32 && tn < hi32) t32 = tn;
      }
      fine = true;
      break;
    }
    if (!kBits && halved && !tried) {
      // out of the model's reach: mostly a root at z_o^2 / c with a tiny z_o
      tried = true;
      const float c = sec_rest32(q, df, zf, o, g);
      const float t = zf[o] * zf[o] * rcp32(c);  // left: c > 0, right: c < 0
      if (t > lo32 && t < hi32) t32 = t;
    }
  }
  // ---- phase 2: one FP64 evaluation and a third-order step
  if (!kBits && fine && maxit >= 2) {
    double fp;
    float g2;
    const double t0 = (double)t32;
    sec_eval_newton(q, d, z, dorg, t0, g, f, fp, g2);
    const double u = quot(f, fp);
    // (everything relative to tau: in absolute terms the test underflowed or overflowed
    // for inputs far from 1 and let any step through)
    const float fpf = (float)fp, at = fabsf(t32), un = (float)u / t32, gr = g2 / fpf;
    const float rest = fabsf(un) * un * un * (2.f * gr * gr + 1.f);  // size of the third-order term
    const double tau = t0 - fma(u, (double)(gr * un), u);
    const float tf = left ? (float)tau : -(float)tau;
    const float far32 = last ? 1.001f * (float)zz : 0.501f * dd32;
    const bool range = at >= 0x1p-120f && at <= 0x1p100f && fpf >= 0x1p-100f && fpf <= 0x1p120f;
    if (range && fabsf(un) <= 1e-3f && rest <= 0x1p-55f * fabsf(od.x * (od.x / t32) + 1.f) && tf > 0.f && tf <= far32) {
      if (iters) *iters = 1;
      *tau_out = tau;
      return true;
    }
    // a root as near to its pole as FP32 reaches (a few of graded problems): the plain
    // step's rest, at most 1e-6 tau, is nothing beside d^2
    if (at < 0x1p-120f && od.x >= 0x1p-30f && od.x <= 0x1p30f && fabs(u) <= 1e-3 * (double)at) {
      if (iters) *iters = 1;
      *tau_out = t0 - u;
      return true;
    }
  }
  // ---- the safeguarded FP64 iteration.  A step below 1e-10 |tau| is accepted
  // without another evaluation: the rational model converges at least
  // quadratically, so the remaining error is far below FP64 resolution.
  double lo, hi, tau, da0 = 0.0, db0 = 0.0;
  if (!last) {
    if (!kBits) dd = (d[i + 1] - d[i]) * (d[i + 1] + d[i]);
    if (left) { lo = 0.0; hi = 0.5 * dd; tau = 0.5 * dd; }
    else { lo = -0.5 * dd; hi = 0.0; tau = -0.5 * dd; }
    da0 = (d[i] - dorg) * (d[i] + dorg);
    db0 = (d[i + 1] - dorg) * (d[i + 1] + dorg);
  } else {
    lo = 0.0; hi = zz; tau = 0.5 * zz;
  }
  if ((double)t32 > lo && (double)t32 < hi) tau = (double)t32;
  bool conv = false;
  int it = 0;
  for (; it < maxit; it++) {
    sec_eval(q, d, z, dorg, tau, split, g, f, psi, dpsi, phi, dphi);
    const double prev = tau;
    if (sec_step<kBits, double>(last, f, psi, dpsi, phi, dphi, da0, db0, DBL_EPSILON, lo, hi, tau, halved)) {
      conv = true;
      break;
    }
    if (fabs(tau - prev) <= 1e-10 * fabs(tau)) {
      conv = true;
      break;
    }
  }
  if (iters) *iters = it;
  *tau_out = tau;
  return conv;
}

// ---------------------------------------------------------------- P2 - P4, one lane group per root
// root i = pos - slot of the node at `slot` with q poles
template <bool kBits, int kG>
__device__ __forceinline__ void dc_root(const DcParams& p, int node, int slot, int pos, int q, int d,
                                        const LaneGroup<kG>& g) {
  int o, its = 0;
  double tau;
  const bool ok = sec_root<kBits>(q, p.dq + slot, p.zq + slot, p.dqf + slot, p.zqf + slot, p.zz[node], pos - slot, g,
                           p.maxit, &o, &tau, &its);
#ifdef DDCSVD_PHASE_TRACE
  if (g.lg == 0 && d < 64) atomicAdd(&g_dc_iters[d * 84 + min(its, 80)], 1u);
#else
  (void)its;
  (void)d;
#endif
  if (g.lg == 0) {
    const double dorg = p.dq[slot + o];
    p.tau[pos] = tau;
    p.dor[pos] = dorg;
    p.rS[pos] = sqrt(dorg * dorg + tau);
    if (!ok) set_error(p.st, DDCSVD_ERR_NOCONV, pos);
  }
}

// z-hat component j = pos - slot (Gu-Eisenstat): the product of
// (sigma_k^2 - d_j^2) / (d_k^2 - d_j^2).  Without kBits numerators and
// denominators are multiplied apart with their exponents in an integer (eight
// FP64 instructions per term; a division in each makes it 13, and the
// operator's 16).
template <bool kBits, int kG>
__device__ __forceinline__ void dc_zhat(const DcParams& p, int slot, int pos, int q, const LaneGroup<kG>& g) {
  const int j = pos - slot;
  const double* dq = p.dq + slot;
  const double* tau = p.tau + slot;
  const double* dor = p.dor + slot;
  const double dj = dq[j];
  constexpr int V = LaneGroup<kG>::kV;
  double prod, pn[V], pd = 1.0;
  int en = 0, ed = 0;
#pragma unroll
  for (int v = 0; v < V; v++) pn[v] = 1.0;
  for (int k0 = g.lg; k0 < q - 1; k0 += V * g.size()) {
#pragma unroll
    for (int v = 0; v < V; v++) {
      const int k = k0 + v * g.size();
      if (v > 0 && k >= q - 1) continue;
      const double dk = dor[k], dd = dq[(k < j) ? k : k + 1];
      const double num = tau[k] - (dj - dk) * (dj + dk);
      const double den = (dd - dj) * (dd + dj);
      if (kBits) {
        pn[v] *= quot_rn(num, den);
      } else {
        pn[v] = take_exponent(pn[v] * num, en);
        pd = take_exponent(pd * den, ed);
      }
    }
  }
#pragma unroll
  for (int h = V / 2; h > 0; h /= 2)
#pragma unroll
    for (int v = 0; v < h; v++) pn[v] *= pn[v + h];
  prod = kBits ? pn[0] : quot(pn[0], pd);
  int ex = en - ed;  // (0 with kBits)
  gprod(g, prod, ex);
  if (g.lg == 0) {
    const double dk = dor[q - 1];
    prod *= tau[q - 1] - (dj - dk) * (dj + dk);
    double a;
    if (kBits) {
      a = sqrt(fabs(prod));
    } else {
      prod = take_exponent(prod, ex);
      if (ex & 1) { prod *= 2.0; ex -= 1; }
      a = ldexp(sqrt(fabs(prod)), ex / 2);
    }
    p.zh[pos] = (p.zq[pos] >= 0.0) ? a : -a;
  }
}

// first / last rows of the merged right vector of root i = pos - slot
template <bool kBits, int kG>
__device__ __forceinline__ void dc_rows(const DcParams& p, int slot, int pos, int q, const LaneGroup<kG>& g) {
  const double* dq = p.dq + slot;
  const double* zh = p.zh + slot;
  const double* fq = p.fq + slot;
  const double* lq = p.lq + slot;
  const double dorg = p.dor[pos], ti = p.tau[pos];
  double acc[3];
  group_sums(g, q, acc, [&](int j, double (&a)[3]) {
    const double dj = dq[j];
    const double del = (dj - dorg) * (dj + dorg) - ti;
    const double v = quotient<kBits>(zh[j], del);
    a[0] += v * v;
    a[1] += v * fq[j];
    a[2] += v * lq[j];
  });
  double nv = acc[0];
  const double sf = acc[1], sl = acc[2];
  if (g.lg == 0) {
    if (kBits) {
      nv = sqrt(nv);
      p.rF[pos] = quot_rn(sf, nv);
      p.rL[pos] = quot_rn(sl, nv);
    } else {
      nv = rsqrt(nv);
      p.rF[pos] = sf * nv;
      p.rL[pos] = sl * nv;
    }
  }
}

// merge node at depth d containing slot position pos (or -1)
__device__ __forceinline__ int find_node(const DcParams& p, int d, int pos) {
  int lo = p.dm_start[d], hi = p.dm_start[d + 1];
  // largest merge node with slot <= pos
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (p.nd_slot[p.depth_merge[mid]] <= pos) lo = mid + 1; else hi = mid;
  }
  if (lo == p.dm_start[d]) return -1;
  int node = p.depth_merge[lo - 1];
  int slot = p.nd_slot[node];
  return (pos < slot + p.nd_nn[node]) ? node : -1;
}

// ---------------------------------------------------------------- P5 final merge
template <bool kBits, class Grp>
__device__ void dc_finish_node(const DcParams& p, int node, int par, bool rows, const Grp& grp) {
  const int t = grp.rank(), nt = grp.size();
  const int nn = p.nd_nn[node], slot = p.nd_slot[node];
  const int q = p.nq[node], nd = nn - q;
  const double* rs = p.rS + slot;
  const double* dd = p.dd + slot;
  double* sig = p.sig[par] + slot;
  double* F = p.F[par] + slot;
  double* L = p.L[par] + slot;
  double nf = 1.0, nl = 1.0;
  if (rows && !kBits) {  // the norms first, then one write of the scaled rows
    const double ph = p.phi[node], ps = p.psi[node];
    double sf = 0.0, sl = 0.0;
    for (int k = t; k < q; k += nt) {
      const double f = p.rF[slot + k], l = p.rL[slot + k];
      sf += f * f;
      sl += l * l;
    }
    for (int k = t; k < nd; k += nt) {
      const double f = p.fd[slot + k], l = p.ld[slot + k];
      sf += f * f;
      sl += l * l;
    }
    nf = sf;
    nl = sl;
    grp.template norms<true>(&nf, ph, &nl, ps);
    if (t == 0) {
      p.phi[node] = ph * nf;
      p.psi[node] = ps * nl;
    }
  }
  for (int k = t; k < q; k += nt) {
    const int pos = k + count_lt(dd, nd, rs[k]);
    sig[pos] = rs[k];
    if (rows) {
      const double f = p.rF[slot + k], l = p.rL[slot + k];
      F[pos] = kBits ? f : f * nf;
      L[pos] = kBits ? l : l * nl;
    }
  }
  for (int k = t; k < nd; k += nt) {
    const int pos = k + count_le(rs, q, dd[k]);
    sig[pos] = dd[k];
    if (rows) {
      const double f = p.fd[slot + k], l = p.ld[slot + k];
      F[pos] = kBits ? f : f * nf;
      L[pos] = kBits ? l : l * nl;
    }
  }
  if (!rows || !kBits) return;
  // kBits: the sums over the merged order, square roots and divisions
  grp.sync();
  double sf = 0.0, sl = 0.0;
  for (int k = t; k < nn; k += nt) { sf += F[k] * F[k]; sl += L[k] * L[k]; }
  const double ph = p.phi[node], ps = p.psi[node];
  grp.template norms<false>(&sf, ph, &sl, ps);
  for (int k = t; k < nn; k += nt) {
    if (sf > 0.0) F[k] = quot_rn(F[k], sf);
    if (sl > 0.0) L[k] = quot_rn(L[k], sl);
  }
  grp.sync();
  if (t == 0) {
    if (sf > 0.0) p.phi[node] = quot_rn(ph, sf);
    if (sl > 0.0) p.psi[node] = quot_rn(ps, sl);
  }
}

#ifdef DDCSVD_PHASE_TRACE
__device__ unsigned long long g_dc_trace[64 * 16];
#endif
// phase marks of CTA 0, one row per depth (slots: 0 start, 1 after P1, 2 after
// its barrier, 3 after P2, 4 barrier, 5 P3, 6 barrier, 7 P4, 8 barrier, 9 P5,
// 10 barrier)
#ifdef DDCSVD_PHASE_TRACE
#define DMARK(slot)                                                               \
  do {                                                                            \
    if (blockIdx.x == 0 && threadIdx.x == 0 && d < 64) g_dc_trace[d * 16 + (slot)] = global_ns(); \
  } while (0)
#else
#define DMARK(slot) \
  do {              \
  } while (0)
#endif

// P2 (phase 0), P3 (1) and P4 (2) of one depth, one lane group per root
template <bool kBits, int kG>
__device__ __forceinline__ void dc_phase(const DcParams& p, int phase, int d, int G, int lane, int gt, int nthreads,
                                         int node0) {
  const LaneGroup<kG> g = make_group<kG>(G, lane);
  const int gid = gt / g.size(), ngroups = nthreads / g.size();
  for (int pos = gid; pos < p.N; pos += ngroups) {
    const int node = (pos == gid) ? node0 : find_node(p, d, pos);
    if (node < 0) continue;
    const int slot = p.nd_slot[node], q = p.nq[node];
    if (pos - slot >= q) continue;
    if (phase == 0) dc_root<kBits>(p, node, slot, pos, q, d, g);
    else if (phase == 1) dc_zhat<kBits>(p, slot, pos, q, g);
    else dc_rows<kBits>(p, slot, pos, q, g);
  }
}

// kCluster: the grid is one thread-block cluster (up to 64 entries, four to a CTA)
// and its hardware barrier, which every CTA reaches whatever the data, stands in
// for the grid's: 0.5 us instead of 1.2, five a depth (64 x 48 factors 482 -> 466 us).
// Beyond 64 entries a cluster's 64 schedulers would take two roots each.
template <bool kBits, bool kCluster>
__global__ void __launch_bounds__(kDcThreads, 1) dc_kernel(DcParams p) {
  __shared__ int shi[40];
  __shared__ double shd[40];
  const int t = threadIdx.x, lane = t & 31;
  // warps numbered across the CTAs first: a depth with fewer lane groups than
  // the grid holds puts one warp on every scheduler before a second on any
  const int gw = (t >> 5) * gridDim.x + blockIdx.x;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int gt = gw * 32 + lane, nthreads = gridDim.x * blockDim.x;
  auto sync = [&](int where) {
    if constexpr (kCluster) {
      cg::this_cluster().sync();
      return true;
    } else {
      return grid_sync(p.bar, p.P, p.st, where);
    }
  };
  for (int d = p.maxdepth; d >= 0; d--) {
    const int par = d & 1;
    const bool rows = d > 0;
    DMARK(0);
    // ---- P1a leaves of this depth (thread each)
    for (int k = p.depth_start[d] + gt; k < p.depth_start[d + 1]; k += nthreads) {
      if (p.nd_K[k] >= 0) continue;
      const int nn = p.nd_nn[k], slot = p.nd_slot[k], r0 = p.nd_r0[k];
      double phi, psi;
      dc_leaf(nn, p.b1 + r0, p.b2 + r0, p.sig[par] + slot, p.F[par] + slot, p.L[par] + slot, &phi, &psi);
      p.phi[k] = phi;
      p.psi[k] = psi;
    }
    // ---- P1b merge set-up: CTA per large node, warp per small node
    {
      const CtaGroup cg{shi, shd};
      for (int mi = p.dm_start[d] + blockIdx.x; mi < p.dm_start[d + 1]; mi += gridDim.x)
        if (p.nd_nn[p.depth_merge[mi]] > kWarpNode) dc_setup_node<kBits>(p, p.depth_merge[mi], par, cg);
      const WarpGroup wg;
      for (int mi = p.dm_start[d] + gw; mi < p.dm_start[d + 1]; mi += nwarps)
        if (p.nd_nn[p.depth_merge[mi]] <= kWarpNode) dc_setup_node<kBits>(p, p.depth_merge[mi], par, wg);
    }
    if (p.dm_start[d + 1] == p.dm_start[d]) {  // only leaves at this depth
      if (d > 0 && !sync(600 + d)) return;
      continue;
    }
    int G = p.dgroup[d];
    if (!kBits) {
      // wider groups while every one still finds a scheduler to itself: an FP64
      // instruction of a lone warp takes 64 cycles, so a lane's chain of terms is
      // the phase's time (kBits: the order of the sums is the host's choice)
      const int wide = min(32, G * p.terms);
      while (G < wide && (long long)p.N * 2 * G <= 128ll * gridDim.x) G *= 2;
    }
    const int gid = gt / G;
    const int node0 = gid < p.N ? find_node(p, d, gid) : -1;  // the forest does not change: ahead of the barrier
    auto phase = [&](int ph) {
      if (G == 32) dc_phase<kBits, 32>(p, ph, d, G, lane, gt, nthreads, node0);
      else dc_phase<kBits, 0>(p, ph, d, G, lane, gt, nthreads, node0);
    };
    DMARK(1);
    if (!sync(100 + d)) return;
    DMARK(2);
    phase(0);  // ---- P2 secular roots
    DMARK(3);
    if (rows) {
      if (!sync(200 + d)) return;
      DMARK(4);
      phase(1);  // ---- P3 z-hat
      DMARK(5);
      if (!sync(300 + d)) return;
      DMARK(6);
      phase(2);  // ---- P4 rows of the merged right vectors
    }
    DMARK(7);
    if (!sync(400 + d)) return;
    DMARK(8);
    // ---- P5 final merge + normalisation (CTA per node)
    {
      const CtaGroup cg{shi, shd};
      for (int mi = p.dm_start[d] + blockIdx.x; mi < p.dm_start[d + 1]; mi += gridDim.x)
        if (p.nd_nn[p.depth_merge[mi]] > kWarpNode) dc_finish_node<kBits>(p, p.depth_merge[mi], par, rows, cg);
      const WarpGroup wg;
      for (int mi = p.dm_start[d] + gw; mi < p.dm_start[d + 1]; mi += nwarps)
        if (p.nd_nn[p.depth_merge[mi]] <= kWarpNode) dc_finish_node<kBits>(p, p.depth_merge[mi], par, rows, wg);
    }
    DMARK(9);
    if (d > 0 && !sync(500 + d)) return;
    DMARK(10);
  }
}

// ---------------------------------------------------------------- tree per CTA
// A forest of many small trees (a batch of small bidiagonals): every CTA takes
// whole trees, largest first, from an atomic counter and runs their depths
// bottom-up with block barriers only -- the same leaf, set-up, root, z-hat,
// row and finish steps as dc_kernel, without its grid barriers (where CTAs
// waited for the slowest one at every phase of every depth).
struct DcTrees {
  int ntrees;
  const int* tree_seg;   // [ntrees + 1] ranges of segments
  const int* seg_lo;     // [nseg + 1] ranges of `nodes` (merges, then leaves)
  const int* seg_mid;    // [nseg] end of the merges
  const int* seg_depth;  // [nseg]
  const int* seg_G;      // [nseg] lanes per root
  const int* nodes;
  const int* order;      // trees, largest first
  int* counter;
};
// 256 threads, or 128 where every node is a warp's: a batch of small problems has
// more trees than 2 x 152 CTAs of the larger size (400 of 36 columns: 443 -> 309 us).  Nodes
// above a warp's keep 256, which is part of the order of their sums.
constexpr int kDcTreeThreads = 256;
constexpr int kDcTreeSmall = 128;

// merge node of segment [lo, mid) containing slot position pos (or -1)
__device__ __forceinline__ int seg_find(const DcParams& p, const int* nodes, int lo, int mid, int pos) {
  int a = lo, b = mid;
  while (a < b) {
    const int c = (a + b) >> 1;
    if (p.nd_slot[nodes[c]] <= pos) a = c + 1; else b = c;
  }
  if (a == lo) return -1;
  const int node = nodes[a - 1];
  return (pos < p.nd_slot[node] + p.nd_nn[node]) ? node : -1;
}

template <int kG>
__device__ __forceinline__ void dc_tree_phase(const DcParams& p, const int* nodes, int lo, int mid, int phase, int d,
                                              int G) {
  const LaneGroup<kG> g = make_group<kG>(G, threadIdx.x & 31);
  const int ngroups = blockDim.x / g.size();
  const int pos0 = p.nd_slot[nodes[lo]];
  const int pos1 = p.nd_slot[nodes[mid - 1]] + p.nd_nn[nodes[mid - 1]];
  for (int pos = pos0 + threadIdx.x / g.size(); pos < pos1; pos += ngroups) {
    const int node = seg_find(p, nodes, lo, mid, pos);
    if (node < 0) continue;
    const int slot = p.nd_slot[node], q = p.nq[node];
    if (pos - slot >= q) continue;
    if (phase == 0) dc_root<true>(p, node, slot, pos, q, d, g);
    else if (phase == 1) dc_zhat<true>(p, slot, pos, q, g);
    else dc_rows<true>(p, slot, pos, q, g);
  }
}

template <int kThreads>
__global__ void __launch_bounds__(kThreads, 512 / kThreads) dc_tree_kernel(DcParams p, DcTrees tr) {
  __shared__ int shi[40];
  __shared__ double shd[40];
  __shared__ int s_tree;
  constexpr int kV = kThreads == kDcTreeSmall ? 2 : 4;
  const int t = threadIdx.x, wid = t >> 5, nw = blockDim.x >> 5;
  while (true) {
    if (t == 0) s_tree = atomicAdd(tr.counter, 1);
    __syncthreads();
    const int qi = s_tree;
    __syncthreads();
    if (qi >= tr.ntrees) break;
    const int tree = tr.order[qi];
    for (int k = tr.tree_seg[tree]; k < tr.tree_seg[tree + 1]; k++) {
      const int lo = tr.seg_lo[k], mid = tr.seg_mid[k], hi = tr.seg_lo[k + 1];
      const int d = tr.seg_depth[k], par = d & 1;
      const bool rows = d > 0;
      // ---- leaves (thread each)
      for (int x = mid + t; x < hi; x += blockDim.x) {
        const int node = tr.nodes[x];
        const int nn = p.nd_nn[node], slot = p.nd_slot[node], r0 = p.nd_r0[node];
        double phi, psi;
        dc_leaf(nn, p.b1 + r0, p.b2 + r0, p.sig[par] + slot, p.F[par] + slot, p.L[par] + slot, &phi, &psi);
        p.phi[node] = phi;
        p.psi[node] = psi;
      }
      if (mid == lo) {  // only leaves at this depth
        __syncthreads();
        continue;
      }
      // ---- merge set-up: the CTA for large nodes, a warp for small ones
      {
        const CtaGroup cg{shi, shd};
        for (int x = lo; x < mid; x++)
          if (p.nd_nn[tr.nodes[x]] > kWarpNode) dc_setup_node<true>(p, tr.nodes[x], par, cg);
        const WarpGroup wg;
        for (int x = lo + wid; x < mid; x += nw)
          if (p.nd_nn[tr.nodes[x]] <= kWarpNode) dc_setup_node<true>(p, tr.nodes[x], par, wg);
      }
      __syncthreads();
      const int G = tr.seg_G[k];
      for (int ph = 0; ph < (rows ? 3 : 1); ph++) {  // secular roots, z-hat, rows
        if (G >= kV) dc_tree_phase<-kV>(p, tr.nodes, lo, mid, ph, d, G / kV);
        else dc_tree_phase<0>(p, tr.nodes, lo, mid, ph, d, G);
        __syncthreads();
      }
      // ---- final merge + normalisation
      {
        const CtaGroup cg{shi, shd};
        for (int x = lo; x < mid; x++)
          if (p.nd_nn[tr.nodes[x]] > kWarpNode) dc_finish_node<true>(p, tr.nodes[x], par, rows, cg);
        const WarpGroup wg;
        for (int x = lo + wid; x < mid; x += nw)
          if (p.nd_nn[tr.nodes[x]] <= kWarpNode) dc_finish_node<true>(p, tr.nodes[x], par, rows, wg);
      }
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------- host: forest
// One tree per unreduced block [lo, hi) of the (split) bidiagonal; a block's
// singular values occupy slots [lo, hi).  Nodes are created depth-first; a
// stable counting sort by depth then gives the order the kernel walks (by
// depth, slots ascending within a depth) without a comparison sort: a batch
// forest has ~10^5 nodes and this runs on the host between two kernels.
namespace {
struct Forest {
  std::vector<int> r0, nn, slot, K, c1, c2, depth;
  int maxdepth = 0;
  int add(int r, int n, int sl, int d) {
    const int id = (int)r0.size();
    r0.push_back(r); nn.push_back(n); slot.push_back(sl);
    K.push_back(-1); c1.push_back(-1); c2.push_back(-1); depth.push_back(d);
    if (d > maxdepth) maxdepth = d;
    return id;
  }
  int build(int r, int n, int sl, int d) {
    const int id = add(r, n, sl, d);
    if (n > 2) {
      const int k = n / 2;
      K[id] = k;
      const int a = build(r, k, sl + 1, d + 1);
      const int b = build(r + k + 1, n - k - 1, sl + k + 1, d + 1);
      c1[id] = a;
      c2[id] = b;
    }
    return id;
  }
};
}  // namespace

void dc_build_host(int N, const std::vector<int>& starts, DcHost& H, int terms_per_lane) {
  Forest T;
  const size_t cap = 2 * (size_t)N + 8;
  T.r0.reserve(cap); T.nn.reserve(cap); T.slot.reserve(cap); T.K.reserve(cap);
  T.c1.reserve(cap); T.c2.reserve(cap); T.depth.reserve(cap);
  std::vector<int> tree_of;  // creation index -> tree
  tree_of.reserve(cap);
  int ntrees = 0;
  for (size_t b = 0; b + 1 < starts.size(); b++) {
    const int lo = starts[b], hi = starts[b + 1];
    if (hi > lo) {
      T.build(lo, hi - lo, lo, 0);
      tree_of.resize(T.r0.size(), ntrees);
      ntrees++;
    }
  }
  const int nnodes = (int)T.r0.size();
  const int md = T.maxdepth;
  // stable counting sort by depth (depth-first creation keeps slots ascending within a depth)
  std::vector<int> ds(md + 2, 0);
  for (int i = 0; i < nnodes; i++) ds[T.depth[i] + 1]++;
  for (int d = 0; d <= md; d++) ds[d + 1] += ds[d];
  std::vector<int> newid(nnodes), fill(ds.begin(), ds.end() - 1);
  for (int i = 0; i < nnodes; i++) newid[i] = fill[T.depth[i]]++;
  std::vector<int> r0(nnodes), nn(nnodes), slot(nnodes), K(nnodes), c1(nnodes), c2(nnodes), dep(nnodes);
  for (int o = 0; o < nnodes; o++) {
    const int i = newid[o];
    dep[i] = T.depth[o];
    r0[i] = T.r0[o]; nn[i] = T.nn[o]; slot[i] = T.slot[o]; K[i] = T.K[o];
    c1[i] = T.c1[o] >= 0 ? newid[T.c1[o]] : -1;
    c2[i] = T.c2[o] >= 0 ? newid[T.c2[o]] : -1;
  }
  std::vector<int> dms(md + 2, 0), dmerge;
  dmerge.reserve(nnodes);
  for (int d = 0; d <= md; d++) {
    dms[d] = (int)dmerge.size();
    for (int i = ds[d]; i < ds[d + 1]; i++) if (K[i] >= 0) dmerge.push_back(i);
  }
  dms[md + 1] = (int)dmerge.size();
  // lanes per root at each depth: about terms_per_lane terms of the largest node per lane
  const int tpl = std::max(1, terms_per_lane);
  std::vector<int> dgroup(md + 2, 1);
  for (int d = 0; d <= md; d++) {
    int mx = 0;
    for (int k = dms[d]; k < dms[d + 1]; k++) mx = std::max(mx, nn[dmerge[k]]);
    int G = 1;
    while (G < 32 && G * tpl < mx) G <<= 1;
    dgroup[d] = G;
  }
  H.nnodes = nnodes;
  H.maxdepth = md;
  H.ndm = (int)dmerge.size();
  H.ints.clear();
  H.ints.reserve(6 * (size_t)nnodes + 3 * (md + 2) + dmerge.size());
  auto app = [&](const std::vector<int>& v) { H.ints.insert(H.ints.end(), v.begin(), v.end()); };
  app(r0); app(nn); app(slot); app(K); app(c1); app(c2); app(ds); app(dms); app(dmerge); app(dgroup);
  // ---- per-tree schedule: each tree's nodes by depth, deepest first; within
  // a depth its merge nodes (ascending slot) then its leaves.  New ids are
  // sorted by (depth, slot), so one ascending pass lists every tree's nodes
  // by depth already.
  // stable counting sort of the node ids by tree (keeps (depth, slot) order)
  std::vector<int> tstart(ntrees + 1, 0), bytree(nnodes);
  for (int o = 0; o < nnodes; o++) tstart[tree_of[o] + 1]++;
  for (int tr = 0; tr < ntrees; tr++) tstart[tr + 1] += tstart[tr];
  {
    std::vector<int> tree_new(nnodes), cur(tstart.begin(), tstart.end() - 1);
    for (int o = 0; o < nnodes; o++) tree_new[newid[o]] = tree_of[o];
    for (int i = 0; i < nnodes; i++) bytree[cur[tree_new[i]]++] = i;
  }
  std::vector<int> tree_seg(ntrees + 1, 0), seg_lo, seg_mid, seg_depth, seg_G, nodes_out, order(ntrees), tsize(ntrees);
  nodes_out.reserve(nnodes);
  seg_lo.reserve(nnodes + 1); seg_mid.reserve(nnodes); seg_depth.reserve(nnodes); seg_G.reserve(nnodes);
  std::vector<int> bounds;  // depth-group boundaries of one tree (reused)
  for (int tr = 0; tr < ntrees; tr++) {
    const int* v = bytree.data() + tstart[tr];
    const int cnt = tstart[tr + 1] - tstart[tr];
    tsize[tr] = cnt ? nn[v[0]] : 0;  // the root (depth 0) comes first
    tree_seg[tr] = (int)seg_lo.size();
    bounds.clear();
    bounds.push_back(0);
    for (int x = 1; x < cnt; x++)
      if (dep[v[x]] != dep[v[x - 1]]) bounds.push_back(x);
    bounds.push_back(cnt);
    for (int gi = (int)bounds.size() - 2; gi >= 0; gi--) {  // deepest first
      const int a = bounds[gi], b = bounds[gi + 1];
      seg_lo.push_back((int)nodes_out.size());
      int mx = 0;
      for (int x = a; x < b; x++)
        if (K[v[x]] >= 0) {
          nodes_out.push_back(v[x]);
          mx = std::max(mx, nn[v[x]]);
        }
      seg_mid.push_back((int)nodes_out.size());
      for (int x = a; x < b; x++)
        if (K[v[x]] < 0) nodes_out.push_back(v[x]);
      seg_depth.push_back(dep[v[a]]);
      int G = 1;
      while (G < 32 && G * tpl < mx) G <<= 1;
      seg_G.push_back(G);
    }
  }
  const int nseg = (int)seg_lo.size();
  tree_seg[ntrees] = nseg;
  seg_lo.push_back((int)nodes_out.size());
  for (int tr = 0; tr < ntrees; tr++) order[tr] = tr;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return tsize[a] > tsize[b]; });
  H.ntrees = ntrees;
  H.nseg = nseg;
  H.maxtree = ntrees ? tsize[order[0]] : 0;
  H.tree_off = H.ints.size();
  app(tree_seg); app(seg_lo); app(seg_mid); app(seg_depth); app(seg_G); app(nodes_out); app(order);
}

// ints of the node table: 9 arrays of at most 2N + 8 entries, the per-depth
// tables, and the per-tree schedule (at most N trees, 2N + 8 segments and nodes)
size_t dc_max_ints(int N) { return 9 * (size_t)(2 * N + 8) + 2 * 64 + 16 + 2 * ((size_t)N + 1) + 5 * (2 * (size_t)N + 9); }


int dc_sigma(ddcsvd_context* ctx, int N, const double* b1, const double* b2, double* sigma,
             const DcHost* H, const int* dints, Arena& a, bool plan_only, bool keep_bits, GridBarrier* zeroed) {
  if (N <= 0) return DDCSVD_ERR_ARG;
  const int maxnodes = 2 * N + 8;
  int* scratch_ints = a.take<int>((size_t)N + maxnodes);
  double* dbl = a.take<double>((size_t)N * 25 + 3 * (size_t)maxnodes + 8);
  float* flt = a.take<float>((size_t)N * 3 + 8);
  GridBarrier* bar = a.take<GridBarrier>(4);
  if (plan_only) return DDCSVD_OK;
  const int nnodes = H->nnodes, md = H->maxdepth;
  DcParams p;
  p.N = N; p.nnodes = nnodes; p.maxdepth = md;
  p.terms = std::max(1, ctx->tune[TK_DC_TERMS]);
  p.maxit = ctx->sec_maxit;
  size_t o = 0;
  p.nd_r0 = dints + o; o += nnodes;
  p.nd_nn = dints + o; o += nnodes;
  p.nd_slot = dints + o; o += nnodes;
  p.nd_K = dints + o; o += nnodes;
  p.nd_c1 = dints + o; o += nnodes;
  p.nd_c2 = dints + o; o += nnodes;
  p.depth_start = dints + o; o += md + 2;
  p.dm_start = dints + o; o += md + 2;
  p.depth_merge = dints + o; o += H->ndm;
  p.dgroup = dints + o; o += md + 2;
  p.defl = scratch_ints;
  p.nq = scratch_ints + N;
  p.b1 = b1; p.b2 = b2;
  double* q = dbl;
  p.sig[0] = sigma;  // depth 0 writes the result in place
  p.sig[1] = q; q += N;
  for (int k = 0; k < 2; k++) { p.F[k] = q; q += N; p.L[k] = q; q += N; }
  p.ds = q; q += N; p.zs = q; q += N; p.hfs = q; q += N; p.hls = q; q += N;
  p.dq = q; q += N; p.zq = q; q += N; p.fq = q; q += N; p.lq = q; q += N;
  p.dd = q; q += N; p.fd = q; q += N; p.ld = q; q += N;
  p.tau = q; q += N; p.dor = q; q += N; p.zh = q; q += N; p.rS = q; q += N; p.rF = q; q += N; p.rL = q; q += N;
  p.zz = q; q += maxnodes; p.phi = q; q += maxnodes; p.psi = q; q += maxnodes;
  p.dqf = reinterpret_cast<float2*>(flt); p.zqf = flt + 2 * (size_t)N;
  if (zeroed) bar = zeroed;
  else DDC_CUDA_TRY(cudaMemsetAsync(bar, 0, sizeof(GridBarrier), ctx->stream));
  p.bar = bar;
  p.st = ctx->d_status;
  // a forest of many small trees: whole trees per CTA, no grid barriers
  if (H->ntrees >= 64 && H->maxtree <= 1024) {
    DcTrees tr;
    size_t q2 = H->tree_off;
    const int nt = H->ntrees, ns = H->nseg;
    tr.ntrees = nt;
    tr.tree_seg = dints + q2; q2 += nt + 1;
    tr.seg_lo = dints + q2; q2 += ns + 1;
    tr.seg_mid = dints + q2; q2 += ns;
    tr.seg_depth = dints + q2; q2 += ns;
    tr.seg_G = dints + q2; q2 += ns;
    tr.nodes = dints + q2; q2 += nnodes;
    tr.order = dints + q2;
    tr.counter = reinterpret_cast<int*>(bar);
    int occ = 0;
    const bool small = H->maxtree <= kWarpNode;
    const int threads = small ? kDcTreeSmall : kDcTreeThreads;
    const auto kern = small ? dc_tree_kernel<kDcTreeSmall> : dc_tree_kernel<kDcTreeThreads>;
    DDC_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, threads, 0));
    const int grid = std::max(1, std::min(nt, ctx->num_sms * std::max(occ, 1)));
    ktimer_begin(ctx, KC_DC);
    kern<<<grid, threads, 0, ctx->stream>>>(p, tr);
    ktimer_end(ctx);
    count_launch();
    DDC_CUDA_TRY(cudaGetLastError());
    return DDCSVD_OK;
  }
  const int P = std::min(ctx->num_sms, std::max(1, ceil_div(N, 4)));
  p.P = P;
  void* argv[] = {&p};
  if (!keep_bits && P <= tail_cluster_size(ctx)) {
    int C = 1;
    while (C < P) C *= 2;
    const void* kern = (const void*)dc_kernel<false, true>;
    if (C > 8) DDC_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(kDcThreads);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    ktimer_begin(ctx, KC_DC);
    DDC_CUDA_TRY(cudaLaunchKernelExC(&cfg, kern, argv));
    ktimer_end(ctx);
    count_launch();
    return DDCSVD_OK;
  }
  int occ = 0;
  const void* kern = keep_bits ? (const void*)dc_kernel<true, false> : (const void*)dc_kernel<false, false>;
  DDC_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kDcThreads, 0));
  if (occ < 1) {
    set_last_error("dc_kernel cannot be resident");
    return DDCSVD_ERR_CUDA;
  }
  ktimer_begin(ctx, KC_DC);
  DDC_CUDA_TRY(cudaLaunchCooperativeKernel(kern, dim3(P), dim3(kDcThreads), argv, 0,
                                           ctx->stream));
  ktimer_end(ctx);
  count_launch();
  DDC_CUDA_TRY(cudaGetLastError());
  return DDCSVD_OK;
}

}  // namespace ddcsvd

#ifdef DDCSVD_PHASE_TRACE
extern "C" int ddcsvd_dc_trace_read(unsigned long long* out) {
  return (int)cudaMemcpyFromSymbol(out, ddcsvd::g_dc_trace, sizeof(ddcsvd::g_dc_trace));
}
extern "C" int ddcsvd_dc_iters_read(unsigned* out) {
  return (int)cudaMemcpyFromSymbol(out, ddcsvd::g_dc_iters, sizeof(ddcsvd::g_dc_iters));
}
#endif
