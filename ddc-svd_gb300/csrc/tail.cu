// tail.cu -- the last columns of the blocked bidiagonalisation on one
// thread-block cluster, the trailing block in registers.
//
// Once the trailing block W[k0:m, k0:n] of the panel factorisation is small
// enough, the remaining columns no longer pay the grid-wide costs of the panel
// kernel (two grid barriers and two reductions over 152 partial records per
// column, ~9 us at any size).  One cluster of C CTAs (up to 16) holds the whole
// block: row r belongs to one warp (row r to warp r mod 8C of the cluster, so
// the work stays even while rows retire), lane l of the warp holds its columns
// l, l + 32, ... in registers.  The algorithm is the unblocked one of the
// reference (bidiag_par.c:310-397, left_update_mat.cl / right_update_mat.cl): per
// column a left reflector and its rank-1 update, then a right reflector and its
// rank-1 update.  Reflector conventions, FP32 compensated norms and the
// LAPACK-form storage are those of the panel kernel.
//
// Per column i the block is read and written once, in registers: the left
// update with (u, tau y), the row's product with v, the right update, and the
// unscaled products sum_r x_r A[r, c] of the next column x with every column.
// Between columns the CTAs exchange vectors along c only (the row-shaped
// vectors never leave their warps):
//   1. each CTA adds its warps' products and sends them, slice by slice (CTA k
//      owns the columns 32 k .. 32 k + 31), to the slice's owner, with the
//      squared norm of its part of x; the warp of row i sends that row;
//   2. each CTA adds the C partial products of its slice, forms the left
//      reflector (every CTA the same one, from the same C norms), tau y and the
//      new row w of its columns, and sends both to every CTA with the slice's
//      part of ||w||^2; every warp then forms the right reflector.
// Both exchanges are remote asynchronous stores that complete on the receiver's
// mbarrier (one way, 340-490 cycles for 2-16 CTAs; stores followed by a hardware
// cluster barrier, whose release waits for their acknowledgement, measured
// 690-1200), and a CTA receives 2 nt floats per column.
//
// What bounds it: the chain of the two exchanges and of the two norms (sums of
// records, a square root and quotients each) -- not arithmetic: a 512 x 512
// block is 32 elements a thread.  The former kernel kept columns instead of
// rows, in shared memory, and let every CTA read all C partial row-vectors
// (64 mt bytes per CTA and column through distributed shared memory at ~8
// bytes a clock).  Us per column, before and now: 64 x 48 3.5 and 1.5, 512 x 256
// 5.3 and 1.9, 900 x 250 8.5 and 2.3, 1000 x 490 9 and 2.8.
#include <cooperative_groups.h>

#include "async.cuh"
#include "internal.hpp"

namespace cg = cooperative_groups;

namespace ddcsvd {

constexpr int kTailThreads = 256;
constexpr int kTailWarps = kTailThreads / 32;
constexpr int kTailMaxC = 16;
constexpr int kEx1Bars = 2;  // barriers of exchange 1 (the kernel says why not one)

struct TailParams {
  int mt, nt;  // trailing block: rows, columns (mt >= nt)
  float* W;    // trailing block (its row 0 / column 0 = the first tail column)
  int ldw;
  float *d, *e, *tauq, *taup;  // offset to the first tail column
  DevStatus* st;
};

// Remote stores that complete on the target CTA's mbarrier (addresses in the
// shared::cluster window, from mapa).
__device__ __forceinline__ uint32_t map_rank(uint32_t a, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_async(uint32_t dst, float v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst),
               "r"(__float_as_uint(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async(uint32_t dst, float a, float b, uint32_t bar) {
  const unsigned long long v = (unsigned long long)__float_as_uint(b) << 32 | __float_as_uint(a);
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst), "l"(v), "r"(bar)
               : "memory");
}

// Waits for the phase of the given parity.  Bounded by the handle's limit: when
// it runs out the status word holds DDCSVD_ERR_TIMEOUT, and then or when it holds
// another CTA's error `dead` is set in this thread: it waits, sends and arms
// barriers no more, and the column loop runs out with meaningless values (leaving
// it instead takes a barrier that agrees on `dead`, 0.1 us a column).
constexpr unsigned long long kTailLateNs = 20000;  // from here on the status word is read (a column takes 1.5-3 us)
__device__ __forceinline__ void tail_wait(uint32_t bar, unsigned parity, bool& dead, DevStatus* st) {
  unsigned long long t0 = 0;
  for (unsigned polls = 0; !dead; polls++) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n"
        " mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return;
    if ((polls & 63u) == 63u) {
      const unsigned long long now = global_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 < kTailLateNs) continue;
      const uint4 s = ld_status(st);
      if (s.x != 0) {
        dead = true;
      } else if (now - t0 > (s.z ? 1000ull * s.z : kWaitLimitNs)) {
        set_error(st, DDCSVD_ERR_TIMEOUT, 700);
        dead = true;
      }
    }
  }
}

// R rows per warp, K columns per lane: blocks of up to 8 C R rows and 32 K
// columns.
template <int R, int K>
__global__ void __launch_bounds__(kTailThreads, 1) bidiag_tail_kernel(TailParams p) {
  constexpr int H = R < 4 ? R : 4;   // rows, and columns per lane, whose work is skipped together
  constexpr int KC = K < 4 ? K : K == 8 ? 8 : 4;  // once they have retired
  constexpr int NS = (K + 7) / 8;    // slices a warp sends to: wid and wid + 8
  constexpr int NT = kTailMaxC / kTailWarps;  // CTAs a warp sends to: the same
  __shared__ float s_part[kTailWarps][32 * K];  // per warp: products of the next column with every column
  __shared__ FF s_nw[kTailWarps];               // per warp: ||x||^2 of the own rows
  __shared__ float s_own[32 * K];               // row i, in the CTA that holds it
  // exchange 1, records and barrier by column parity.  A CTA may send column
  // i + 1's records to one that still reads column i's, or still waits for some
  // of them: it has come through exchange 2 of column i, for which the owners of
  // the slices left needed every CTA's record of column i at themselves, but
  // nobody needed it at a CTA without a slice.  On one barrier its bytes would
  // count for those still missing.  It cannot send column i + 2's: the owners
  // then had that CTA's record of column i + 1, sent after its last read of
  // column i.
  __shared__ __align__(16) float s_in[2][kTailMaxC][32];  // partial products of the own slice by sender
  __shared__ __align__(16) float s_row[2][32];            // row i of the own slice
  __shared__ __align__(16) FF s_n1[2][kTailMaxC];         // ||x||^2 by sender
  __shared__ float s_x0[2];                               // A[i, i]
  // exchange 2 (sent after exchange 1 has completed, so after every read of
  // the previous column's)
  __shared__ __align__(16) float2 s_yw[32 * K];  // (tau y, w) of every column
  __shared__ __align__(16) FF s_n2[kTailMaxC];   // ||w||^2 over the columns > i + 1 by slice
  __shared__ __align__(8) uint64_t s_bar[kEx1Bars + 1];  // exchange 1 by column parity, exchange 2
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const int mt = p.mt, nt = p.nt, ldw = p.ldw;
  const int GW = kTailWarps * C, gw = wid * C + rank;  // row r: warp r mod GW, slot r / GW
  const int c_own = 32 * rank + lane;                  // the lane's column of the CTA's slice
  const int slice_cols = min(32, nt - 32 * rank);      // (<= 0: no slice)
  const uint32_t bar0 = smem_u32(&s_bar[0]), bar2 = smem_u32(&s_bar[kEx1Bars]);
  // a shared address of this CTA plus such a difference is the same place in
  // CTA lane's / CTA (wid + 8 j)'s shared memory
  const uint32_t to_lane = map_rank(bar0, min(lane, C - 1)) - bar0;
  uint32_t to_cta[NT];
#pragma unroll
  for (int j = 0; j < NT; j++) to_cta[j] = map_rank(bar0, min(wid + 8 * j, C - 1)) - bar0;
  bool dead = false;
  // the handle's extra arrivals stand for a CTA whose norm never comes (tests of the bounded waits)
  const bool lost = rank == 0 && ld_status(p.st).w != 0;

  float A[R][K];
#pragma unroll
  for (int s = 0; s < R; s++)
#pragma unroll
    for (int k = 0; k < K; k++) {
      const int r = s * GW + gw, c = lane + 32 * k;
      A[s][k] = (r < mt && c < nt) ? p.W[r + (size_t)c * ldw] : 0.f;
    }
  float x[R];  // the current column's entries of the own rows (zero for retired rows)
#pragma unroll
  for (int s = 0; s < R; s++) {
    const float v = __shfl_sync(0xffffffffu, A[s][0], 0);
    x[s] = (s * GW + gw > 0) ? v : 0.f;
  }
  float acc[K];
#pragma unroll
  for (int k = 0; k < K; k++) {
    acc[k] = 0.f;
#pragma unroll
    for (int s = 0; s < R; s++) acc[k] += x[s] * A[s][k];
  }
  // records of absent CTAs and columns read as zero
  for (int q = t; q < 2 * kTailMaxC * 32; q += kTailThreads) (&s_in[0][0][0])[q] = 0.f;
  if (t < 2 * kTailMaxC) (&s_n1[0][0])[t] = FF{0.f, 0.f};
  if (t == 0) {
    for (int q = 0; q <= kEx1Bars; q++) mbar_init(&s_bar[q], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  cluster.sync();  // every CTA runs and is ready before the first remote store

  int islot = 0, iwarp = 0;  // slot and warp of row i
  for (int i = 0; i < nt; i++) {
    const int b = i & 1;
    const uint32_t bar1 = smem_u32(&s_bar[b]);
    const unsigned ph1 = (unsigned)(i >> 1) & 1u;  // a phase of it every other column
    const unsigned ph2 = (unsigned)b;              // and of exchange 2's in each
    const int kf = (i + 1) >> 5;            // first slice with a column > i
    const bool mine = gw == iwarp;          // this warp holds row i
    // ---- exchange 1: products of column i, its norm, row i
    if (t == 0 && !dead) {
      unsigned bytes = 8u * C + 4u;
      if (rank >= kf && slice_cols > 0) bytes += 4u * (C + 1) * slice_cols;
      mbar_arrive_expect_tx(&s_bar[b], bytes);
      if (i < nt - 1)
        mbar_arrive_expect_tx(&s_bar[kEx1Bars], 8u * (unsigned)((nt + 31) / 32 - kf) + 8u * (unsigned)(nt - 32 * kf));
    }
#pragma unroll
    for (int k = 0; k < K; k++) s_part[wid][lane + 32 * k] = acc[k];
    {
      FF n[R];
#pragma unroll
      for (int s = 0; s < R; s++) n[s] = ff_square(x[s]);
#pragma unroll
      for (int m = R; m > 1; m = (m + 1) / 2)
#pragma unroll
        for (int s = 0; s < m / 2; s++) n[s] = ff_acc(n[s], n[s + (m + 1) / 2]);
      if (lane == 0) s_nw[wid] = n[0];
    }
    if (mine) {
#pragma unroll
      for (int r = 0; r < R; r++)
        if (r == islot) {
#pragma unroll
          for (int k = 0; k < K; k++) s_own[lane + 32 * k] = A[r][k];
        }
    }
    __syncthreads();
    const bool holds = rank == (iwarp & (C - 1));  // row i is in this CTA
#pragma unroll
    for (int j = 0; j < NS; j++) {
      const int c = t + kTailThreads * j;  // warp wid: slice wid + 8 j
      if (c >= 32 * kf && c < nt && !dead) {
        float v[kTailWarps];
#pragma unroll
        for (int w = 0; w < kTailWarps; w++) v[w] = s_part[w][c];
        if (holds) st_async(smem_u32(&s_row[b][lane]) + to_cta[j], s_own[c], bar1 + to_cta[j]);
        const float sum = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
        st_async(smem_u32(&s_in[b][rank][lane]) + to_cta[j], sum, bar1 + to_cta[j]);
      }
    }
    if (wid == kTailWarps - 1) {
      const FF n = ff_lanes<kTailWarps>(s_nw[lane & (kTailWarps - 1)]);
      if (lane < C && !dead) {
        if (!lost) st_async(smem_u32(&s_n1[b][rank]) + to_lane, n.hi, n.lo, bar1 + to_lane);
        if (holds) st_async(smem_u32(&s_x0[b]) + to_lane, s_own[i], bar1 + to_lane);
      }
    }
    tail_wait(bar1, ph1, dead, p.st);
    // ---- left reflector, and exchange 2: tau y and the new row of the own
    // slice (every warp forms them; warp w sends them to the CTAs w, w + 8)
    float alpha, tq, sq, w = 0.f;
    {
      const FF n1 = ff_lanes<kTailMaxC>(s_n1[b][lane & (kTailMaxC - 1)]);
      const bool in = c_own < nt && c_own > i;
      float v[kTailMaxC];
#pragma unroll
      for (int q = 0; q < kTailMaxC; q++) v[q] = s_in[b][q][lane];
#pragma unroll
      for (int h = kTailMaxC / 2; h > 0; h >>= 1)
#pragma unroll
        for (int q = 0; q < h; q++) v[q] += v[q + h];
      const float row = s_row[b][lane];
      householder_fast(s_x0[b], n1, &alpha, &tq, &sq);
      const float ty = in ? tq * (row + sq * v[0]) : 0.f;
      w = in ? row - ty : 0.f;
      if (i < nt - 1 && rank >= kf && slice_cols > 0) {
#pragma unroll
        for (int j = 0; j < NT; j++)
          if (c_own < nt && wid + 8 * j < C && !dead)
            st_async(smem_u32(&s_yw[c_own]) + to_cta[j], ty, w, bar2 + to_cta[j]);
        const FF n2 = ff_lanes<32>(c_own > i + 1 ? ff_square(w) : FF{0.f, 0.f});
#pragma unroll
        for (int j = 0; j < NT; j++)
          if (lane == 0 && wid + 8 * j < C && !dead)
            st_async(smem_u32(&s_n2[rank]) + to_cta[j], n2.hi, n2.lo, bar2 + to_cta[j]);
      }
    }
    if (rank == 0 && t == 0) {
      p.d[i] = alpha;
      p.tauq[i] = tq;
    }
    // column i of W: 1 on the diagonal, u below
    {
      float v = 0.f;
#pragma unroll
      for (int s = 0; s < R; s++) {
        x[s] *= sq;  // now u
        if (lane == s) v = x[s];
      }
      const int r = lane * GW + gw;
      if (lane < R && r >= i && r < mt) p.W[r + (size_t)i * ldw] = (r == i) ? 1.f : v;
    }
    if (i == nt - 1) break;
    tail_wait(bar2, ph2, dead, p.st);
    // ---- right reflector (every warp); row i of W
    float tp = 0.f, sp = 0.f;
    {
      const float w1 = s_yw[i + 1].y;
      float beta = w1;  // one element left: no reflection (bidiag.c:125-129)
      if (i < nt - 2) {
        const int q = lane & (kTailMaxC - 1);
        const FF n2 = ff_lanes<kTailMaxC>((q >= kf && 32 * q < nt) ? s_n2[q] : FF{0.f, 0.f});
        householder_fast(w1, n2, &beta, &tp, &sp);
      }
      if (rank == 0 && t == 0) {
        p.e[i] = beta;
        p.taup[i] = tp;
      }
      if (wid == 1 && c_own > i && c_own < nt)
        p.W[i + (size_t)c_own * ldw] = (c_own == i + 1) ? (tp != 0.f ? 1.f : 0.f) : sp * w;
    }
    // ---- left update, products with v = (1, sp w), per row
    float z[R], nx[R];
#pragma unroll
    for (int s = 0; s < R; s++) z[s] = nx[s] = 0.f;
    auto vcol = [&](int c, float wv) { return (c == i + 1) ? 1.f : (c > i + 1 && c < nt) ? sp * wv : 0.f; };
#pragma unroll
    for (int k0 = 0; k0 < K; k0 += KC) {
      if (k0 + KC <= kf) continue;
      float ty[KC], v[KC];
#pragma unroll
      for (int k = 0; k < KC; k++) {
        const int c = lane + 32 * (k0 + k);
        const float2 yw = s_yw[c];
        ty[k] = (c > i && c < nt) ? yw.x : 0.f;
        v[k] = vcol(c, yw.y);
      }
#pragma unroll
      for (int h = 0; h < R; h += H) {
        if ((h + H - 1) * GW + gw <= i) continue;
#pragma unroll
        for (int s = h; s < h + H; s++)
#pragma unroll
          for (int k = 0; k < KC; k++) {
            A[s][k0 + k] -= x[s] * ty[k];
            z[s] += A[s][k0 + k] * v[k];
          }
      }
#pragma unroll
      for (int k = 0; k < KC; k++)
        if (k0 + k == kf) {
#pragma unroll
          for (int s = 0; s < R; s++) nx[s] = A[s][k0 + k];
        }
    }
    {
      constexpr int P = R < 8 ? R : (R & 8) ? 8 : 16;  // R = 2, 4 or a sum of 16s, 8s and a 4
#pragma unroll
      for (int q = 0; q + P <= R; q += P) warp_sums<P>(z, q, lane);
      if (R % P) warp_sums<(R % P) ? R % P : 1>(z, R - R % P, lane);
    }
#pragma unroll
    for (int s = 0; s < R; s++) {
      z[s] *= tp;
      const float v = __shfl_sync(0xffffffffu, nx[s], (i + 1) & 31) - z[s];
      x[s] = (s * GW + gw > i + 1) ? v : 0.f;
    }
    // ---- right update and the products of the next column
#pragma unroll
    for (int k0 = 0; k0 < K; k0 += KC) {
      if (k0 + KC <= kf) continue;
      float v[KC];
#pragma unroll
      for (int k = 0; k < KC; k++) {
        const int c = lane + 32 * (k0 + k);
        v[k] = vcol(c, s_yw[c].y);
        acc[k0 + k] = 0.f;
      }
#pragma unroll
      for (int h = 0; h < R; h += H) {
        if ((h + H - 1) * GW + gw <= i) continue;
#pragma unroll
        for (int s = h; s < h + H; s++)
#pragma unroll
          for (int k = 0; k < KC; k++) {
            A[s][k0 + k] -= z[s] * v[k];
            acc[k0 + k] += x[s] * A[s][k0 + k];
          }
      }
    }
    if (++iwarp == GW) {
      iwarp = 0;
      islot++;
    }
  }
  if (dead) __nanosleep(100000);  // remote stores still under way land before any CTA leaves
  cluster.sync();
}

// The kernel for R rows per warp and K columns per lane (at most 192
// registers of the block per thread; the three largest tiles spill a few
// hundred bytes and still beat the panel kernel, whose trailing updates would
// also cost accuracy on tall blocks: a tensor-core GEMM rounds towards zero).
static const void* tail_kernel(int R, int K) {
#define DDC_TAIL(r, k) \
  if (R == r && K == k) return (const void*)bidiag_tail_kernel<r, k>
  DDC_TAIL(2, 2); DDC_TAIL(4, 2); DDC_TAIL(8, 2); DDC_TAIL(16, 2); DDC_TAIL(24, 2);
  DDC_TAIL(2, 4); DDC_TAIL(4, 4); DDC_TAIL(8, 4); DDC_TAIL(16, 4); DDC_TAIL(24, 4);
  DDC_TAIL(2, 8); DDC_TAIL(4, 8); DDC_TAIL(8, 8); DDC_TAIL(16, 8); DDC_TAIL(24, 8);
  DDC_TAIL(4, 12); DDC_TAIL(8, 12); DDC_TAIL(12, 12); DDC_TAIL(16, 12);
  DDC_TAIL(4, 16); DDC_TAIL(8, 16); DDC_TAIL(12, 16);
#undef DDC_TAIL
  return nullptr;
}

// Cluster size the device can co-schedule (16, else 8, else 0), cached.
int tail_cluster_size(ddcsvd_context* ctx) {
  if (ctx->tail_cluster >= 0) return ctx->tail_cluster;
  int best = 0;
  for (int c : {16, 8}) {
    const void* fn = tail_kernel(8, 16);
    if (c > 8 && cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) continue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(kTailThreads);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = c;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int nclusters = 0;
    if (cudaOccupancyMaxActiveClusters(&nclusters, fn, &cfg) == cudaSuccess && nclusters >= 1) {
      best = c;
      break;
    }
  }
  cudaGetLastError();  // a refused attribute or query only means no cluster tail
  ctx->tail_cluster = best;
  return best;
}

// Cluster size and register tile for an mt x nt block (C = 0: it does not fit):
// the fewest CTAs that leave two rows a warp, else the largest cluster.  The
// exchanges cost nearly the same for any C, the rows' work shrinks with it
// (us per column: 64 x 48 C = 4 1.52, C = 2 1.61; 256^2 C = 16 1.74, C = 8 1.87;
// 512 x 256 C = 16 1.89, C = 8 2.25).
struct TailConfig {
  int C, R, K;
};
static TailConfig tail_config(int mt, int nt, int cmax) {
  TailConfig g{0, 0, 0};
  for (int K : {2, 4, 8, 12, 16})
    if (32 * K >= nt) {
      g.K = K;
      break;
    }
  if (g.K == 0) return g;
  int C = 1;
  while (32 * C < nt) C *= 2;  // a slice of columns is at most one warp wide
  for (; C <= cmax; C *= 2)
    for (int R : {2, 4, 8, 12, 16, 24})
      if (kTailWarps * C * R >= mt && tail_kernel(R, g.K) && (R <= 2 || C == cmax)) {
        g.C = C;
        g.R = R;
        return g;
      }
  return g;
}

int bidiag_tail_columns(ddcsvd_context* ctx, int m, int n, int k0) {
  const int cap = ctx->tune[TK_PANEL_TAIL];
  const int mt = m - k0, nt = n - k0;
  if (cap <= 0 || nt > cap || nt <= 0 || mt < nt) return 0;
  return tail_config(mt, nt, tail_cluster_size(ctx)).C > 0 ? nt : 0;
}

int bidiag_tail(ddcsvd_context* ctx, int m, int n, int k0, float* W, int ldw, float* d, float* e, float* tauq,
                float* taup) {
  TailParams p;
  p.mt = m - k0;
  p.nt = n - k0;
  const TailConfig g = tail_config(p.mt, p.nt, tail_cluster_size(ctx));
  if (g.C == 0) return DDCSVD_ERR_UNSUPPORTED;
  p.W = W + k0 + (size_t)k0 * ldw;
  p.ldw = ldw;
  p.d = d + k0;
  p.e = e + k0;
  p.tauq = tauq + k0;
  p.taup = taup + k0;
  p.st = ctx->d_status;
  const void* fn = tail_kernel(g.R, g.K);
  if (g.C > 8) DDC_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g.C);
  cfg.blockDim = dim3(kTailThreads);
  cfg.stream = ctx->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = g.C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  void* args[] = {&p};
  DDC_CUDA_TRY(cudaLaunchKernelExC(&cfg, fn, args));
  count_launch();
  return DDCSVD_OK;
}

}  // namespace ddcsvd
