// resident.cu -- the columns of the blocked bidiagonalisation between the panels
// and the cluster tail, the trailing block in the registers of the whole grid.
//
// Once the trailing block fits the register files (2432 rows by 2048 columns on
// 152 SMs), the unblocked algorithm of the tail (tail.cu; reflector conventions,
// compensated FP32 norms and storage are the same) runs on one persistent
// cooperative grid.  CTA b holds the R rows from b R on; thread t of its 512 holds
// columns t, t + 512, ..., so the products of a column with the others are sums
// inside a thread, and the right update's row sums one reduce-scatter per warp.
// Per column i:
//   1. each CTA writes its part of x^T A (x: the unscaled column i) and of ||x||^2;
//      the owner of row i writes that row;
//   2. after a grid barrier each CTA adds the P parts of its slice of the columns
//      (every CTA forms the same reflector from the P norms in a warp of its own),
//      and writes tau y of the slice and its part of ||w||^2, w the new row i;
//   3. after a second barrier every CTA reads y, updates its rows, forms their
//      products with v (the scale follows in a seventeenth warp meanwhile), applies
//      the right update and hands on column i + 1.
//
// What bounds it: the two barriers (1.3 us each) and the two round trips to L2
// behind them; the arithmetic is 4 R K multiply-adds a thread.  The panel kernel
// reads the trailing block from L2 for every column, sums 152 records of 2 j
// values twice and one 152-part row product: 11-13 us a column at 1000-2000
// columns, where this takes @@ (the trailing update's product comes on top there).
#include "internal.hpp"

namespace ddcsvd {

namespace {

constexpr int kResThreads = 512;             // threads that hold the block
constexpr int kResWarps = kResThreads / 32;  // and the warp of the norms behind them
constexpr int kResSlice = 16;                // most columns of a CTA's slice

struct ResParams {
  int mt, nt, cols;  // trailing block and the columns to take
  int ldw, ldp, ldr;
  float* W;  // trailing block
  float *d, *e, *tauq, *taup;
  float* part;      // P x ldp: x^T A by CTA
  float* y;         // tau y
  float* row;       // 2 x ldr: row i, by column parity
  float2 *cn, *rn;  // P: compensated parts of ||x||^2 and ||w||^2
  GridBarrier* bar;
  DevStatus* st;
};

template <int R, int K>
__global__ void __launch_bounds__(kResThreads + 32, 1) bidiag_resident_kernel(ResParams p) {
  constexpr int B = R > 8 ? 16 : 8;  // rows of the reduce-scatter
  static_assert(R % 4 == 0 && R <= 16, "rows come in float4s, sixteen warps finish their sums");
  __shared__ __align__(16) float s_x[R], s_u[R], s_z[R];  // own rows of x, u and of the right update
  __shared__ float s_c1[R], s_red[kResWarps][B], s_sl[kResWarps][kResSlice], s_q[2], s_p[2];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5, b = blockIdx.x, P = gridDim.x;
  const bool main = t < kResThreads;
  const int mt = p.mt, nt = p.nt, r0 = b * R, ldw = p.ldw;
  float a[R][K];
  if (main) {
#pragma unroll
    for (int k = 0; k < K; k++) {
      const int c = t + k * kResThreads;
      const float* col = p.W + r0 + (size_t)c * ldw;
#pragma unroll
      for (int r = 0; r < R; r += 4) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < nt && r0 + r < mt) {  // (the last float4 may end in padding rows: ldw is a multiple of 32)
          v = __ldcg(reinterpret_cast<const float4*>(col + r));
          if (r0 + r + 1 >= mt) v.y = 0.f;
          if (r0 + r + 2 >= mt) v.z = 0.f;
          if (r0 + r + 3 >= mt) v.w = 0.f;
        }
        a[r][k] = v.x; a[r + 1][k] = v.y; a[r + 2][k] = v.z; a[r + 3][k] = v.w;
      }
    }
    if (t == 0) {
#pragma unroll
      for (int r = 0; r < R; r++) s_x[r] = a[r][0];
    }
  }
  __syncthreads();
  for (int i = 0; i < p.cols; i++) {
    float* row = p.row + (i & 1) * p.ldr;
    const bool own = i >= r0 && i < r0 + R;  // row i is here
    // ---- 1. parts of x^T A and ||x||^2 (rows below i), row i
    if (main) {
      float s[K];
#pragma unroll
      for (int k = 0; k < K; k++) s[k] = 0.f;
#pragma unroll
      for (int r = 0; r < R; r += 4) {
        const float4 xv = *reinterpret_cast<const float4*>(s_x + r);
        const float x4[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const float x = (r0 + r + u > i) ? x4[u] : 0.f;
#pragma unroll
          for (int k = 0; k < K; k++) s[k] += a[r + u][k] * x;
        }
      }
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int c = t + k * kResThreads;
        if (c > i && c < nt) p.part[(size_t)b * p.ldp + c] = s[k];
      }
      if (own) {
#pragma unroll
        for (int r = 0; r < R; r++)
          if (r0 + r == i) {
#pragma unroll
            for (int k = 0; k < K; k++) {
              const int c = t + k * kResThreads;
              if (c >= i && c < nt) row[c] = a[r][k];
            }
          }
      }
    } else {
      FF n{0.f, 0.f};
      if (lane < R && r0 + lane > i) n = ff_add_sq(n, s_x[lane]);
      n = warp_sum_ff(n);
      if (lane == 0) p.cn[b] = make_float2(n.hi, n.lo);
    }
    if (!grid_sync(p.bar, P, p.st, 50)) return;
    // ---- 2. left reflector; tau y and the new row on the CTA's slice of the columns
    const int ncol = nt - (i + 1), cc = (ncol + P - 1) / P;  // (at most kResSlice: the host's choice of shapes)
    const int c0 = i + 1 + b * cc, nc = max(0, min(cc, nt - c0));
    float rw[K], wic = 0.f;
    if (main) {
      const int lg = cc > 8 ? 4 : cc > 4 ? 3 : 2, w = 1 << lg;  // lanes per record
      const int cl = t & (w - 1), nrec = kResThreads >> lg;
      if (wid == 0 && lane < nc) wic = __ldcg(row + c0 + lane);
      float s = 0.f;
      for (int q = t >> lg; q < P; q += 5 * nrec) {
        float v[5];
#pragma unroll
        for (int u = 0; u < 5; u++)
          v[u] = (cl < nc && q + u * nrec < P) ? __ldcg(p.part + (size_t)(q + u * nrec) * p.ldp + c0 + cl) : 0.f;
#pragma unroll
        for (int u = 0; u < 5; u++) s += v[u];
      }
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int c = t + k * kResThreads;
        rw[k] = (c > i && c < nt) ? __ldcg(row + c) : 0.f;
      }
      for (int o = 16; o >= w; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane < w) s_sl[wid][lane] = s;
    } else {
      float alpha, tq, sq;
      const float x0 = __ldcg(row + i);
      FF n{0.f, 0.f};
      for (int q = lane; q < P; q += 32 * 5) {
        float2 v[5];
#pragma unroll
        for (int u = 0; u < 5; u++) v[u] = (q + 32 * u < P) ? __ldcg(p.cn + q + 32 * u) : make_float2(0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 5; u++) n = ff_add(n, FF{v[u].x, v[u].y});
      }
      n = warp_sum_ff(n);
      householder_ff(x0, n, &alpha, &tq, &sq);
      if (lane == 0) {
        s_q[0] = tq;
        s_q[1] = sq;
        if (b == 0) {
          p.d[i] = alpha;
          p.tauq[i] = tq;
        }
      }
    }
    __syncthreads();
    const float tq = s_q[0], sq = s_q[1];
    if (wid == 0) {
      const int cl = lane & 15, h = lane >> 4;
      float s = 0.f;
      if (cl < nc) {
#pragma unroll
        for (int q = 0; q < kResWarps / 2; q++) s += s_sl[h * (kResWarps / 2) + q][cl];
      }
      s += __shfl_xor_sync(0xffffffffu, s, 16);
      FF n{0.f, 0.f};
      if (lane < nc) {
        const float y = tq * (wic + sq * s);
        p.y[c0 + lane] = y;
        if (c0 + lane > i + 1) n = ff_add_sq(n, wic - y);
      }
      n = warp_sum_ff(n);
      if (lane == 0) p.rn[b] = make_float2(n.hi, n.lo);
    } else if (wid == 1 && lane < R) {
      const int r = r0 + lane;
      const float u = s_x[lane] * sq;
      s_u[lane] = r > i ? u : 0.f;
      if (r >= i && r < mt) p.W[r + (size_t)i * ldw] = r > i ? u : 1.f;
    }
    if (!grid_sync(p.bar, P, p.st, 51)) return;
    // ---- 3. left update, products with the new row, right update
    if (main) {
      float z[B];
#pragma unroll
      for (int r = 0; r < B; r++) z[r] = 0.f;
      float y[K], v[K];
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int c = t + k * kResThreads;
        y[k] = (c > i && c < nt) ? __ldcg(p.y + c) : 0.f;
        rw[k] -= y[k];  // the new row
        v[k] = c > i + 1 ? rw[k] : 0.f;
      }
#pragma unroll
      for (int r = 0; r < R; r += 4) {
        const float4 uv = *reinterpret_cast<const float4*>(s_u + r);
        const float u4[4] = {uv.x, uv.y, uv.z, uv.w};
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
          for (int k = 0; k < K; k++) {
            a[r + q][k] -= u4[q] * y[k];
            z[r + q] += a[r + q][k] * v[k];
          }
      }
#pragma unroll
      for (int k = 0; k < K; k++)
        if (t + k * kResThreads == i + 1) {
#pragma unroll
          for (int r = 0; r < R; r++) s_c1[r] = a[r][k];
        }
      const float zs = warp_reduce_scatter<B>(z, lane);
      constexpr int G = 32 / B;
      if (lane % G == 0) s_red[wid][lane / G] = zs;
    } else {
      float beta, tp, sp;
      const float x0 = __ldcg(row + i + 1) - __ldcg(p.y + i + 1);
      FF n{0.f, 0.f};
      for (int q = lane; q < P; q += 32 * 5) {
        float2 v[5];
#pragma unroll
        for (int u = 0; u < 5; u++) v[u] = (q + 32 * u < P) ? __ldcg(p.rn + q + 32 * u) : make_float2(0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 5; u++) n = ff_add(n, FF{v[u].x, v[u].y});
      }
      n = warp_sum_ff(n);
      householder_ff(x0, n, &beta, &tp, &sp);
      if (lane == 0) {
        s_p[0] = tp;
        s_p[1] = sp;
        if (b == 0) {
          p.e[i] = beta;
          p.taup[i] = tp;
        }
      }
    }
    __syncthreads();
    const float tp = s_p[0], sp = s_p[1];
    if (wid < R) {  // one warp per row finishes its product
      float s = lane < kResWarps ? s_red[lane][wid] : 0.f;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) s_z[wid] = (r0 + wid > i) ? tp * (s_c1[wid] + sp * s) : 0.f;
    }
    __syncthreads();
    if (main) {
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int c = t + k * kResThreads;
        rw[k] = c > i + 1 ? rw[k] * sp : (c == i + 1 && tp != 0.f) ? 1.f : 0.f;  // v
        if (own && c > i && c < nt) p.W[i + (size_t)c * ldw] = rw[k];
      }
#pragma unroll
      for (int r = 0; r < R; r += 4) {
        const float4 zv = *reinterpret_cast<const float4*>(s_z + r);
        const float z4[4] = {zv.x, zv.y, zv.z, zv.w};
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
          for (int k = 0; k < K; k++) a[r + q][k] -= z4[q] * rw[k];
      }
#pragma unroll
      for (int k = 0; k < K; k++)
        if (t + k * kResThreads == i + 1) {
#pragma unroll
          for (int r = 0; r < R; r++) s_x[r] = a[r][k];
        }
    }
    __syncthreads();
  }
  if (main) {
#pragma unroll
    for (int k = 0; k < K; k++) {
      const int c = t + k * kResThreads;
      if (c >= p.cols && c < nt) {
#pragma unroll
        for (int r = 0; r < R; r++)
          if (r0 + r >= p.cols && r0 + r < mt) p.W[r0 + r + (size_t)c * ldw] = a[r][k];
      }
    }
  }
}

using ResKernel = void (*)(ResParams);
struct ResConfig {
  int R, K;
  ResKernel fn;
};
// smallest first
const ResConfig kResConfigs[] = {{8, 2, bidiag_resident_kernel<8, 2>},   {12, 2, bidiag_resident_kernel<12, 2>},
                                 {16, 2, bidiag_resident_kernel<16, 2>}, {8, 4, bidiag_resident_kernel<8, 4>},
                                 {12, 4, bidiag_resident_kernel<12, 4>}, {16, 4, bidiag_resident_kernel<16, 4>}};

const ResConfig* res_config(int mt, int nt, int P) {
  for (const ResConfig& g : kResConfigs)
    if ((long long)g.R * P >= mt && g.K * kResThreads >= nt && nt <= kResSlice * P) return &g;
  return nullptr;
}

}  // namespace

// Runs down to the first panel boundary that the tail takes over from, or to one
// where a configuration with fewer registers holds the rest (each launch loads
// and stores the block once, ~20 us; a pass over half of it saves ~0.2 us a
// column).
int bidiag_resident_columns(ddcsvd_context* ctx, int m, int n, int k0, int P) {
  if (m - k0 < n - k0 || bidiag_tail_columns(ctx, m, n, k0) > 0) return 0;
  const ResConfig* g = res_config(m - k0, n - k0, P);
  if (!g || ctx->tune[TK_PANEL_TAIL] <= 0) return 0;
  bool tail = false;  // does the tail take over before the end?
  int cols = 0;
  for (int k1 = k0 + kPanel; n - k1 > 1 && !tail; k1 += kPanel) {
    tail = bidiag_tail_columns(ctx, m, n, k1) > 0;
    if (cols == 0 && (tail || (k1 - k0 >= 4 * kPanel && res_config(m - k1, n - k1, P) != g))) cols = k1 - k0;
  }
  return tail ? cols : 0;
}

int bidiag_resident(ddcsvd_context* ctx, int m, int n, int k0, int cols, float* W, int ldw, float* d, float* e,
                    float* tauq, float* taup, const BidiagWork& w) {
  const ResConfig* g = res_config(m - k0, n - k0, w.P);
  if (!g || !w.xpart) return DDCSVD_ERR_UNSUPPORTED;
  ResParams p;
  p.mt = m - k0;
  p.nt = n - k0;
  p.cols = cols;
  p.ldw = ldw;
  p.ldp = w.ldxp;
  p.ldr = w.ldn;
  p.W = W + k0 + (size_t)k0 * ldw;
  p.d = d + k0;
  p.e = e + k0;
  p.tauq = tauq + k0;
  p.taup = taup + k0;
  p.part = w.xpart;  // the panels' buffers: none is in use between panels
  p.y = w.Y;
  p.row = w.VT;
  p.cn = reinterpret_cast<float2*>(w.colpart);
  p.rn = reinterpret_cast<float2*>(w.rowpart);
  p.bar = w.bar;
  p.st = ctx->d_status;
  DDC_CUDA_TRY(cudaMemsetAsync(w.bar, 0, sizeof(GridBarrier), ctx->stream));
  void* args[] = {&p};
  DDC_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)g->fn, dim3(w.P), dim3(kResThreads + 32), args, 0,
                                           ctx->stream));
  count_launch();
  return DDCSVD_OK;
}

}  // namespace ddcsvd
