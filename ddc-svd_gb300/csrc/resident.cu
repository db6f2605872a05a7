// resident.cu -- the columns of the blocked bidiagonalisation between the panels
// and the cluster tail, the trailing block on chip in the whole grid.
//
// Once the trailing block fits the register files and shared memory (3648 rows
// and columns on 152 SMs), the unblocked algorithm of the tail (tail.cu; reflector
// conventions, compensated FP32 norms and storage are the same) runs on one
// persistent cooperative grid.  CTA b holds the R rows from b R on.  The last K T
// columns are in registers, T threads with column S + t, S + t + T, ... each; the
// first S, which retire first, are in shared memory.  Either way a thread has all
// R entries of its columns, so the products of a column with the others are sums
// inside a thread, and the right update's row sums one reduce-scatter per warp.
// Per column i, with x its entries below row i:
//   1. each CTA writes its part of x^T A and of ||x||^2; the owner of row i writes
//      that row (all from the sweep that ends the column before);
//   2. after a grid barrier each CTA adds the P parts of its slice of the columns
//      (every CTA forms the same reflector from the P norms in a warp of its own),
//      and writes tau y of the slice and its part of ||w||^2, w the new row i;
//   3. after a second barrier every CTA reads y and sweeps its columns twice: left
//      update and products with w (the reflector of w follows in the extra warp
//      meanwhile), then right update and products with column i + 1, which the
//      row sums already determine.
//
// What bounds it: the two barriers (1.3 us each) and the two round trips to L2
// behind them; the arithmetic is 4 multiply-adds an entry, and the columns in
// shared memory pass through its port four times.  The panel kernel reads the
// trailing block from L2 for every column, sums 152 records of 2 j values twice
// and one 152-part row product, and its trailing update comes on top.
// @@
#include "internal.hpp"

namespace ddcsvd {

namespace {

constexpr int kResSlice = 32;  // most columns of a CTA's slice

struct ResParams {
  int mt, nt, cols;  // trailing block and the columns to take
  int S;             // columns in shared memory
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

// entry q of a float4 held in registers (q a constant after unrolling)
__device__ __forceinline__ float el(const float4& v, int q) { return q == 0 ? v.x : q == 1 ? v.y : q == 2 ? v.z : v.w; }

// the sum of P compensated records in one warp
__device__ __forceinline__ FF sum_records(const float2* rec, int P, int lane) {
  FF n{0.f, 0.f};
  for (int q = lane; q < P; q += 32 * 5) {
    float2 v[5];
#pragma unroll
    for (int u = 0; u < 5; u++) v[u] = (q + 32 * u < P) ? __ldcg(rec + q + 32 * u) : make_float2(0.f, 0.f);
#pragma unroll
    for (int u = 0; u < 5; u++) n = ff_add(n, FF{v[u].x, v[u].y});
  }
  return warp_sum_ff(n);
}

// T threads hold the block, one more warp forms the norms.
template <int R, int K, int T>
__global__ void __launch_bounds__(T + 32, 1) bidiag_resident_kernel(ResParams p) {
  constexpr int W = T / 32, R4 = R / 4;
  constexpr int B = R > 16 ? 32 : R > 8 ? 16 : 8;  // rows of the reduce-scatter
  constexpr int U = T > 256 ? 6 : 11;              // slice loads in flight per thread
  static_assert(R % 4 == 0 && R <= 32, "rows come in float4s");
  extern __shared__ __align__(16) float4 s_a[];                 // [R4][S], then S floats: w of these columns
  __shared__ __align__(16) float s_x[R], s_u[R], s_z[R];        // own rows of x, u and of the right update
  __shared__ float s_c1[R], s_red[W][B], s_sl[W][kResSlice], s_q[2], s_p[2];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5, b = blockIdx.x, P = gridDim.x;
  const bool main = t < T;
  const int mt = p.mt, nt = p.nt, S = p.S, r0 = b * R, ldw = p.ldw;
  float* s_w = reinterpret_cast<float*>(s_a + (size_t)R4 * S);
  float a[R][K];
  auto load4 = [&](int c, int r) {  // rows r0 + r .. + 3 of column c (the last ones may be padding: ldw is a multiple of 4)
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < nt && r0 + r < mt) {
      v = __ldcg(reinterpret_cast<const float4*>(p.W + r0 + r + (size_t)c * ldw));
      if (r0 + r + 1 >= mt) v.y = 0.f;
      if (r0 + r + 2 >= mt) v.z = 0.f;
      if (r0 + r + 3 >= mt) v.w = 0.f;
    }
    return v;
  };
  if (main) {
    for (int c = t; c < S; c += T)
#pragma unroll
      for (int q = 0; q < R4; q++) s_a[q * S + c] = load4(c, 4 * q);
#pragma unroll
    for (int k = 0; k < K; k++)
#pragma unroll
      for (int q = 0; q < R4; q++) {
        const float4 v = load4(S + t + k * T, 4 * q);
        a[4 * q][k] = v.x; a[4 * q + 1][k] = v.y; a[4 * q + 2][k] = v.z; a[4 * q + 3][k] = v.w;
      }
  } else if (lane < R4) {
    *reinterpret_cast<float4*>(s_x + 4 * lane) = load4(0, 4 * lane);
    *reinterpret_cast<float4*>(s_z + 4 * lane) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (t == 0) s_p[0] = s_p[1] = 0.f;
  __syncthreads();
  float rw[K];
#pragma unroll
  for (int k = 0; k < K; k++) rw[k] = 0.f;
  for (int c = t; main && c < S; c += T) s_w[c] = 0.f;
  // i = -1: only the second sweep (nothing to update), for column 0
  for (int i = -1; i < p.cols; i++) {
    const bool own = i >= r0 && i < r0 + R;  // row i is here
    if (i >= 0) {
      float* row = p.row + (i & 1) * p.ldr;
      if (!grid_sync(p.bar, P, p.st, 50)) return;
      // ---- left reflector; tau y and the new row on the CTA's slice of the columns
      const int ncol = nt - (i + 1), cc = (ncol + P - 1) / P;  // (at most kResSlice: the host's choice of shapes)
      const int c0 = i + 1 + b * cc, nc = max(0, min(cc, nt - c0));
      const int lg = cc > 16 ? 5 : cc > 8 ? 4 : cc > 4 ? 3 : 2, w = 1 << lg;  // lanes per record
      float wic = 0.f;
      if (main) {
        const int cl = t & (w - 1), nrec = T >> lg;
        if (wid == 0 && lane < nc) wic = __ldcg(row + c0 + lane);
        float s = 0.f;
        for (int q = t >> lg; q < P; q += U * nrec) {
          float v[U];
#pragma unroll
          for (int u = 0; u < U; u++)
            v[u] = (cl < nc && q + u * nrec < P) ? __ldcg(p.part + (size_t)(q + u * nrec) * p.ldp + c0 + cl) : 0.f;
#pragma unroll
          for (int u = 0; u < U; u++) s += v[u];
        }
        for (int o = 16; o >= w; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane < w) s_sl[wid][lane] = s;
      } else {
        float alpha, tq, sq;
        const float x0 = __ldcg(row + i);
        householder_ff(x0, sum_records(p.cn, P, lane), &alpha, &tq, &sq);
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
        // the warps' sums: two lanes per column share them while a slice has at most 16
        constexpr int H = (W + 1) / 2;
        const int cl = lg == 5 ? lane : lane & 15, q0 = lg == 5 || lane < 16 ? 0 : H;
        float s = 0.f;
#pragma unroll
        for (int q = 0; q < H; q++) s += (cl < nc && q0 + q < W) ? s_sl[q0 + q][cl] : 0.f;
        if (lg == 5) {
#pragma unroll
          for (int q = H; q < W; q++) s += cl < nc ? s_sl[q][cl] : 0.f;
        } else {
          s += __shfl_xor_sync(0xffffffffu, s, 16);
        }
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
      // ---- left update and products with the new row
      if (main) {
        float z[B];
#pragma unroll
        for (int r = 0; r < B; r++) z[r] = 0.f;
        float y[K], v[K];
#pragma unroll
        for (int k = 0; k < K; k++) {
          const int c = S + t + k * T;
          const bool in = c > i && c < nt;
          y[k] = in ? __ldcg(p.y + c) : 0.f;
          rw[k] = in ? __ldcg(row + c) : 0.f;
        }
        // (columns in shared memory: the next one's y and w are on their way while one is swept)
        int c = t + (t <= i ? (i - t + T) / T * T : 0);  // the thread's first column beyond i
        float yn = c < S ? __ldcg(p.y + c) : 0.f, wn = c < S ? __ldcg(row + c) : 0.f;
        for (; c < S; c += T) {
          const float yc = yn, wc = wn - yc;
          if (c + T < S) {
            yn = __ldcg(p.y + c + T);
            wn = __ldcg(row + c + T);
          }
          const float vc = c > i + 1 ? wc : 0.f;
          s_w[c] = wc;
#pragma unroll
          for (int q = 0; q < R4; q++) {
            const float4 uv = *reinterpret_cast<const float4*>(s_u + 4 * q);
            float4 av = s_a[q * S + c];
            av.x -= uv.x * yc; av.y -= uv.y * yc; av.z -= uv.z * yc; av.w -= uv.w * yc;
            z[4 * q] += av.x * vc; z[4 * q + 1] += av.y * vc; z[4 * q + 2] += av.z * vc; z[4 * q + 3] += av.w * vc;
            s_a[q * S + c] = av;
            if (c == i + 1) {
              s_c1[4 * q] = av.x; s_c1[4 * q + 1] = av.y; s_c1[4 * q + 2] = av.z; s_c1[4 * q + 3] = av.w;
            }
          }
        }
#pragma unroll
        for (int k = 0; k < K; k++) {
          rw[k] -= y[k];  // the new row
          v[k] = S + t + k * T > i + 1 ? rw[k] : 0.f;
        }
#pragma unroll
        for (int q = 0; q < R4; q++) {
          const float4 uv = *reinterpret_cast<const float4*>(s_u + 4 * q);
#pragma unroll
          for (int h = 0; h < 4; h++)
#pragma unroll
            for (int k = 0; k < K; k++) {
              a[4 * q + h][k] -= el(uv, h) * y[k];
              z[4 * q + h] += a[4 * q + h][k] * v[k];
            }
        }
#pragma unroll
        for (int k = 0; k < K; k++)
          if (S + t + k * T == i + 1) {
#pragma unroll
            for (int r = 0; r < R; r++) s_c1[r] = a[r][k];
          }
        const float zs = warp_reduce_scatter<B>(z, lane);
        constexpr int G = 32 / B;
        if (lane % G == 0) s_red[wid][lane / G] = zs;
      } else {
        float beta, tp, sp;
        const float x0 = __ldcg(row + i + 1) - __ldcg(p.y + i + 1);
        householder_ff(x0, sum_records(p.rn, P, lane), &beta, &tp, &sp);
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
      {  // one warp per row finishes its product; column i + 1 follows from it
        const float tp = s_p[0], sp = s_p[1];
        for (int r = wid; r < R; r += W + 1) {
          float s = lane < W ? s_red[lane][r] : 0.f;
#pragma unroll
          for (int o = W > 8 ? 8 : 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
          if (lane == 0) {
            const float z = (r0 + r > i) ? tp * (s_c1[r] + sp * s) : 0.f;
            s_z[r] = z;
            s_x[r] = tp != 0.f ? s_c1[r] - z : s_c1[r];
          }
        }
      }
      __syncthreads();
    }
    // ---- right update, and for column i + 1 the parts of x^T A and ||x||^2 and row i + 1
    const float tp = s_p[0], sp = s_p[1];
    const int i1 = i + 1;
    const bool more = i1 < p.cols;
    float* row1 = p.row + (i1 & 1) * p.ldr;
    float* part = p.part + (size_t)b * p.ldp;
    const bool own1 = more && i1 >= r0 && i1 < r0 + R;
    if (main) {
      for (int c = t; c < S; c += T) {
        if (c <= i) continue;
        const float vc = c > i1 ? s_w[c] * sp : tp != 0.f ? 1.f : 0.f;
        if (own) p.W[i + (size_t)c * ldw] = vc;
        float s = 0.f;
#pragma unroll
        for (int q = 0; q < R4; q++) {
          const float4 zv = *reinterpret_cast<const float4*>(s_z + 4 * q);
          const float4 xv = *reinterpret_cast<const float4*>(s_x + 4 * q);
          float4 av = s_a[q * S + c];
          av.x -= zv.x * vc; av.y -= zv.y * vc; av.z -= zv.z * vc; av.w -= zv.w * vc;
          s_a[q * S + c] = av;
#pragma unroll
          for (int h = 0; h < 4; h++) s += (r0 + 4 * q + h > i1) ? el(av, h) * el(xv, h) : 0.f;
        }
        if (more && c > i1) part[c] = s;
        if (own1) row1[c] = reinterpret_cast<const float*>(s_a + ((i1 - r0) >> 2) * S + c)[(i1 - r0) & 3];
      }
      float s[K];
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int c = S + t + k * T;
        rw[k] = c > i1 ? rw[k] * sp : (c == i1 && tp != 0.f) ? 1.f : 0.f;  // v
        if (own && c > i && c < nt) p.W[i + (size_t)c * ldw] = rw[k];
        s[k] = 0.f;
      }
#pragma unroll
      for (int q = 0; q < R4; q++) {
        const float4 zv = *reinterpret_cast<const float4*>(s_z + 4 * q);
        const float4 xv = *reinterpret_cast<const float4*>(s_x + 4 * q);
#pragma unroll
        for (int h = 0; h < 4; h++) {
          const float x = (r0 + 4 * q + h > i1) ? el(xv, h) : 0.f;
#pragma unroll
          for (int k = 0; k < K; k++) {
            a[4 * q + h][k] -= el(zv, h) * rw[k];
            s[k] += a[4 * q + h][k] * x;
          }
        }
      }
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int c = S + t + k * T;
        if (more && c > i1 && c < nt) part[c] = s[k];
      }
      if (own1) {
#pragma unroll
        for (int r = 0; r < R; r++)
          if (r0 + r == i1) {
#pragma unroll
            for (int k = 0; k < K; k++) {
              const int c = S + t + k * T;
              if (c >= i1 && c < nt) row1[c] = a[r][k];
            }
          }
      }
    } else if (more) {
      FF n{0.f, 0.f};
      if (lane < R && r0 + lane > i1) n = ff_add_sq(n, s_x[lane]);
      n = warp_sum_ff(n);
      if (lane == 0) p.cn[b] = make_float2(n.hi, n.lo);
    }
  }
  // ---- the rest back (the columns taken are stored already)
  if (main) {
    for (int c = t; c < S; c += T) {
      if (c < p.cols) continue;
      for (int r = 0; r < R; r++)
        if (r0 + r >= p.cols && r0 + r < mt)
          p.W[r0 + r + (size_t)c * ldw] = reinterpret_cast<const float*>(s_a + (r >> 2) * S + c)[r & 3];
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      const int c = S + t + k * T;
      if (c >= p.cols && c < nt) {
#pragma unroll
        for (int r = 0; r < R; r++)
          if (r0 + r >= p.cols && r0 + r < mt) p.W[r0 + r + (size_t)c * ldw] = a[r][k];
      }
    }
  }
}

struct ResConfig {
  int R, K, T;
  const void* fn;
};
template <int R, int K, int T>
ResConfig res_entry() {
  return {R, K, T, (const void*)bidiag_resident_kernel<R, K, T>};
}

size_t res_smem(const ResConfig& g, int nt) {
  return (size_t)std::max(0, nt - g.K * g.T) * (g.R + 1) * sizeof(float);
}

// The smallest configuration that has the rows and keeps all but a few columns in
// registers, else the largest with the rest of them in shared memory.  Up to 16
// rows run on 15 + 1 warps (128 registers a thread; 16 + 1 leave 96, and 16 x 4
// entries then spill: 2048^2 12.0 ms against 11.3), 24 on 7 + 1 (255).
const ResConfig* res_config(int mt, int nt, int P, size_t smem_max) {
  static const ResConfig tab[] = {res_entry<8, 2, 480>(),  res_entry<8, 3, 480>(),  res_entry<8, 4, 480>(),
                                  res_entry<12, 2, 480>(), res_entry<12, 3, 480>(), res_entry<12, 4, 480>(),
                                  res_entry<16, 2, 480>(), res_entry<16, 3, 480>(), res_entry<16, 4, 480>(),
                                  res_entry<24, 7, 224>()};
  for (const ResConfig& g : tab)
    if ((long long)g.R * P >= mt && nt <= kResSlice * P && res_smem(g, nt) <= smem_max &&
        (g.K < 4 ? nt <= g.K * g.T + 64 : true))
      return &g;
  return nullptr;
}

size_t res_smem_max(const ddcsvd_context* ctx) { return ctx->smem_optin > 8192 ? ctx->smem_optin - 8192 : 0; }

}  // namespace

// Runs down to the first panel boundary that the tail takes over from, or to one
// where a configuration with fewer registers holds the rest (each launch loads
// and stores the block once, ~20 us; a smaller configuration saves 0.2 us or more
// a column).
int bidiag_resident_columns(ddcsvd_context* ctx, int m, int n, int k0, int P) {
  if (ctx->tune[TK_PANEL_TAIL] <= 0 || bidiag_tail_columns(ctx, m, n, k0) > 0) return 0;
  const size_t sm = res_smem_max(ctx);
  const ResConfig* g = res_config(m - k0, n - k0, P, sm);
  if (!g) return 0;
  bool tail = false;  // does the tail take over before the end?
  int cols = 0;
  for (int k1 = k0 + kPanel; n - k1 > 1 && !tail; k1 += kPanel) {
    tail = bidiag_tail_columns(ctx, m, n, k1) > 0;
    if (cols == 0 && (tail || (k1 - k0 >= 4 * kPanel && res_config(m - k1, n - k1, P, sm) != g))) cols = k1 - k0;
  }
  return tail ? cols : 0;
}

int bidiag_resident(ddcsvd_context* ctx, int m, int n, int k0, int cols, float* W, int ldw, float* d, float* e,
                    float* tauq, float* taup, const BidiagWork& w) {
  const ResConfig* g = res_config(m - k0, n - k0, w.P, res_smem_max(ctx));
  if (!g || !w.xpart) return DDCSVD_ERR_UNSUPPORTED;
  ResParams p;
  p.mt = m - k0;
  p.nt = n - k0;
  p.cols = cols;
  p.S = std::max(0, p.nt - g->K * g->T);
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
  const size_t smem = res_smem(*g, p.nt);
  DDC_CUDA_TRY(cudaFuncSetAttribute(g->fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  DDC_CUDA_TRY(cudaMemsetAsync(w.bar, 0, sizeof(GridBarrier), ctx->stream));
  void* args[] = {&p};
  DDC_CUDA_TRY(cudaLaunchCooperativeKernel(g->fn, dim3(w.P), dim3(g->T + 32), args, smem, ctx->stream));
  count_launch();
  return DDCSVD_OK;
}

}  // namespace ddcsvd
