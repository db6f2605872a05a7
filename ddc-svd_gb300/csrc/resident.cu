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
//   2. each CTA adds the P parts of its slice of the columns (every CTA forms the
//      same reflector from the P norms in a warp of its own), and writes tau y of
//      the slice and its part of ||w||^2, w the new row i;
//   3. every CTA reads y and sweeps its columns twice: left update and products
//      with w (the reflector of w follows in the extra warp meanwhile), then right
//      update and products with column i + 1, which the row sums already determine.
//
// What bounds it: the two exchanges of a column and the compensated norms behind
// them; the arithmetic is 4 multiply-adds an entry, and the columns in shared
// memory pass through its port three times.  The panel kernel reads the trailing
// block from L2 for every column, sums 152 records of 2 j values twice and one
// 152-part row product, and its trailing update comes on top.  Us per column,
// panels and here: 512-1024 columns 11.3 and 4.0, 1024-2048 13 to 15 and 4.9,
// 2048-3648 15 to 18 and 6 (16 rows per CTA) to 12 (20 and 24, with grid barriers).
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
  unsigned tag0;  // tag of the first column
  // exchanged words (value, tag of the column)
  uint2* part;      // P x ldp: x^T A by CTA
  uint2* y;         // tau y
  uint2* row;       // 2 x ldr: row i, by column parity
  uint2 *cn, *rn;   // P x 2: compensated parts of ||x||^2 and ||w||^2
  GridBarrier* bar;
  DevStatus* st;
};

// Exchanged words carry their column's tag beside the value: one 8-byte store
// publishes both, and a reader polls until the tag is there.  No word is
// overwritten before its readers are through:
//  * parts, norms cn and row of column i + 1 are written after their CTA has read
//    the norms rn of column i from every CTA, and a CTA writes its rn after it has
//    read the parts, cn and its slice of the row of column i;
//  * y and rn of column i + 1 are written after their CTA has read cn of column
//    i + 1 from every CTA, and a CTA writes its cn after it has read y, rn and the
//    row of column i;
//  * the row of column i may still be read while its successor is written: one
//    buffer per parity.
__device__ __forceinline__ void put(uint2* w, float v, unsigned tag) {
  const unsigned long long x = __float_as_uint(v) | ((unsigned long long)tag << 32);
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(w), "l"(x) : "memory");
}
__device__ __forceinline__ uint2 get(const uint2* w) {
  unsigned long long x;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(x) : "l"(w) : "memory");
  return make_uint2((unsigned)x, (unsigned)(x >> 32));
}
// One unsuccessful poll: false when the wait is over (another CTA's error, or the limit).
struct Waiter {
  DevStatus* st;
  unsigned polls = 0;
  unsigned long long t0 = 0;
  __device__ __forceinline__ bool again() {
    if ((++polls & 31u) != 0) return true;
    const uint4 s = ld_status(st);
    if (s.x != 0) return false;
    const unsigned long long now = global_ns();
    if (t0 == 0) t0 = now;
    if (now - t0 <= (s.z ? 1000ull * s.z : kWaitLimitNs)) return true;
    set_error(st, DDCSVD_ERR_TIMEOUT, 50);
    return false;
  }
};
// Reads the words at(0..N-1) that `want` asks for (others: zero); those missing are
// polled together.  False: gave up.
// Without kTag a grid barrier has ordered the words already, and their values are
// read alone.
template <bool kTag, int N, class At, class Want>
__device__ __forceinline__ bool take(float (&v)[N], unsigned tag, Waiter& wt, At at, Want want) {
  if constexpr (!kTag) {
#pragma unroll
    for (int u = 0; u < N; u++) v[u] = want(u) ? __ldcg(reinterpret_cast<const float*>(at(u))) : 0.f;
  } else {
    uint2 w[N];
#pragma unroll
    for (int u = 0; u < N; u++) w[u] = make_uint2(0u, want(u) ? tag - 1u : tag);
    while (true) {
      bool all = true;
#pragma unroll
      for (int u = 0; u < N; u++)
        if (w[u].y != tag) w[u] = get(at(u));
#pragma unroll
      for (int u = 0; u < N; u++) all = all && w[u].y == tag;
      if (all) break;
      if (!wt.again()) return false;
    }
#pragma unroll
    for (int u = 0; u < N; u++) v[u] = __uint_as_float(w[u].x);
  }
  return true;
}

// entry q of a float4 held in registers (q a constant after unrolling)
__device__ __forceinline__ float el(const float4& v, int q) { return q == 0 ? v.x : q == 1 ? v.y : q == 2 ? v.z : v.w; }

// the sum of P compensated records (two words each) in one warp
template <bool kTag>
__device__ __forceinline__ FF sum_records(const uint2* rec, int P, unsigned tag, int lane, Waiter& wt, bool& ok) {
  FF n{0.f, 0.f};
  for (int q = lane; q < P; q += 32 * 5) {
    float v[10];
    ok = take<kTag, 10>(v, tag, wt, [&](int u) { return rec + 2 * (q + 32 * (u >> 1)) + (u & 1); },
                  [&](int u) { return q + 32 * (u >> 1) < P; }) && ok;
#pragma unroll
    for (int u = 0; u < 5; u++) n = ff_add(n, FF{v[2 * u], v[2 * u + 1]});
  }
  __syncwarp();
  return warp_sum_ff(n);
}

// T threads hold the block, one more warp forms the norms.
template <int R, int K, int T>
__global__ void __launch_bounds__(T + 32, 1) bidiag_resident_kernel(ResParams p) {
  constexpr int W = T / 32, R4 = R / 4;
  constexpr int B = R > 16 ? 32 : R > 8 ? 16 : 8;  // rows of the reduce-scatter
  constexpr int NG = R > 16 ? 3 : 2;               // columns in shared memory swept together
  constexpr int U = T > 256 ? 6 : 22;              // slice loads in flight per thread (24 rows: all of them)
  // 20 and 24 rows leave no registers to poll from: barriers there (3648^2: stage 1 26.0 ms
  // against 28.4 polling; with fewer rows 2048^2 takes 8.4 ms polling, 10.8 with
  // barriers)
  constexpr bool kTag = T > 256;
  static_assert(R % 4 == 0 && R <= 32, "rows come in float4s");
  extern __shared__ __align__(16) float4 s_a[];                 // [R4][S], then w and y of these columns
  __shared__ __align__(16) float s_x[R], s_u[R], s_z[R];        // own rows of x, u and of the right update
  __shared__ float s_c1[R], s_red[W][B], s_sl[W][kResSlice], s_q[2], s_p[2], s_row[kResSlice];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5, b = blockIdx.x, P = gridDim.x;
  const bool main = t < T;
  const int mt = p.mt, nt = p.nt, S = p.S, r0 = b * R, ldw = p.ldw;
  float *s_w = reinterpret_cast<float*>(s_a + (size_t)R4 * S), *s_y = s_w + S;
  // the handle's extra arrivals stand for a CTA whose norms never come (tests of the bounded waits)
  const bool lost = kTag && b == 0 && ld_status(p.st).w != 0;
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
    float4 x = load4(0, 4 * lane);
    if (b == 0 && lane == 0) x.x = 0.f;
    *reinterpret_cast<float4*>(s_x + 4 * lane) = x;
    *reinterpret_cast<float4*>(s_u + 4 * lane) = *reinterpret_cast<float4*>(s_z + 4 * lane) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (t == 0) s_p[0] = s_p[1] = 0.f;
  __syncthreads();
  float rw[K];
#pragma unroll
  for (int k = 0; k < K; k++) rw[k] = 0.f;
  for (int c = t; main && c < S; c += T) s_w[c] = s_y[c] = 0.f;
  // i = -1: only the second sweep (nothing to update), for column 0
  for (int i = -1; i < p.cols; i++) {
    if (i >= 0) {
      uint2* row = p.row + (i & 1) * p.ldr;
      const unsigned tag = p.tag0 + i;
      Waiter wt{p.st};
      bool ok = true;
      if (!kTag && !grid_sync(p.bar, P, p.st, 50)) return;
      // ---- left reflector; tau y and the new row on the CTA's slice of the columns
      const int ncol = nt - (i + 1), cc = (ncol + P - 1) / P;  // (at most kResSlice: the host's choice of shapes)
      const int c0 = i + 1 + b * cc, nc = max(0, min(cc, nt - c0));
      const int lg = cc > 16 ? 5 : cc > 8 ? 4 : cc > 4 ? 3 : 2, w = 1 << lg;  // lanes per record
      float wic = 0.f;
      if (main) {
        const int cl = t & (w - 1), nrec = T >> lg;
        float s = 0.f;
        for (int q = t >> lg; q < P; q += U * nrec) {
          float v[U];
          ok = take<kTag, U>(v, tag, wt, [&](int u) { return p.part + (size_t)(q + u * nrec) * p.ldp + c0 + cl; },
                       [&](int u) { return cl < nc && q + u * nrec < P; }) && ok;
#pragma unroll
          for (int u = 0; u < U; u++) s += v[u];
        }
        if (wid == 0) {
          float v[1];
          ok = take<kTag, 1>(v, tag, wt, [&](int) { return row + c0 + lane; }, [&](int) { return lane < nc; }) && ok;
          wic = v[0];
        }
        __syncwarp();
        for (int o = 16; o >= w; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane < w) s_sl[wid][lane] = s;
      } else {
        float alpha, tq, sq;
        float x0[1];
        const FF n2 = sum_records<kTag>(p.cn, P, tag, lane, wt, ok);
        ok = take<kTag, 1>(x0, tag, wt, [&](int) { return row + i; }, [](int) { return true; }) && ok;
        householder_ff(x0[0], n2, &alpha, &tq, &sq);
        if (lane == 0) {
          s_q[0] = tq;
          s_q[1] = sq;
          if (b == 0) {
            p.d[i] = alpha;
            p.tauq[i] = tq;
          }
        }
      }
      if (__syncthreads_or(!ok)) return;
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
          put(p.y + c0 + lane, y, tag);
          s_row[lane] = wic - y;
          if (c0 + lane > i + 1) n = ff_add_sq(n, wic - y);
        }
        n = warp_sum_ff(n);
        if (lane < 2) put(p.rn + 2 * b + lane, lane ? n.lo : n.hi, tag);
      } else if (wid == 1 && lane < R) {
        const int r = r0 + lane;
        const float u = s_x[lane] * sq;
        s_u[lane] = u;
        if (r >= i && r < mt) p.W[r + (size_t)i * ldw] = r > i ? u : 1.f;
      }
      if (!kTag) {
        if (!grid_sync(p.bar, P, p.st, 51)) return;
      } else {
        __syncthreads();  // s_u
      }
      // ---- left update and products with the new row
      if (main) {
        float z[B];
#pragma unroll
        for (int r = 0; r < B; r++) z[r] = 0.f;
        float y[K], v[K];
        const auto reg_at = [&](int k) { return S + t + k * T; };
        const auto reg_want = [&](int k) { return reg_at(k) > i && reg_at(k) < nt; };
        {
          float yw[2 * K];
          ok = take<kTag, 2 * K>(yw, tag, wt, [&](int u) { return (u < K ? p.y : row) + reg_at(u < K ? u : u - K); },
                           [&](int u) { return reg_want(u < K ? u : u - K); }) && ok;
#pragma unroll
          for (int k = 0; k < K; k++) {
            y[k] = yw[k];
            rw[k] = yw[K + k];
          }
        }
        // columns in shared memory: y and w of a few at a time
        constexpr int C = T > 256 ? 2 : 5;
        const int c1 = t + (t <= i ? (i - t + T) / T * T : 0);  // the thread's first column beyond i
        for (int c = c1; c < S; c += C * T) {
          float yw[2 * C];
          ok = take<kTag, 2 * C>(yw, tag, wt, [&](int u) { return (u < C ? p.y : row) + c + (u < C ? u : u - C) * T; },
                                 [&](int u) { return c + (u < C ? u : u - C) * T < S; }) && ok;
#pragma unroll
          for (int u = 0; u < C; u++)
            if (c + u * T < S) {
              s_y[c + u * T] = yw[u];
              s_w[c + u * T] = yw[C + u] - yw[u];
            }
        }
        // (NG columns at a time share the reads of u; the updated entries are not
        // written here but formed again in the second sweep: a read and a write
        // less of the port that bounds both)
        for (int c = c1; c < S; c += NG * T) {
          float yc[NG], vc[NG];
          const float4* col[NG];  // (beyond S: the first column again, times zero)
#pragma unroll
          for (int g = 0; g < NG; g++) {
            const int cg = c + g * T;
            const bool in = cg < S;
            yc[g] = in ? s_y[cg] : 0.f;
            vc[g] = in && cg > i + 1 ? s_w[cg] : 0.f;
            col[g] = s_a + (in ? cg : c);
          }
#pragma unroll
          for (int q = 0; q < R4; q++) {
            const float4 uv = *reinterpret_cast<const float4*>(s_u + 4 * q);
#pragma unroll
            for (int g = 0; g < NG; g++) {
              float4 av = col[g][q * S];
              av.x -= uv.x * yc[g]; av.y -= uv.y * yc[g]; av.z -= uv.z * yc[g]; av.w -= uv.w * yc[g];
              z[4 * q] += av.x * vc[g]; z[4 * q + 1] += av.y * vc[g];
              z[4 * q + 2] += av.z * vc[g]; z[4 * q + 3] += av.w * vc[g];
            }
          }
        }
        if (i + 1 < S && c1 == i + 1) {  // column i + 1, updated on the left
          const float yc = s_y[i + 1];
#pragma unroll
          for (int q = 0; q < R4; q++) {
            const float4 uv = *reinterpret_cast<const float4*>(s_u + 4 * q), av = s_a[q * S + i + 1];
            s_c1[4 * q] = av.x - uv.x * yc; s_c1[4 * q + 1] = av.y - uv.y * yc;
            s_c1[4 * q + 2] = av.z - uv.z * yc; s_c1[4 * q + 3] = av.w - uv.w * yc;
          }
        }
        __syncwarp();
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
        float x0[2];
        // (y first: it comes earlier than the norms, and the wait for it keeps 152 warps
        // from polling the norms' words while they are written: 2048^2 9.8 -> 8.4 ms)
        ok = take<kTag, 2>(x0, tag, wt, [&](int u) { return (u ? p.y : row) + i + 1; }, [](int) { return true; }) && ok;
        const FF n2 = sum_records<kTag>(p.rn, P, tag, lane, wt, ok);
        householder_ff(x0[0] - x0[1], n2, &beta, &tp, &sp);
        if (lane == 0) {
          s_p[0] = tp;
          s_p[1] = sp;
          if (b == 0) {
            p.e[i] = beta;
            p.taup[i] = tp;
          }
        }
      }
      if (__syncthreads_or(!ok)) return;
      {  // one warp per row finishes its product; column i + 1 follows from it
        const float tp = s_p[0], sp = s_p[1];
        for (int r = wid; r < R; r += W + 1) {
          float s = lane < W ? s_red[lane][r] : 0.f;
#pragma unroll
          for (int o = W > 8 ? 8 : 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
          if (lane == 0) {
            const float z = (r0 + r > i) ? tp * (s_c1[r] + sp * s) : 0.f;
            s_z[r] = z;
            s_x[r] = (r0 + r > i + 1) ? (tp != 0.f ? s_c1[r] - z : s_c1[r]) : 0.f;  // (rows below i + 1)
          }
        }
      }
      __syncthreads();
    }
    // ---- right update, and for column i + 1 the parts of x^T A and ||x||^2 and row i + 1
    const float tp = s_p[0], sp = s_p[1];
    const int i1 = i + 1;
    const bool more = i1 < p.cols;
    uint2* row1 = p.row + (i1 & 1) * p.ldr;
    uint2* part = p.part + (size_t)b * p.ldp;
    const unsigned tag1 = p.tag0 + i1;
    const bool own1 = more && i1 >= r0 && i1 < r0 + R;
    if (main) {
      for (int c = t + (t <= i ? (i - t + T) / T * T : 0); c < S; c += NG * T) {
        float vc[NG], yc[NG], s[NG];
        float4* col[NG];
#pragma unroll
        for (int g = 0; g < NG; g++) {
          const int cg = c + g * T;
          const bool in = cg < S;
          vc[g] = in && cg > i1 ? s_w[cg] * sp : tp != 0.f ? 1.f : 0.f;
          yc[g] = in ? s_y[cg] : 0.f;
          s[g] = 0.f;
          col[g] = s_a + (in ? cg : c);
        }
#pragma unroll
        for (int q = 0; q < R4; q++) {
          const float4 uv = *reinterpret_cast<const float4*>(s_u + 4 * q);
          const float4 zv = *reinterpret_cast<const float4*>(s_z + 4 * q);
          const float4 xv = *reinterpret_cast<const float4*>(s_x + 4 * q);
#pragma unroll
          for (int g = 0; g < NG; g++) {
            float4 av = col[g][q * S];
            av.x -= uv.x * yc[g]; av.y -= uv.y * yc[g]; av.z -= uv.z * yc[g]; av.w -= uv.w * yc[g];
            av.x -= zv.x * vc[g]; av.y -= zv.y * vc[g]; av.z -= zv.z * vc[g]; av.w -= zv.w * vc[g];
            if (c + g * T < S) col[g][q * S] = av;
            s[g] += av.x * xv.x + av.y * xv.y + av.z * xv.z + av.w * xv.w;
          }
        }
#pragma unroll
        for (int g = 0; g < NG; g++) {
          const int cg = c + g * T;
          if (!more || cg >= S) continue;
          if (cg > i1) put(part + cg, s[g], tag1);
          if (own1)
            put(row1 + cg, reinterpret_cast<const float*>(s_a + ((i1 - r0) >> 2) * S + cg)[(i1 - r0) & 3], tag1);
        }
      }
      float s[K];
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int c = S + t + k * T;
        rw[k] = c > i1 ? rw[k] * sp : (c == i1 && tp != 0.f) ? 1.f : 0.f;  // v
        s[k] = 0.f;
      }
#pragma unroll
      for (int q = 0; q < R4; q++) {
        const float4 zv = *reinterpret_cast<const float4*>(s_z + 4 * q);
        const float4 xv = *reinterpret_cast<const float4*>(s_x + 4 * q);
#pragma unroll
        for (int h = 0; h < 4; h++) {
#pragma unroll
          for (int k = 0; k < K; k++) {
            a[4 * q + h][k] -= el(zv, h) * rw[k];
            s[k] += a[4 * q + h][k] * el(xv, h);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int c = S + t + k * T;
        if (more && c > i1 && c < nt) put(part + c, s[k], tag1);
      }
      if (own1) {
#pragma unroll
        for (int r = 0; r < R; r++)
          if (r0 + r == i1) {
#pragma unroll
            for (int k = 0; k < K; k++) {
              const int c = S + t + k * T;
              if (c >= i1 && c < nt) put(row1 + c, a[r][k], tag1);
            }
          }
      }
      if (wid == 1 && i >= 0) {  // the slice's part of the right reflector into row i
        const int cc = (nt - i1 + P - 1) / P, c = i1 + b * cc + lane;
        if (lane < cc && c < nt) p.W[i + (size_t)c * ldw] = c > i1 ? s_row[lane] * sp : tp != 0.f ? 1.f : 0.f;
      }
    } else if (more) {
      FF n{0.f, 0.f};
      if (lane < R) n = ff_add_sq(n, s_x[lane]);
      n = warp_sum_ff(n);
      if (lane < 2 && !lost) put(p.cn + 2 * b + lane, lane ? n.lo : n.hi, tag1);
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
  return (size_t)std::max(0, nt - g.K * g.T) * (g.R + 2) * sizeof(float);
}

// The smallest configuration that has the rows and keeps all but a few columns in
// registers, else the largest with the rest of them in shared memory.  Up to 16
// rows run on 15 + 1 warps (128 registers a thread; 16 + 1 leave 96, and 16 x 4
// entries then spill: 2048^2 12.0 ms against 11.3), 20 and 24 on 7 + 1 (255;
// 2900^2 16.6 ms with 24 alone, 16.1 with 20 before it).
const ResConfig* res_config(int mt, int nt, int P, size_t smem_max) {
  static const ResConfig tab[] = {res_entry<8, 2, 480>(),  res_entry<8, 3, 480>(),  res_entry<8, 4, 480>(),
                                  res_entry<12, 2, 480>(), res_entry<12, 3, 480>(), res_entry<12, 4, 480>(),
                                  res_entry<16, 2, 480>(), res_entry<16, 3, 480>(), res_entry<16, 4, 480>(),
                                  res_entry<20, 7, 224>(), res_entry<24, 7, 224>()};
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

// Words of the exchange buffer for all launches of one factorisation (none where
// the tail is off or takes the matrix whole, or with too many rows).
size_t bidiag_resident_words(ddcsvd_context* ctx, int m, int n, int P, int* ld) {
  *ld = (int)round_up(std::min(n, kResSlice * P), 32);  // the most columns a launch starts with
  if (ctx->tune[TK_PANEL_TAIL] <= 0 || m - n > 24 * P || bidiag_tail_columns(ctx, m, n, 0) > 0) return 0;
  return (size_t)(P + 3) * *ld + 4 * (size_t)P;
}

int bidiag_resident(ddcsvd_context* ctx, int m, int n, int k0, int cols, float* W, int ldw, float* d, float* e,
                    float* tauq, float* taup, const BidiagWork& w) {
  const ResConfig* g = res_config(m - k0, n - k0, w.P, res_smem_max(ctx));
  if (!g || !w.rpart) return DDCSVD_ERR_UNSUPPORTED;
  ResParams p;
  p.mt = m - k0;
  p.nt = n - k0;
  p.cols = cols;
  p.S = std::max(0, p.nt - g->K * g->T);
  p.ldw = ldw;
  p.ldp = p.ldr = w.ldr;
  p.W = W + k0 + (size_t)k0 * ldw;
  p.d = d + k0;
  p.e = e + k0;
  p.tauq = tauq + k0;
  p.taup = taup + k0;
  p.tag0 = (unsigned)k0 + 1u;
  p.part = w.rpart;
  p.y = p.part + (size_t)w.P * p.ldp;
  p.row = p.y + p.ldr;
  p.cn = p.row + 2 * p.ldr;
  p.rn = p.cn + 2 * w.P;
  p.bar = w.bar;
  p.st = ctx->d_status;
  DDC_CUDA_TRY(cudaMemsetAsync(w.bar, 0, sizeof(GridBarrier), ctx->stream));
  const size_t smem = res_smem(*g, p.nt);
  DDC_TRY(allow_smem(ctx, g->fn));
  void* args[] = {&p};
  DDC_CUDA_TRY(cudaLaunchCooperativeKernel(g->fn, dim3(w.P), dim3(g->T + 32), args, smem, ctx->stream));
  count_launch();
  return DDCSVD_OK;
}

}  // namespace ddcsvd
