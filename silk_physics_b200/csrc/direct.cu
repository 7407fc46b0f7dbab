// Direct solve of the ADMM system: see direct.cuh.
//
// Factorisation (per ADMM solve): level by level from the leaves, every front
// [A_SS A_SB; . A_BB] is assembled in FP64 (upper triangle), its own block is
// inverted in place by symmetric block sweeps of kDirectPanel pivots, and two
// products give G = A_SS^-1 A_SB and the Schur complement A_BB - A_SB^T G.
// The own block's inverse is stored rather than its triangular factor: an
// application is then a product, not a chain of m dependent rows.  (Sweeping
// whole fronts would read and write all of them once per 32 pivots: 5.9 ms a
// factorisation at 100K vertices, bound by that traffic.)
//
// Application: forward u = G^T f and backward x = [A_SS^-1 | -G] [f; x_B] are
// the same product y = M^T v, so both run through one routine.
//
// Why at all: within an ADMM solve the matrix is fixed and the CG is bound by
// the latency of its barriers (7.7 us an iteration at 6,400 vertices, 18 us at
// 100K, 60 to 140 iterations a solve).  An application reads 6.7 MB of factors
// at 6,400 vertices and 140 MB at 100K once and leaves a relative residual of
// 1e-6 to 1e-5, so one or two take the place of a CG solve: 60 us in place of
// 440 at 6,400 vertices, 174 in place of 1,910 at 100K (one application).
#include <cmath>

#include "direct.cuh"
#include "grid_barrier.cuh"
#include "mas_cg.cuh"
#include "per_device.hpp"

namespace silkb {

namespace {

constexpr int kP = kDirectPanel;
constexpr int kT = kDirectTile;

__device__ __forceinline__ long long up(int N, int i, int j) {
  return i <= j ? (long long)i * N + j : (long long)j * N + i;
}

__global__ void direct_begin_kernel(int* state, unsigned* barrier, const int* skip) {
  if (skip && *skip) return;
  state[kDirectFailed] = 0;
  state[kDirectSolved] = 0;
  barrier[0] = barrier[1] = barrier[2] = 0;
}

// Matrix entries of a level's fronts (the buffer was zeroed; each entry of A
// has one destination) and the dynamic diagonal on top of them.
__global__ void __launch_bounds__(256) direct_fill_kernel(DirectFactorArgs a, int ent0, int n) {
  if (a.skip && *a.skip) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a.F[a.ent_dst[ent0 + i]] = a.Lvals[a.ent_src[ent0 + i]];
}

__global__ void __launch_bounds__(256) direct_diag_kernel(DirectFactorArgs a, int d0, int n) {
  if (a.skip && *a.skip) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a.F[a.diag_dst[d0 + i]] += (double)a.dyn[a.diag_id[d0 + i]];
}

// Schur complements of the children in one slot added into their parents'
// fronts (one child per parent, so no two blocks add to an entry).
__global__ void __launch_bounds__(256) direct_add_kernel(DirectFactorArgs a,
                                                         const DirectNodeDev* kids,
                                                         const int4* tiles) {
  if (a.skip && *a.skip) return;
  const int4 q = tiles[blockIdx.x];  // child, parent, tile row, tile column
  const DirectNodeDev c = kids[q.x], p = a.nodes[q.y];
  const int Nc = c.m + c.b, Np = p.m + p.b;
  __shared__ int mi[kT], mj[kT];
  const int i0 = q.z * kT, j0 = q.w * kT;
  if (threadIdx.x < kT)
    mi[threadIdx.x] = i0 + (int)threadIdx.x < c.b ? a.cmap[c.u + i0 + threadIdx.x] : 0;
  else if (threadIdx.x < 2 * kT)
    mj[threadIdx.x - kT] =
        j0 + (int)threadIdx.x - kT < c.b ? a.cmap[c.u + j0 + threadIdx.x - kT] : 0;
  __syncthreads();
  const double* U = a.Fc + c.front;
  double* F = a.F + p.front;
  for (int e = threadIdx.x; e < kT * kT; e += blockDim.x) {
    const int i = e / kT, j = e % kT;
    if (i0 + i > j0 + j || j0 + j >= c.b) continue;
    F[up(Np, mi[i], mj[j])] += U[(long long)(c.m + i0 + i) * Nc + c.m + j0 + j];
  }
}

// Symmetric Gauss-Jordan of a 32 x 32 block by one warp: lane j holds column j
// in registers.  A pivot publishes its row (by symmetry its column) through
// shared memory, one double per lane.  The next pivot's row is updated first,
// so that its reciprocal is under way while the rest of the block follows.
// False if a pivot is not positive and finite.
__device__ bool invert_warp(double (&x)[kP], double (*row)[kP], int lane) {
  bool good = true;
  row[0][lane] = x[0];
  double p = __shfl_sync(0xffffffffu, x[0], 0), inv = __drcp_rn(p);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < kP; ++k) {
    good = good && p > 0.0 && inv > 0.0 && isfinite(inv);
    const double* s = row[k & 1];
    // Column k itself becomes s * inv, the others lose s * (their entry of
    // row k) * inv; row k is scaled.
    const bool own = lane == k;
    const double f = own ? -inv : x[k] * inv;
    double next = 1.0;
    if (k + 1 < kP) {
      x[k + 1] = fma(-s[k + 1], f, own ? 0.0 : x[k + 1]);
      row[(k + 1) & 1][lane] = x[k + 1];
      p = __shfl_sync(0xffffffffu, x[k + 1], k + 1);
      next = __drcp_rn(p);
    }
#pragma unroll
    for (int i = 0; i < kP; ++i)
      if (i != k && i != k + 1) x[i] = fma(-s[i], f, own ? 0.0 : x[i]);
    x[k] = f;
    inv = next;
    __syncwarp();
  }
  return good;
}

// Pivot block of step `step` of the own blocks inverted (the pivots of a
// positive definite matrix stay positive, anything else marks the
// factorisation as failed), and the pivot rows V and W = P V of 64 columns.
// Every block inverts the pivot block itself, which is cheaper than another
// launch.  Bound by the chain of 32 pivots: with a block barrier per pivot
// and the block spread over 256 threads a launch took 25 us.
__global__ void __launch_bounds__(256) direct_panel_kernel(DirectFactorArgs a, const int4* tasks,
                                                           int step) {
  if (a.skip && *a.skip) return;
  const int4 q = tasks[blockIdx.x];  // node, first column, node within the level
  const DirectNodeDev n = a.nodes[q.x];
  const int k0 = step * kP;
  if (k0 >= n.m) return;
  const int nb = min(kP, n.m - k0), N = n.m + n.b;
  const double* F = a.F + n.front;
  __shared__ double A[kP][kP + 1];
  __shared__ double V[kP][kT + 1];
  __shared__ double row[2][kP];
  const int tid = threadIdx.x, c0 = q.y;
  if (tid < 32) {
    double x[kP];
#pragma unroll
    for (int i = 0; i < kP; ++i)
      x[i] = i < nb && tid < nb ? F[up(N, k0 + i, k0 + tid)] : (i == tid ? 1.0 : 0.0);
    if (!invert_warp(x, row, tid) && tid == 0) atomicOr(a.state, 1);
#pragma unroll
    for (int i = 0; i < kP; ++i) A[i][tid] = -x[i];
    if (c0 == 0) {
      double* P = a.P + (long long)q.z * kP * kP;
#pragma unroll
      for (int i = 0; i < kP; ++i) P[i * kP + tid] = -x[i];
    }
  } else {
    // Columns at or right of the pivots are read along rows, those left of
    // them (eliminated before) along columns of the upper triangle.
    for (int e = tid - 32; e < kP * kT; e += 224) {
      const int r = c0 >= k0 ? e / kT : e % kP, c = c0 >= k0 ? e % kT : e / kP;
      V[r][c] = r < nb && c0 + c < n.m ? F[up(N, k0 + r, c0 + c)] : 0.0;
    }
  }
  __syncthreads();
  double* Vg = a.V + (long long)n.panel * kP;
  double* Wg = a.W + (long long)n.panel * kP;
  const int ty = tid / 16, tx = tid % 16;
  double w[2][4] = {};
#pragma unroll 8
  for (int k = 0; k < kP; ++k) {
    const double a0 = A[2 * ty][k], a1 = A[2 * ty + 1][k];
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const double x = V[k][tx + 16 * y];
      w[0][y] = fma(a0, x, w[0][y]);
      w[1][y] = fma(a1, x, w[1][y]);
    }
  }
#pragma unroll
  for (int y = 0; y < 4; ++y) {
    const int c = c0 + tx + 16 * y;
    if (c >= n.m) continue;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      Vg[(long long)(2 * ty + x) * N + c] = V[2 * ty + x][tx + 16 * y];
      Wg[(long long)(2 * ty + x) * N + c] = w[x][y];
    }
  }
}

// F -= V^T W on one 64 x 64 tile of the own block's upper triangle; the
// pivots' rows and columns become W, their block -P.
__global__ void __launch_bounds__(256) direct_update_kernel(DirectFactorArgs a,
                                                            const int4* tiles, int step) {
  if (a.skip && *a.skip) return;
  const int4 q = tiles[blockIdx.x];  // node, tile row, tile column, node within the level
  const DirectNodeDev n = a.nodes[q.x];
  const int k0 = step * kP;
  if (k0 >= n.m) return;
  const int nb = min(kP, n.m - k0), N = n.m + n.b;
  double* F = a.F + n.front;
  const double* Vg = a.V + (long long)n.panel * kP;
  const double* Wg = a.W + (long long)n.panel * kP;
  const double* P = a.P + (long long)q.w * kP * kP;
  __shared__ double Vs[kP][kT], Ws[kP][kT];
  const int i0 = q.y * kT, j0 = q.z * kT, tid = threadIdx.x;
  for (int e = tid; e < kP * kT; e += 256) {
    const int k = e / kT, c = e % kT;
    Vs[k][c] = i0 + c < n.m ? Vg[(long long)k * N + i0 + c] : 0.0;
    Ws[k][c] = j0 + c < n.m ? Wg[(long long)k * N + j0 + c] : 0.0;
  }
  const int ty = tid / 16, tx = tid % 16;
  double acc[4][4];
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const int i = i0 + ty + 16 * x, j = j0 + tx + 16 * y;
      acc[x][y] = i <= j && j < n.m ? F[(long long)i * N + j] : 0.0;
    }
  __syncthreads();
#pragma unroll 8
  for (int k = 0; k < kP; ++k) {
    double v[4], w[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      v[x] = Vs[k][ty + 16 * x];
      w[x] = Ws[k][tx + 16 * x];
    }
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y) acc[x][y] = fma(-v[x], w[y], acc[x][y]);
  }
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const int i = i0 + ty + 16 * x, j = j0 + tx + 16 * y;
      if (i > j || j >= n.m) continue;
      const bool ik = i >= k0 && i < k0 + nb, jk = j >= k0 && j < k0 + nb;
      double v = acc[x][y];
      if (ik && jk) v = -P[(i - k0) * kP + (j - k0)];
      else if (ik) v = Wg[(long long)(i - k0) * N + j];
      else if (jk) v = Wg[(long long)(j - k0) * N + i];
      F[(long long)i * N + j] = v;
    }
}

// Inverse of the own blocks, one 32 x 32 tile of the upper triangle: FP32
// into T (both triangles) and FP64 mirrored into F's lower triangle, where
// the product below reads whole rows.
__global__ void __launch_bounds__(256) direct_store_kernel(DirectFactorArgs a,
                                                           const int4* tiles) {
  if (a.skip && *a.skip) return;
  const int4 q = tiles[blockIdx.x];  // node, tile row, tile column
  const DirectNodeDev n = a.nodes[q.x];
  const int N = n.m + n.b, i0 = q.y * 32, j0 = q.z * 32;
  double* F = a.F + n.front;
  float* T = a.T + n.t;
  __shared__ double s[32][33];
  const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;
  bool finite = true;
  for (int r = ty; r < 32; r += 8) {
    const int i = i0 + r, j = j0 + tx;
    double v = 0.0;
    if (j < n.m && i <= j) {
      v = -F[(long long)i * N + j];
      finite &= isfinite((float)v) != 0;
      T[(long long)i * n.ms + j] = (float)v;
    }
    s[r][tx] = v;
  }
  if (!finite) atomicOr(a.state, 1);
  __syncthreads();
  for (int r = ty; r < 32; r += 8) {
    const int j = j0 + r, i = i0 + tx;
    if (j < n.m && i < j) {
      T[(long long)j * n.ms + i] = (float)s[tx][r];
      F[(long long)j * N + i] = -s[tx][r];
    }
  }
}

// One 64 x 64 tile of G = A_SS^-1 A_SB (kSchur = false: FP64 for the Schur
// complement, FP32 into G and, negated, T) or of A_BB -= A_SB^T G (kSchur =
// true, upper triangle).  Both are products L^T R over the m own rows, read
// in slices of 32 one slice ahead.  Bound by the FP64 pipe and, equally, the
// shared-memory passes of its operands (4 x 4 results a thread).
template <bool kSchur>
__global__ void __launch_bounds__(256) direct_product_kernel(DirectFactorArgs a,
                                                             const int4* tiles) {
  if (a.skip && *a.skip) return;
  const int4 q = tiles[blockIdx.x];  // node, tile row, tile column
  const DirectNodeDev n = a.nodes[q.x];
  const int N = n.m + n.b, m = n.m, nb = n.b;
  double* F = a.F + n.front;
  double* Gd = a.Gd + n.gd;
  const int i0 = q.y * kT, j0 = q.z * kT, tid = threadIdx.x;
  const double* L = kSchur ? F + m : F;
  const double* R = kSchur ? Gd : F + m;
  const long long ldr = kSchur ? nb : N;
  const int rows = kSchur ? nb : m;  // of the result
  __shared__ double Ls[kP][kT], Rs[kP][kT];
  const int ty = tid / 16, tx = tid % 16;
  // Slice k: rows k .. k + 31; thread's entries: rows tid / 64 + 4 e, column
  // tid % 64.
  const int lc = tid % kT, lr = tid / kT;
  double l[8], r[8];
  auto load = [&](int k) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int kk = k + lr + 4 * e;
      l[e] = kk < m && i0 + lc < rows ? L[(long long)kk * N + i0 + lc] : 0.0;
      r[e] = kk < m && j0 + lc < nb ? R[(long long)kk * ldr + j0 + lc] : 0.0;
    }
  };
  double acc[4][4] = {};
  load(0);
  for (int k = 0; k < m; k += kP) {
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      Ls[lr + 4 * e][lc] = l[e];
      Rs[lr + 4 * e][lc] = r[e];
    }
    __syncthreads();
    if (k + kP < m) load(k + kP);
#pragma unroll 8
    for (int kk = 0; kk < kP; ++kk) {
      double x[4], y[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        x[u] = Ls[kk][ty + 16 * u];
        y[u] = Rs[kk][tx + 16 * u];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int w = 0; w < 4; ++w) acc[u][w] = fma(-x[u], y[w], acc[u][w]);
    }
  }
  bool finite = true;
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const int i = i0 + ty + 16 * u, j = j0 + tx + 16 * w;
      if (i >= rows || j >= nb) continue;
      if (kSchur) {
        if (i <= j) F[(long long)(m + i) * N + m + j] += acc[u][w];
      } else {
        // The mirrored block holds -A_SS^-1, so acc is G.
        const float g = (float)acc[u][w];
        finite &= isfinite(g) != 0;
        Gd[(long long)i * nb + j] = acc[u][w];
        a.G[n.g + (long long)i * n.bs + j] = g;
        a.T[n.t + (long long)(m + j) * n.ms + i] = -g;
      }
    }
  if (!finite) atomicOr(a.state, 1);
}

__device__ __forceinline__ void group_sync(int group, int warps) {
  if (warps == 1)
    __syncwarp();
  else
    asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(warps * 32) : "memory");
}

// Fixed-order sum of one double per thread; every thread gets it.
__device__ double block_total(double v) {
  __shared__ double sh[kDirectThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  double t = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

__device__ double grid_total(const double* partials, int n) {
  double v = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) v += __ldcg(partials + i);
  return block_total(v);
}

__device__ __forceinline__ void add3(float4& a, const float4& b) {
  a.x += b.x;
  a.y += b.y;
  a.z += b.z;
}

// Sum of the updates listed in g.
__device__ __forceinline__ float4 direct_updates(const DirectArgs& a, const int4& g) {
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (g.x >= 0) add3(s, __ldcg(a.u + g.x));
  if (g.y >= 0) add3(s, __ldcg(a.u + g.y));
  if (g.z >= 0) add3(s, __ldcg(a.u + g.z));
  if (g.w >= 0) add3(s, __ldcg(a.u + g.w));
  return s;
}

// One tree level of the forward (updates of the boundaries) or backward
// (correction of the own vertices) sweep.  A task is 32 columns of one
// front's factor M (R x C, row stride ld): a group of st.warps warps gathers
// the R-vector v into shared memory, splits the rows, and its first warp adds
// the partial sums in warp order.  Rows are loaded in whole batches of
// kBatch, the last one padded with zeros: a row loop behind the batches
// would wait for every load in turn.
constexpr int kBatch = 12;
template <bool kForward>
__device__ void direct_level(const DirectArgs& a, const DirectStage& st, bool root, float4* sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = st.warps, group = warp / g, w = warp % g, groups = (kDirectThreads / 32) / g;
  float4* v = sm + (size_t)group * st.rows_max;
  float4* red = sm + (size_t)groups * st.rows_max + (size_t)(warp - w) * 32;
  for (int t = blockIdx.x + gridDim.x * group; t < st.tasks; t += gridDim.x * groups) {
    const int2 q = a.tasks[st.task + t];
    const DirectNodeDev n = a.nodes[q.x];
    const int c = q.y + lane;
    const int R = kForward ? n.m : n.m + n.b, C = kForward ? n.b : n.m;
    const int ld = kForward ? n.bs : n.ms;
    const float* M = (kForward ? a.G + n.g : a.T + n.t) + c;
    const bool live = c < C;
    float e[kBatch];
    auto load = [&](int i) {
#pragma unroll
      for (int k = 0; k < kBatch; ++k)
        e[k] = live && i + k * g < R ? __ldg(M + (size_t)(i + k * g) * ld) : 0.0f;
    };
    load(w);  // in flight while the vector is gathered
    for (int i = w * 32 + lane; i < R; i += g * 32) {
      const int id = a.ids[n.ids + i];
      float4 s;
      if (i >= n.m) {
        s = __ldcg(a.dx + id);
      } else if (kForward || root) {
        const int4 k = a.gat[n.ids + i];
        s = __ldcg(a.r + id);
        const float4 d = direct_updates(a, k);
        s.x -= d.x;
        s.y -= d.y;
        s.z -= d.z;
        if (kForward && q.y == 0) a.f[id] = s;
      } else {
        s = __ldcg(a.f + id);
      }
      v[i] = s;
    }
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    // Updates that pass through to the output, fetched beside the vector.
    float4 through = make_float4(0.f, 0.f, 0.f, 0.f);
    if (kForward && w == 0 && live) through = direct_updates(a, a.gat[n.ids + n.m + c]);
    group_sync(group, g);
    for (int i = w; i < R;) {
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        // A padded row multiplies some gathered row by zero.
        const float4 s = v[min(i + k * g, R - 1)];
        acc.x += e[k] * s.x;
        acc.y += e[k] * s.y;
        acc.z += e[k] * s.z;
      }
      i += kBatch * g;
      if (i < R) load(i);
    }
    if (g > 1) {
      red[w * 32 + lane] = acc;
      group_sync(group, g);
      if (w == 0)
#pragma unroll 4
        for (int k = 1; k < g; ++k) add3(acc, red[k * 32 + lane]);
    }
    if (w == 0 && live) {
      if (kForward) {
        add3(acc, through);
        a.u[n.u + c] = acc;
      } else {
        a.dx[a.ids[n.ids + c]] = acc;
      }
    }
    group_sync(group, g);
  }
}

// Residual rows: r = b - A x (first) or r -= A dx and xn += dx, products and
// sums of a row in FP64.  Returns this thread's share of r . r.
__device__ double direct_residual(const DirectArgs& a, bool first, bool second) {
  const int lane = threadIdx.x & 31;
  const int nwarps = gridDim.x * (kDirectThreads / 32);
  const float4* v = first ? a.x : a.dx;
  double rr = 0.0;
  for (int s = blockIdx.x + gridDim.x * (threadIdx.x >> 5); s < a.nslices; s += nwarps) {
    const int row = 32 * s + lane;
    if (row >= a.nv) continue;
    const int base = a.sl_ptr[s], width = a.sl_w[s];
    const float4 vi = __ldcg(v + row);
    const double d = (double)a.Ldiag[row] + (double)a.dyn[row];
    double yx = d * vi.x, yy = d * vi.y, yz = d * vi.z;
#pragma unroll 4
    for (int k = 0; k < width; ++k) {
      const int2 e = a.ent[base + k * 32 + lane];
      const double val = (double)__int_as_float(e.y);
      const float4 vj = __ldcg(v + e.x);
      yx += val * vj.x;
      yy += val * vj.y;
      yz += val * vj.z;
    }
    const float4 o = first ? a.b[row] : a.r[row];
    const float4 r = make_float4((float)(o.x - yx), (float)(o.y - yy), (float)(o.z - yz), 0.f);
    a.r[row] = r;
    if (!first) {
      float4 x = second ? a.x[row] : a.xn[row];
      x.x += vi.x;
      x.y += vi.y;
      x.z += vi.z;
      a.xn[row] = x;
    }
    rr += (double)r.x * r.x + (double)r.y * r.y + (double)r.z * r.z;
  }
  return rr;
}

__global__ void __launch_bounds__(kDirectThreads, 1) direct_solve_kernel(DirectArgs a) {
  if (a.skip && *a.skip) return;  // the ADMM solve already ended (every block alike)
  if (a.state[kDirectFailed] != 0) {  // no factors (every block alike)
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      a.state[kDirectSolved] = 0;
      *a.failed = 1;
    }
    return;
  }
  extern __shared__ float4 sm[];
  GridBarrier bar{a.barrier, a.barrier + 1, nullptr, gridDim.x};
  if (a.barrier_spin_limit > 0) bar.limit = a.barrier_spin_limit;
  if (a.withhold_block >= 0) bar.withhold = (unsigned)a.withhold_block;
  // Reported by every block whose wait gave up: block 0's own may have
  // succeeded on the same barrier.
  auto sync = [&]() {
    if (bar.sync()) return true;
    if (threadIdx.x == 0) {
      if (a.fail) atomicOr(a.fail, kFailBarrier);
      if (blockIdx.x == 0) a.state[kDirectSolved] = 0;
    }
    return false;
  };
  const float rel_tol = a.rel_tol_dev ? *a.rel_tol_dev : a.rel_tol;
  const double rel2 = (double)rel_tol * rel_tol, abs2 = (double)a.abs_tol * a.abs_tol;
  double p = block_total(direct_residual(a, true, false));
  // Two banks of partials: a block may write the next total's while another
  // still reads this one's.
  if (threadIdx.x == 0) a.partials[blockIdx.x] = p;
  if (!sync()) return;
  const double rr0 = grid_total(a.partials, gridDim.x);
  double rr = rr0;
  bool ok = false;
  int app = 0;
  while (app < kDirectMaxApplications) {
    for (int l = a.levels - 1; l > 0; --l) {
      direct_level<true>(a, a.fwd[l], false, sm);
      if (!sync()) return;
    }
    for (int l = 0; l < a.levels; ++l) {
      direct_level<false>(a, a.bwd[l], l == 0, sm);
      if (!sync()) return;
    }
    p = block_total(direct_residual(a, false, app == 0));
    ++app;
    double* part = a.partials + (size_t)(app & 1) * gridDim.x;
    if (threadIdx.x == 0) part[blockIdx.x] = p;
    if (!sync()) return;
    const double now = grid_total(part, gridDim.x);
    ok = now <= abs2 || now <= rel2 * rr0;
    if (ok || !(now < 0.0625 * rr)) break;
    rr = now;
  }
  // The last block to leave clears the barrier for the next solve.
  if (threadIdx.x == 0 && atomicAdd(a.barrier + 2, 1u) == gridDim.x - 1)
    a.barrier[0] = a.barrier[2] = 0u;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.state[kDirectSolved] = ok ? 1 : 0;
    // Reductions whose result is not waited for, but for a miss.
    atomicAdd(a.stats + kStatDirectApplied, app);
    if (ok)
      atomicAdd(a.stats + kStatDirectSolves, 1);
    // Given up once it has missed more often than not in this step: the
    // tries then cost no more than the solves before them have saved.
    else if (atomicAdd(a.stats + kStatDirectMisses, 1) >= a.stats[kStatDirectSolves])
      a.state[kDirectFailed] = *a.failed = 1;
  }
  if (!ok) return;  // the CG launched after this solves from the unchanged start
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.nv; i += gridDim.x * blockDim.x)
    a.x[i] = __ldcg(a.xn + i);
}

}  // namespace

int direct_max_blocks(size_t smem) {
  static PerDevice<int> sm_count;
  const int dev = current_device();
  const int sms = sm_count.get(dev, [dev] {
    int n = 0;
    CUDA_CHECK(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    CUDA_CHECK(cudaFuncSetAttribute(direct_solve_kernel,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    return n;
  });
  int per_sm = 0;
  if (smem > 200 * 1024 ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, direct_solve_kernel, kDirectThreads,
                                                    smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return per_sm > 0 ? sms : 0;
}

void launch_direct_begin(int* state, unsigned* barrier, const int* skip, cudaStream_t st) {
  direct_begin_kernel<<<1, 1, 0, st>>>(state, barrier, skip);
  SILK_LAUNCHED();
}

void launch_direct_fill(const DirectFactorArgs& a, int ent0, int ent1, int diag0, int diag1,
                        cudaStream_t st) {
  if (ent1 > ent0) {
    direct_fill_kernel<<<div_up(ent1 - ent0, 256), 256, 0, st>>>(a, ent0, ent1 - ent0);
    SILK_LAUNCHED();
  }
  if (diag1 > diag0) {
    direct_diag_kernel<<<div_up(diag1 - diag0, 256), 256, 0, st>>>(a, diag0, diag1 - diag0);
    SILK_LAUNCHED();
  }
}

void launch_direct_add(const DirectFactorArgs& a, const DirectNodeDev* kids, const int4* tiles,
                       int n, cudaStream_t st) {
  if (n == 0) return;
  direct_add_kernel<<<n, 256, 0, st>>>(a, kids, tiles);
  SILK_LAUNCHED();
}

void launch_direct_panel(const DirectFactorArgs& a, const int4* tasks, int n, int step,
                         cudaStream_t st) {
  if (n == 0) return;
  direct_panel_kernel<<<n, 256, 0, st>>>(a, tasks, step);
  SILK_LAUNCHED();
}

void launch_direct_update(const DirectFactorArgs& a, const int4* tiles, int n, int step,
                          cudaStream_t st) {
  if (n == 0) return;
  direct_update_kernel<<<n, 256, 0, st>>>(a, tiles, step);
  SILK_LAUNCHED();
}

void launch_direct_store(const DirectFactorArgs& a, const int4* tiles, int n, cudaStream_t st) {
  if (n == 0) return;
  direct_store_kernel<<<n, 256, 0, st>>>(a, tiles);
  SILK_LAUNCHED();
}

void launch_direct_products(const DirectFactorArgs& a, const int4* gtiles, int ng,
                            const int4* stiles, int ns, cudaStream_t st) {
  if (ng > 0) {
    direct_product_kernel<false><<<ng, 256, 0, st>>>(a, gtiles);
    SILK_LAUNCHED();
  }
  if (ns > 0) {
    direct_product_kernel<true><<<ns, 256, 0, st>>>(a, stiles);
    SILK_LAUNCHED();
  }
}

void launch_direct_solve(const DirectArgs& a, int blocks, size_t smem, cudaStream_t st) {
  void* args[] = {(void*)&a};
  CUDA_CHECK(cudaLaunchCooperativeKernel((const void*)direct_solve_kernel, dim3(blocks),
                                         dim3(kDirectThreads), args, smem, st));
  SILK_LAUNCHED();
}

}  // namespace silkb
