// Direct solve of the ADMM system: see direct.cuh.
//
// Factorisation (per ADMM solve): level by level from the leaves, every front
// [A_SS A_SB; . A_BB] is assembled in FP64 (upper triangle) and its own block
// is eliminated with symmetric block sweeps of kDirectPanel pivots, which
// leave -A_SS^-1, G = A_SS^-1 A_SB and the Schur complement in place.  The
// own block's inverse is stored rather than its triangular factor: an
// application is then a product, not a chain of m dependent rows.
//
// Application: forward u = G^T f and backward x = [A_SS^-1 | -G] [f; x_B] are
// the same product y = M^T v, so both run through one routine.
//
// Why at all: within an ADMM solve the matrix is fixed and the CG is bound by
// the latency of its barriers (7.7 us an iteration at 6,400 vertices, 18 us at
// 100K, 60 to 140 iterations a solve).  An application reads 6.7 MB of factors
// at 6,400 vertices and 140 MB at 100K once and leaves a relative residual of
// 1e-6 to 1e-5, so one or two take the place of a CG solve.  A contact step of
// the 80 x 80 scene went from 243 to 99 ms with it, the first contact step of
// the 100K-vertex drape from 1,681 to 512 ms.
#include <cmath>

#include "direct.cuh"
#include "grid_barrier.cuh"
#include "mas_cg.cuh"

namespace silkb {

namespace {

constexpr int kP = kDirectPanel;
constexpr int kT = kDirectTile;

__device__ __forceinline__ long long up(int N, int i, int j) {
  return i <= j ? (long long)i * N + j : (long long)j * N + i;
}

__global__ void direct_begin_kernel(int* state, const int* skip) {
  if (skip && *skip) return;
  state[0] = 0;
  state[1] = 0;
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

// Pivot block of step `step` inverted (Gauss-Jordan; the pivots of a positive
// definite matrix stay positive, anything else marks the factorisation as
// failed), the pivot rows V and W = P V of 64 columns.  Every block inverts
// the pivot block itself, which is cheaper than another launch.
__global__ void __launch_bounds__(256) direct_panel_kernel(DirectFactorArgs a, const int4* tasks,
                                                           int step) {
  if (a.skip && *a.skip) return;
  const int4 q = tasks[blockIdx.x];  // node, first column
  const DirectNodeDev n = a.nodes[q.x];
  const int k0 = step * kP;
  if (k0 >= n.m) return;
  const int nb = min(kP, n.m - k0), N = n.m + n.b;
  const double* F = a.F + n.front;
  __shared__ double A[kP][kP + 1];
  __shared__ double V[kP][kT + 1];
  __shared__ double col[kP], row[kP];
  __shared__ int bad;
  const int tid = threadIdx.x;
  if (tid == 0) bad = 0;
  for (int e = tid; e < kP * kP; e += 256) {
    const int i = e / kP, j = e % kP;
    A[i][j] = i < nb && j < nb ? F[up(N, k0 + i, k0 + j)] : (i == j ? 1.0 : 0.0);
  }
  const int c0 = q.y;
  // Columns at or right of the pivots are read along rows, those left of
  // them (eliminated before) along columns of the upper triangle.
  for (int e = tid; e < kP * kT; e += 256) {
    if (c0 >= k0) {
      const int i = e / kT, j = e % kT;
      V[i][j] = i < nb && c0 + j < N ? F[up(N, k0 + i, c0 + j)] : 0.0;
    } else {
      const int i = e % kP, j = e / kP;
      V[i][j] = i < nb && c0 + j < N ? F[up(N, k0 + i, c0 + j)] : 0.0;
    }
  }
  __syncthreads();
  for (int k = 0; k < nb; ++k) {
    if (tid < kP) {
      col[tid] = A[tid][k];
      row[tid] = A[k][tid];
    }
    __syncthreads();
    const double p = col[k];
    const double inv = 1.0 / p;
    if (tid == 0 && !(p > 0.0 && isfinite(inv))) bad = 1;
#pragma unroll
    for (int e = tid; e < kP * kP; e += 256) {
      const int i = e / kP, j = e % kP;
      double v;
      if (i == k && j == k) v = inv;
      else if (i == k) v = row[j] * inv;
      else if (j == k) v = -col[i] * inv;
      else v = A[i][j] - col[i] * row[j] * inv;
      A[i][j] = v;
    }
    __syncthreads();
  }
  if (bad) {
    if (tid == 0) atomicOr(a.state, 1);
  }
  if (c0 == 0) {
    double* P = a.P + (long long)q.z * kP * kP;
    for (int e = tid; e < kP * kP; e += 256) P[e] = A[e / kP][e % kP];
  }
  double* Vg = a.V + (long long)n.panel * kP;
  double* Wg = a.W + (long long)n.panel * kP;
  for (int e = tid; e < kP * kT; e += 256) {
    const int i = e / kT, j = e % kT;
    if (c0 + j >= N) continue;
    double w = 0.0;
#pragma unroll 8
    for (int k = 0; k < kP; ++k) w += A[i][k] * V[k][j];
    Vg[(long long)i * N + c0 + j] = V[i][j];
    Wg[(long long)i * N + c0 + j] = w;
  }
}

// F -= V^T W on one 64 x 64 tile of the upper triangle; the pivots' rows and
// columns become W, their block -P.  Bound by the FP64 pipe at 64 x 64 x 32
// products per 64 KB of fronts read and written.
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
    Vs[k][c] = i0 + c < N ? Vg[(long long)k * N + i0 + c] : 0.0;
    Ws[k][c] = j0 + c < N ? Wg[(long long)k * N + j0 + c] : 0.0;
  }
  const int ty = tid / 16, tx = tid % 16;
  double acc[4][4];
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const int i = i0 + ty + 16 * x, j = j0 + tx + 16 * y;
      acc[x][y] = i <= j && j < N ? F[(long long)i * N + j] : 0.0;
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
      for (int y = 0; y < 4; ++y) acc[x][y] -= v[x] * w[y];
  }
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const int i = i0 + ty + 16 * x, j = j0 + tx + 16 * y;
      if (i > j || j >= N) continue;
      const bool ik = i >= k0 && i < k0 + nb, jk = j >= k0 && j < k0 + nb;
      double v = acc[x][y];
      if (ik && jk) v = -P[(i - k0) * kP + (j - k0)];
      else if (ik) v = Wg[(long long)(i - k0) * N + j];
      else if (jk) v = Wg[(long long)(j - k0) * N + i];
      F[(long long)i * N + j] = v;
    }
}

// FP32 factors of one 32 x 32 tile of a level's own rows.
__global__ void __launch_bounds__(256) direct_store_kernel(DirectFactorArgs a,
                                                           const int4* tiles) {
  if (a.skip && *a.skip) return;
  const int4 q = tiles[blockIdx.x];  // node, tile row, tile column
  const DirectNodeDev n = a.nodes[q.x];
  const int N = n.m + n.b, i0 = q.y * 32, j0 = q.z * 32;
  const double* F = a.F + n.front;
  float* T = a.T + n.t;
  float* G = a.G + n.g;
  __shared__ float s[32][33];
  const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;
  bool finite = true;
  for (int r = ty; r < 32; r += 8) {
    const int i = i0 + r, j = j0 + tx;
    float v = 0.0f;
    if (i < n.m && j < N && i <= j) {
      v = -(float)F[(long long)i * N + j];
      finite &= isfinite(v) != 0;
      if (j < n.m)
        T[(long long)i * n.ms + j] = v;
      else
        G[(long long)i * n.bs + j - n.m] = -v;
    }
    s[r][tx] = v;
  }
  if (!finite) atomicOr(a.state, 1);
  __syncthreads();
  for (int r = ty; r < 32; r += 8) {
    const int j = j0 + r, i = i0 + tx;
    if (i < n.m && j < N && i <= j) T[(long long)j * n.ms + i] = s[tx][r];
  }
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

// One tree level of the forward (updates of the boundaries) or backward
// (correction of the own vertices) sweep.  A task is 32 columns of one
// front's factor M (R x C, row stride ld): a group of st.warps warps gathers
// the R-vector v into shared memory, splits the rows, and its first warp adds
// the partial sums in warp order.
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
    for (int i = w * 32 + lane; i < R; i += g * 32) {
      const int id = a.ids[n.ids + i];
      float4 s;
      if (i >= n.m) {
        s = __ldcg(a.dx + id);
      } else if (kForward || root) {
        s = __ldcg(a.r + id);
        for (int k = a.gat_off[n.ids + i]; k < a.gat_off[n.ids + i + 1]; ++k) {
          const float4 e = __ldcg(a.u + a.gat[k]);
          s.x -= e.x;
          s.y -= e.y;
          s.z -= e.z;
        }
        if (kForward && q.y == 0) a.f[id] = s;
      } else {
        s = __ldcg(a.f + id);
      }
      v[i] = s;
    }
    group_sync(group, g);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < C) {
      const int ld = kForward ? n.bs : n.ms;
      const float* M = (kForward ? a.G + n.g : a.T + n.t) + c;
      int i = w;
      for (; i + 7 * g < R; i += 8 * g) {
        float e[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) e[k] = __ldg(M + (size_t)(i + k * g) * ld);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float4 s = v[i + k * g];
          acc.x += e[k] * s.x;
          acc.y += e[k] * s.y;
          acc.z += e[k] * s.z;
        }
      }
      for (; i < R; i += g) {
        const float e = __ldg(M + (size_t)i * ld);
        const float4 s = v[i];
        acc.x += e * s.x;
        acc.y += e * s.y;
        acc.z += e * s.z;
      }
    }
    if (g > 1) {
      red[w * 32 + lane] = acc;
      group_sync(group, g);
      if (w == 0)
        for (int k = 1; k < g; ++k) add3(acc, red[k * 32 + lane]);
    }
    if (w == 0 && c < C) {
      if (kForward) {
        const int at = n.ids + n.m + c;
        for (int k = a.gat_off[at]; k < a.gat_off[at + 1]; ++k) add3(acc, __ldcg(a.u + a.gat[k]));
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
  if (a.state[0] != 0) return;    // no factorisation (every block alike)
  extern __shared__ float4 sm[];
  GridBarrier bar{a.barrier, a.barrier + 1, nullptr, gridDim.x};
  if (a.barrier_spin_limit > 0) bar.limit = a.barrier_spin_limit;
  auto sync = [&]() {
    if (bar.sync()) return true;
    if (blockIdx.x == 0 && threadIdx.x == 0 && a.fail) atomicOr(a.fail, kFailBarrier);
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
  for (int app = 0; app < kDirectMaxApplications; ++app) {
    for (int l = a.levels - 1; l > 0; --l) {
      direct_level<true>(a, a.fwd[l], false, sm);
      if (!sync()) return;
    }
    for (int l = 0; l < a.levels; ++l) {
      direct_level<false>(a, a.bwd[l], l == 0, sm);
      if (!sync()) return;
    }
    p = block_total(direct_residual(a, false, app == 0));
    double* part = a.partials + (size_t)((app + 1) & 1) * gridDim.x;
    if (threadIdx.x == 0) part[blockIdx.x] = p;
    if (!sync()) return;
    const double now = grid_total(part, gridDim.x);
    ok = now <= abs2 || now <= rel2 * rr0;
    if (ok || !(now < 0.0625 * rr)) break;
    rr = now;
  }
  if (!ok) return;  // the CG launched after this solves from the unchanged start
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.nv; i += gridDim.x * blockDim.x)
    a.x[i] = __ldcg(a.xn + i);
  if (blockIdx.x == 0 && threadIdx.x == 0) a.state[1] = 1;
}

// Clears the previous solve's verdict (state[1]) and the barrier words.
__global__ void direct_reset_kernel(int* state, unsigned* barrier) {
  state[1] = 0;
  barrier[0] = 0;
  barrier[1] = 0;
}

}  // namespace

int direct_max_blocks(size_t smem) {
  static const int sms = [] {
    int dev = 0, n = 0;
    CUDA_CHECK(cudaGetDevice(&dev));
    CUDA_CHECK(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    CUDA_CHECK(cudaFuncSetAttribute(direct_solve_kernel,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    return n;
  }();
  int per_sm = 0;
  if (smem > 200 * 1024 ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, direct_solve_kernel, kDirectThreads,
                                                    smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return per_sm > 0 ? sms : 0;
}

void launch_direct_begin(int* state, const int* skip, cudaStream_t st) {
  direct_begin_kernel<<<1, 1, 0, st>>>(state, skip);
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

void launch_direct_solve(const DirectArgs& a, int blocks, size_t smem, cudaStream_t st) {
  direct_reset_kernel<<<1, 1, 0, st>>>(a.state, a.barrier);
  SILK_LAUNCHED();
  void* args[] = {(void*)&a};
  CUDA_CHECK(cudaLaunchCooperativeKernel((const void*)direct_solve_kernel, dim3(blocks),
                                         dim3(kDirectThreads), args, smem, st));
  SILK_LAUNCHED();
}

}  // namespace silkb
