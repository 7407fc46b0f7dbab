// Direct solve of a cloth's ADMM system (L + diag(dyn)) (x) I3: nested
// dissection factorisation in FP64 on the GPU, factors stored in FP32 and
// applied with iterative refinement by one cooperative kernel per solve.
#pragma once

#include "common.cuh"
#include "direct_plan.hpp"

namespace silkb {

// Device copy of one front (see DirectNode).
struct DirectNodeDev {
  int m, b, ids, u, front, panel, ms, bs;
  long long g, t, gd;
};

// Work of one tree level in the application kernel: tasks (node, first
// column) of 32 columns each, run by groups of `warps` warps (1, 4, 8, 16 or
// 32) that split the rows.
struct DirectStage {
  int task = 0, tasks = 0, warps = 1, rows_max = 0;
};

constexpr int kDirectMaxLevels = 12;
constexpr int kDirectThreads = 1024;
constexpr int kDirectMaxApplications = 4;

// Words of DirectArgs::state.
enum DirectState {
  kDirectFailed = 0,  // no usable factors, or given up
  kDirectSolved = 1,  // the last solve met its tolerance
  kDirectWords = 2
};

struct DirectArgs {
  int nv = 0, nslices = 0, levels = 0;
  const int* sl_ptr = nullptr;
  const int* sl_w = nullptr;
  const int2* ent = nullptr;
  const float* Ldiag = nullptr;
  const float* dyn = nullptr;
  const float4* b = nullptr;
  float4* x = nullptr;
  const DirectNodeDev* nodes = nullptr;
  const int* ids = nullptr;
  const int4* gat = nullptr;  // per entry of ids: updates summed into it (-1 none)
  const int2* tasks = nullptr;
  DirectStage fwd[kDirectMaxLevels], bwd[kDirectMaxLevels];
  const float* G = nullptr;
  const float* T = nullptr;
  float4* u = nullptr;    // updates of the boundaries
  float4* f = nullptr;    // condensed residual of the own vertices
  float4* r = nullptr;    // residual
  float4* dx = nullptr;   // correction of the current application
  float4* xn = nullptr;   // x plus the corrections so far
  double* partials = nullptr;
  unsigned* barrier = nullptr;  // [count, err, blocks that left]
  int* state = nullptr;  // kDirectWords words
  int* stats = nullptr;   // CgArgs::stats
  int* failed = nullptr;  // AdmmControl::direct_failed
  int* fail = nullptr;   // kFail* word of the solver
  const int* skip = nullptr;
  const float* rel_tol_dev = nullptr;
  float rel_tol = 1e-3f, abs_tol = 1e-7f;
  long long barrier_spin_limit = 0;
  int withhold_block = -1;  // >= 0: that block skips its barrier arrivals (tests)
};

// One level of the factorisation.
struct DirectFactorArgs {
  const DirectNodeDev* nodes = nullptr;
  const int* ids = nullptr;
  const int* cmap = nullptr;
  const int* ent_src = nullptr;
  const int* ent_dst = nullptr;
  const int* diag_id = nullptr;
  const int* diag_dst = nullptr;
  const double* Lvals = nullptr;
  const float* dyn = nullptr;
  double* F = nullptr;        // fronts of this level
  const double* Fc = nullptr;  // fronts of the children's level
  double* V = nullptr;        // panel scratch: old and eliminated pivot rows
  double* W = nullptr;
  double* P = nullptr;        // inverted pivot blocks
  double* Gd = nullptr;       // G of this level in FP64
  float* G = nullptr;
  float* T = nullptr;
  int* state = nullptr;
  const int* skip = nullptr;
};

// Blocks of the application kernel that are resident at once on this device
// with `smem` bytes of dynamic shared memory (0: not launchable).
int direct_max_blocks(size_t smem);
void launch_direct_begin(int* state, unsigned* barrier, const int* skip, cudaStream_t st);
void launch_direct_fill(const DirectFactorArgs& a, int ent0, int ent1, int diag0, int diag1,
                        cudaStream_t st);
// tiles: (child node, tile row, tile column) of one child slot.
void launch_direct_add(const DirectFactorArgs& a, const DirectNodeDev* kids, const int4* tiles,
                       int n, cudaStream_t st);
void launch_direct_panel(const DirectFactorArgs& a, const int4* tasks, int n, int step,
                         cudaStream_t st);
void launch_direct_update(const DirectFactorArgs& a, const int4* tiles, int n, int step,
                          cudaStream_t st);
void launch_direct_store(const DirectFactorArgs& a, const int4* tiles, int n, cudaStream_t st);
void launch_direct_products(const DirectFactorArgs& a, const int4* gtiles, int ng,
                            const int4* stiles, int ns, cudaStream_t st);
void launch_direct_solve(const DirectArgs& a, int blocks, size_t smem, cudaStream_t st);

}  // namespace silkb
