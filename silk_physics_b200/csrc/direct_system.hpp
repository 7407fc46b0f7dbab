// Direct solve of one cloth's ADMM system: device copy of its plan, factors
// and the launches of a factorisation and of a solve.
#pragma once

#include "direct.cuh"
#include "world.hpp"

namespace silkb {

class DirectSystem {
 public:
  // Builds the plan and its device arrays on `st`.  usable() is false when
  // the fronts would not pay or do not fit the device's free memory.
  DirectSystem(const ClothSetup& S, const std::vector<float>& rest, cudaStream_t st);
  bool usable() const { return usable_; }
  // Factorises L + diag(dyn) (kernels return at entry once *skip is set).
  void factorize(const double* Lvals, const float* dyn, const int* skip, cudaStream_t st);
  // Solves into a.x, to the tolerance of the CG solve `cg` stands for.
  void solve(const CgArgs& cg, cudaStream_t st);
  // Set when the last solve met its tolerance (the CG then has nothing to do).
  const int* solved() const { return state_.p + 1; }

 private:
  struct Level {
    int nodes = 0, steps = 0;
    int ent0 = 0, ent1 = 0, diag0 = 0, diag1 = 0;
    int64_t front = 0;
    int panel_task = 0, panel_tasks = 0;
    int tile = 0, tiles = 0;
    int add[4] = {0, 0, 0, 0}, adds[4] = {0, 0, 0, 0};
    int store = 0, stores = 0;
  };
  void upload(DirectPlan& P, const std::vector<DirectNodeDev>& nd,
              const std::vector<int2>& tasks, const std::vector<int4>& lists,
              const int64_t (&front)[2], int panel, int level_nodes, int nv, cudaStream_t st);
  void release();

  bool usable_ = false;
  int blocks_ = 0;
  size_t smem_ = 0;
  std::vector<Level> levels_;
  DirectArgs args_;
  DevBuf<DirectNodeDev> nodes_;
  DevBuf<int> ids_, gat_off_, gat_, cmap_, ent_src_, ent_dst_, diag_id_, diag_dst_;
  DevBuf<int2> tasks_;
  DevBuf<int4> lists_;  // panel tasks, update tiles, add tiles and store tiles
  DevBuf<double> fronts_[2], V_, W_, P_, partials_;
  DevBuf<float> G_, T_;
  DevBuf<float4> u_, f_, r_, dx_, xn_;
  DevBuf<unsigned> barrier_;
  DevBuf<int> state_;
};

}  // namespace silkb
