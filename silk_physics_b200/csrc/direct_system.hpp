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
  // Nor is it after give_up(), until the next step.
  bool usable() const { return usable_ && !given_up_; }
  void give_up() { given_up_ = true; }
  // Factorises L + diag(dyn) (kernels return at entry once *skip is set).
  void factorize(const double* Lvals, const float* dyn, const int* skip, cudaStream_t st);
  // Solves into a.x, to the tolerance of the CG solve `cg` stands for; sets
  // *failed where it has no factors or gives up.
  void solve(const CgArgs& cg, int* failed, cudaStream_t st);
  // Set when the last solve met its tolerance (the CG then has nothing to do).
  const int* solved() const { return state_ + kDirectSolved; }
  const int* state() const { return state_; }  // kDirectWords words on the device
  void begin_step() {
    factorisations_ = 0;
    given_up_ = false;
  }
  int factorisations() const { return factorisations_; }  // queued in this step
  // Compulsory DRAM bytes of one application: the factors once, the matrix
  // rows and the vectors of its residual.
  double application_bytes() const { return application_bytes_; }

 private:
  struct Level {
    int nodes = 0, steps = 0;
    int ent0 = 0, ent1 = 0, diag0 = 0, diag1 = 0;
    int64_t front = 0;
    int panel_task = 0, panel_tasks = 0;
    int tile = 0, tiles = 0;
    int add[4] = {0, 0, 0, 0}, adds[4] = {0, 0, 0, 0};
    int store = 0, stores = 0, product = 0, products = 0, schur = 0, schurs = 0;
  };
  void upload(const DirectPlan& P, const std::vector<DirectNodeDev>& nd,
              const std::vector<int2>& tasks, const std::vector<int4>& lists,
              const int64_t (&front)[2], int64_t gd, int panel, int level_nodes, int nv,
              cudaStream_t st);

  bool usable_ = false, given_up_ = false;
  int blocks_ = 0, factorisations_ = 0;
  size_t smem_ = 0;
  double application_bytes_ = 0.0;
  std::vector<Level> levels_;
  DirectArgs args_;
  // Everything on the device, in one allocation.
  DevBuf<char> arena_;
  DirectNodeDev* nodes_ = nullptr;
  int *ids_ = nullptr, *gat_ = nullptr, *cmap_ = nullptr, *ent_src_ = nullptr,
      *ent_dst_ = nullptr, *diag_id_ = nullptr, *diag_dst_ = nullptr;
  int2* tasks_ = nullptr;
  int4* lists_ = nullptr;  // panel tasks and the tiles of the other kernels
  double *fronts_[2] = {nullptr, nullptr}, *V_ = nullptr, *W_ = nullptr, *P_ = nullptr,
         *Gd_ = nullptr, *partials_ = nullptr;
  float *G_ = nullptr, *T_ = nullptr;
  float4 *u_ = nullptr, *f_ = nullptr, *r_ = nullptr, *dx_ = nullptr, *xn_ = nullptr;
  unsigned* barrier_ = nullptr;
  int* state_ = nullptr;
};

}  // namespace silkb
