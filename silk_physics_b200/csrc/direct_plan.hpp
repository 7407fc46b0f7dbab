// Nested-dissection plan of a cloth's scalar system (host, once per cloth):
// the tree of dense fronts that the direct ADMM solve factorises and applies
// on the GPU (direct.cu).
#pragma once

#include <cstdint>
#include <vector>

namespace silkb {

// Edge of a factorisation tile and of a column chunk of its panels.
constexpr int kDirectTile = 64;
// Pivots eliminated per factorisation step.
constexpr int kDirectPanel = 32;

// One front: m own vertices (a separator, or a leaf region), then b boundary
// vertices, the vertices of enclosing separators that its region touches.
struct DirectNode {
  int m = 0, b = 0;
  int level = 0;      // depth, 0 = root
  int parent = -1;
  int slot = 0;       // index among the parent's children (0..3)
  int ids = 0;        // first entry in DirectPlan::ids (own, then boundary)
  int u = 0;          // first boundary entry in the update vector / cmap
  int64_t front = 0;  // first entry in its level's front buffer, row-major N x N
  int panel = 0;      // first column in the panel scratch
  int ms = 0, bs = 0;  // row strides of the stored factors
  int64_t g = 0, t = 0;  // first entries of the m x b and (m + b) x m factors
};

struct DirectPlan {
  std::vector<DirectNode> nodes;        // by level, root first
  std::vector<int> level_off;           // per level: first node (levels + 1 entries)
  std::vector<int> ids;                 // solver vertex ids of every front
  std::vector<int> gat;                 // per entry of ids: 4 update entries summed into it (-1 none)
  std::vector<int> cmap;                // per boundary entry: position in the parent's front
  std::vector<int64_t> level_front;     // per level: entries of its front buffer
  std::vector<int> level_panel;         // per level: columns of its panel scratch
  // Matrix entries of each level's fronts: source in Lvals, destination in
  // the level's buffer; vertex ids of the diagonal entries.
  std::vector<int> ent_off, diag_off;   // per level (levels + 1)
  std::vector<int> ent_src, ent_dst, diag_id, diag_dst;
  int64_t g_total = 0, t_total = 0;
  int u_total = 0;
  int levels() const { return (int)level_off.size() - 1; }
};

// Builds the plan of the nv x nv symmetric matrix with CSR pattern rows /
// cols (diagonal included), bisecting by the rest positions pos (3 per
// vertex, solver order).  False when the fronts would be too large to pay
// (the plan is then empty).
bool build_direct_plan(int nv, const std::vector<int>& rows, const std::vector<int>& cols,
                       const std::vector<float>& pos, DirectPlan& plan);

}  // namespace silkb
