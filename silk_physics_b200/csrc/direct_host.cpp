// Host side of the direct ADMM solve (see direct_system.hpp).
#include <algorithm>
#include <type_traits>

#include "direct_system.hpp"

namespace silkb {

namespace {

constexpr int kWarps = kDirectThreads / 32;
constexpr size_t kSolveSmem = 128 * 1024;  // gathered vectors of a block

// Warps that share a task: as many as fill the chip in one round of tasks
// while each still has eight rows, and enough that the gathered vectors of
// a block's groups fit its shared memory.
int group_warps(int tasks, int rows, int sms) {
  int g = 32;
  for (int c : {1, 4, 8, 16})
    if ((int64_t)tasks * c * 2 > (int64_t)sms * kWarps || rows <= 8 * c) {
      g = c;
      break;
    }
  while (g < 32 && (size_t)(kWarps / g) * rows * sizeof(float4) > kSolveSmem)
    g = g == 1 ? 4 : 2 * g;
  return g;
}

}  // namespace

DirectSystem::DirectSystem(const ClothSetup& S, const std::vector<float>& rest,
                           cudaStream_t st) {
  std::vector<float> pos(3 * (size_t)S.nv);
  for (int i = 0; i < S.nv; ++i)
    for (int d = 0; d < 3; ++d) pos[3 * (size_t)S.perm[i] + d] = rest[3 * (size_t)i + d];
  DirectPlan P;
  if (!build_direct_plan(S.nv, S.Lrows, S.Lcols, pos, P)) return;
  const int nl = P.levels();
  if (nl > kDirectMaxLevels) return;
  int64_t front[2] = {0, 0};
  int panel = 0, level_nodes = 0;
  int64_t gd = 1;  // most entries of a level's G
  std::vector<int64_t> node_gd(P.nodes.size(), 0);
  for (int l = 0; l < nl; ++l) {
    int64_t at = 0;
    for (int i = P.level_off[l]; i < P.level_off[l + 1]; ++i) {
      node_gd[i] = at;
      at += (int64_t)P.nodes[i].m * P.nodes[i].b;
    }
    gd = std::max(gd, at);
    front[l & 1] = std::max(front[l & 1], P.level_front[l]);
    panel = std::max(panel, P.level_panel[l]);
    level_nodes = std::max(level_nodes, P.level_off[l + 1] - P.level_off[l]);
  }
  {
    const size_t need = (size_t)(front[0] + front[1] + gd) * 8 + (size_t)(P.g_total + P.t_total) * 4 +
                        (size_t)panel * kDirectPanel * 16;
    size_t free_b = 0, total_b = 0;
    CUDA_CHECK(cudaMemGetInfo(&free_b, &total_b));
    if (need > free_b / 4) return;
  }
  std::vector<DirectNodeDev> nd;
  for (size_t i = 0; i < P.nodes.size(); ++i) {
    const DirectNode& n = P.nodes[i];
    nd.push_back({n.m, n.b, n.ids, n.u, (int)n.front, n.panel, n.ms, n.bs, (long long)n.g,
                  (long long)n.t, (long long)node_gd[i]});
  }
  std::vector<std::vector<int>> kids(P.nodes.size());
  for (int i = 1; i < (int)P.nodes.size(); ++i) kids[P.nodes[i].parent].push_back(i);
  int dev = 0, sms = 0;
  CUDA_CHECK(cudaGetDevice(&dev));
  CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  std::vector<int2> tasks;
  std::vector<int4> lists;
  levels_.resize(nl);
  int want = 1;
  size_t vec = 0;
  for (int l = 0; l < nl; ++l) {
    Level& L = levels_[l];
    const int n0 = P.level_off[l], n1 = P.level_off[l + 1];
    L.nodes = n1 - n0;
    L.ent0 = P.ent_off[l];
    L.ent1 = P.ent_off[l + 1];
    L.diag0 = P.diag_off[l];
    L.diag1 = P.diag_off[l + 1];
    L.front = P.level_front[l];
    DirectStage fw, bw;
    fw.task = (int)tasks.size();
    for (int i = n0; i < n1; ++i) {
      const DirectNode& n = P.nodes[i];
      // A front without a boundary still condenses its own residual.
      for (int c = 0; c < std::max(n.b, 1); c += 32) tasks.push_back(make_int2(i, c));
      fw.rows_max = std::max(fw.rows_max, n.m);
      bw.rows_max = std::max(bw.rows_max, n.m + n.b);
      L.steps = std::max(L.steps, div_up(n.m, kDirectPanel));
    }
    fw.tasks = (int)tasks.size() - fw.task;
    bw.task = (int)tasks.size();
    for (int i = n0; i < n1; ++i)
      for (int c = 0; c < P.nodes[i].m; c += 32) tasks.push_back(make_int2(i, c));
    bw.tasks = (int)tasks.size() - bw.task;
    for (DirectStage* s : {&fw, &bw}) {
      s->warps = group_warps(s->tasks, s->rows_max, sms);
      const int groups = kWarps / s->warps;
      vec = std::max(vec, (size_t)groups * s->rows_max);
      if (l > 0 || s == &bw) want = std::max(want, div_up(s->tasks, groups));
    }
    args_.fwd[l] = fw;
    args_.bwd[l] = bw;
    L.panel_task = (int)lists.size();
    for (int i = n0; i < n1; ++i) {
      const DirectNode& n = P.nodes[i];
      if (n.m == 0) continue;
      for (int c = 0; c < n.m; c += kDirectTile)
        lists.push_back(make_int4(i, c, i - n0, 0));
    }
    L.panel_tasks = (int)lists.size() - L.panel_task;
    L.tile = (int)lists.size();
    for (int i = n0; i < n1; ++i) {
      const DirectNode& n = P.nodes[i];
      if (n.m == 0) continue;
      const int k = div_up(n.m, kDirectTile);
      for (int x = 0; x < k; ++x)
        for (int y = x; y < k; ++y) lists.push_back(make_int4(i, x, y, i - n0));
    }
    L.tiles = (int)lists.size() - L.tile;
    for (int s = 0; s < 4; ++s) {
      L.add[s] = (int)lists.size();
      for (int i = n0; i < n1; ++i) {
        if (s >= (int)kids[i].size()) continue;
        const int k = div_up(P.nodes[kids[i][s]].b, kDirectTile);
        for (int x = 0; x < k; ++x)
          for (int y = x; y < k; ++y) lists.push_back(make_int4(kids[i][s], i, x, y));
      }
      L.adds[s] = (int)lists.size() - L.add[s];
    }
    L.store = (int)lists.size();
    for (int i = n0; i < n1; ++i) {
      const DirectNode& n = P.nodes[i];
      for (int x = 0; x < div_up(n.m, 32); ++x)
        for (int y = x; y < div_up(n.m, 32); ++y) lists.push_back(make_int4(i, x, y, 0));
    }
    L.stores = (int)lists.size() - L.store;
    L.product = (int)lists.size();
    for (int i = n0; i < n1; ++i)
      for (int x = 0; x < div_up(P.nodes[i].m, kDirectTile); ++x)
        for (int y = 0; y < div_up(P.nodes[i].b, kDirectTile); ++y)
          lists.push_back(make_int4(i, x, y, 0));
    L.products = (int)lists.size() - L.product;
    L.schur = (int)lists.size();
    for (int i = n0; i < n1; ++i)
      for (int x = 0; x < (P.nodes[i].m ? div_up(P.nodes[i].b, kDirectTile) : 0); ++x)
        for (int y = x; y < div_up(P.nodes[i].b, kDirectTile); ++y)
          lists.push_back(make_int4(i, x, y, 0));
    L.schurs = (int)lists.size() - L.schur;
  }
  smem_ = (vec + (size_t)kWarps * 32) * sizeof(float4);
  const int most = direct_max_blocks(smem_);
  if (most == 0) return;
  blocks_ = std::min(want, most);
  try {
    upload(P, nd, tasks, lists, front, gd, panel, level_nodes, S.nv, st);
  } catch (const CudaError&) {
    // Other worlds took the memory meanwhile: the CG needs none of this.
    cudaGetLastError();
    arena_.reset();
    return;
  }
  // Factors; 8 B per entry of L and 16 B per vertex for dx, r, xn (read and
  // written), Ldiag and dyn.
  application_bytes_ = 4.0 * (double)(P.g_total + P.t_total) +
                       8.0 * (double)(S.Lcols.size() - (size_t)S.nv) + (5 * 16.0 + 8.0) * S.nv;
  args_.nv = S.nv;
  args_.levels = nl;
  args_.nodes = nodes_;
  args_.ids = ids_;
  args_.gat = reinterpret_cast<const int4*>(gat_);
  args_.tasks = tasks_;
  args_.G = G_;
  args_.T = T_;
  args_.u = u_;
  args_.f = f_;
  args_.r = r_;
  args_.dx = dx_;
  args_.xn = xn_;
  args_.partials = partials_;
  args_.barrier = barrier_;
  args_.state = state_;
  usable_ = true;
}

// One allocation for everything (a first solve otherwise spends longer in
// two dozen allocations than in its factorisation).
void DirectSystem::upload(const DirectPlan& P, const std::vector<DirectNodeDev>& nd,
                          const std::vector<int2>& tasks, const std::vector<int4>& lists,
                          const int64_t (&front)[2], int64_t gd, int panel, int level_nodes,
                          int nv, cudaStream_t st) {
  size_t need = 0;
  char* base = nullptr;
  auto place = [&](auto*& p, size_t count) {
    p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(base + need);
    need += (std::max<size_t>(count, 1) * sizeof(*p) + 255) / 256 * 256;
  };
  for (int pass = 0; pass < 2; ++pass) {
    need = 0;
    place(nodes_, nd.size());
    place(ids_, P.ids.size());
    place(gat_, P.gat.size());
    place(cmap_, P.cmap.size());
    place(ent_src_, P.ent_src.size());
    place(ent_dst_, P.ent_dst.size());
    place(diag_id_, P.diag_id.size());
    place(diag_dst_, P.diag_dst.size());
    place(tasks_, tasks.size());
    place(lists_, lists.size());
    place(fronts_[0], front[0]);
    place(fronts_[1], front[1]);
    place(V_, (size_t)panel * kDirectPanel);
    place(W_, (size_t)panel * kDirectPanel);
    place(P_, (size_t)level_nodes * kDirectPanel * kDirectPanel);
    place(Gd_, gd);
    place(G_, P.g_total);
    place(T_, P.t_total);
    place(u_, P.u_total);
    for (float4** v : {&f_, &r_, &dx_, &xn_}) place(*v, nv);
    place(partials_, 2 * (size_t)blocks_);
    place(barrier_, 3);
    place(state_, kDirectWords);
    if (pass == 0) {
      arena_.alloc(need);
      base = arena_.p;
    }
  }
  auto copy = [&](auto* to, const auto& from) {
    if (!from.empty())
      CUDA_CHECK(cudaMemcpyAsync(to, from.data(), from.size() * sizeof(from[0]),
                                 cudaMemcpyHostToDevice, st));
  };
  copy(nodes_, nd);
  copy(ids_, P.ids);
  copy(gat_, P.gat);
  copy(cmap_, P.cmap);
  copy(ent_src_, P.ent_src);
  copy(ent_dst_, P.ent_dst);
  copy(diag_id_, P.diag_id);
  copy(diag_dst_, P.diag_dst);
  copy(tasks_, tasks);
  copy(lists_, lists);
  CUDA_CHECK(cudaMemsetAsync(state_, 0, kDirectWords * sizeof(int), st));
}

void DirectSystem::factorize(const double* Lvals, const float* dyn, const int* skip,
                             cudaStream_t st) {
  DirectFactorArgs a;
  a.nodes = nodes_;
  a.ids = ids_;
  a.cmap = cmap_;
  a.ent_src = ent_src_;
  a.ent_dst = ent_dst_;
  a.diag_id = diag_id_;
  a.diag_dst = diag_dst_;
  a.Lvals = Lvals;
  a.dyn = dyn;
  a.V = V_;
  a.W = W_;
  a.P = P_;
  a.Gd = Gd_;
  a.G = G_;
  a.T = T_;
  a.state = state_;
  a.skip = skip;
  ++factorisations_;
  launch_direct_begin(state_, barrier_, skip, st);
  for (int l = (int)levels_.size() - 1; l >= 0; --l) {
    const Level& L = levels_[l];
    a.F = fronts_[l & 1];
    a.Fc = fronts_[(l + 1) & 1];
    CUDA_CHECK(cudaMemsetAsync(a.F, 0, (size_t)L.front * sizeof(double), st));
    launch_direct_fill(a, L.ent0, L.ent1, L.diag0, L.diag1, st);
    for (int s = 0; s < 4; ++s)
      launch_direct_add(a, nodes_, lists_ + L.add[s], L.adds[s], st);
    for (int k = 0; k < L.steps; ++k) {
      launch_direct_panel(a, lists_ + L.panel_task, L.panel_tasks, k, st);
      launch_direct_update(a, lists_ + L.tile, L.tiles, k, st);
    }
    launch_direct_store(a, lists_ + L.store, L.stores, st);
    launch_direct_products(a, lists_ + L.product, L.products, lists_ + L.schur, L.schurs, st);
  }
}

void DirectSystem::solve(const CgArgs& cg, int* failed, cudaStream_t st) {
  DirectArgs a = args_;
  a.nslices = cg.nslices;
  a.sl_ptr = cg.sl_ptr;
  a.sl_w = cg.sl_w;
  a.ent = cg.ent;
  a.Ldiag = cg.Ldiag;
  a.dyn = cg.dyn;
  a.b = cg.b;
  a.x = cg.x;
  a.fail = cg.fail;
  a.stats = cg.stats;
  a.failed = failed;
  a.skip = cg.skip;
  a.rel_tol_dev = cg.rel_tol_dev;
  a.rel_tol = cg.rel_tol;
  a.abs_tol = cg.abs_tol;
  a.barrier_spin_limit = cg.barrier_spin_limit;
  a.withhold_block = cg.withhold_block;
  launch_direct_solve(a, blocks_, smem_, st);
}

}  // namespace silkb
