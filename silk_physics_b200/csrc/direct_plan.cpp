// Nested dissection, symbolic factorisation and index plans of the direct
// ADMM solve (no reference counterpart: the reference solves every ADMM
// iteration by MAS-CG, mas_cg_solver.cu:193-311).
#include "direct_plan.hpp"

#include <algorithm>
#include <cmath>
#include <utility>

namespace silkb {

namespace {

// Regions of at most this many vertices are leaves: the mean size of a region
// some quartings deep, with room for uneven ones, so that (nearly) all leaves
// lie on one level.  Small systems are bound by the number of levels (two
// grid barriers each and application), large ones by the bytes of the
// factors, which small leaves keep low.
int leaf_limit(int nv) {
  if (nv <= 256) return 256;
  const double target = nv <= 20000 ? 100.0 : 45.0;
  double mean = nv;
  while (mean > target) mean *= 0.25;
  return (int)(1.3 * mean) + 1;
}

// Fronts above this need more time to factorise than the CG iterations they
// replace (a well shaped sheet of a million vertices stays below).
constexpr int kMaxFront = 12000;
constexpr int kMaxEntriesPerVertex = 3000;

struct Builder {
  int nv;
  const std::vector<int>& rows;
  const std::vector<int>& cols;
  const std::vector<float>& pos;
  std::vector<int> side;  // scratch: the vertex's side of the current cut, or -1
  std::vector<std::pair<float, int>> line;  // scratch: the region along the cut axis
  std::vector<float> reach;  // per vertex and axis: (just over) the farthest entry's distance
  struct Region {
    std::vector<int> own;
    int parent, slot, level;
  };
  std::vector<Region> regions;  // parents before children

  // Splits `set` along its longest extent into two parts without a matrix
  // entry between them and the separator that was removed to get there.
  void bisect(std::vector<int>& set, std::vector<int>& a, std::vector<int>& b,
              std::vector<int>& sep) {
    int axis = 0;
    float best = -1.0f;
    for (int d = 0; d < 3; ++d) {
      float lo = pos[3 * set[0] + d], hi = lo;
      for (int v : set) {
        lo = std::min(lo, pos[3 * v + d]);
        hi = std::max(hi, pos[3 * v + d]);
      }
      if (hi - lo > best) {
        best = hi - lo;
        axis = d;
      }
    }
    // Cut near the middle where the coordinate jumps: between two mesh lines
    // rather than inside one, whose noise would fray the separator.  Only the
    // middle third has to be in order for that.
    const int n = (int)set.size(), w = n / 6;
    const int lo = std::max(1, n / 2 - w), hi = std::min(n - 1, n / 2 + w);
    line.resize(n);
    for (int i = 0; i < n; ++i) line[i] = {pos[3 * set[i] + axis], set[i]};
    std::nth_element(line.begin(), line.begin() + lo - 1, line.end());
    std::nth_element(line.begin() + lo, line.begin() + hi, line.end());
    std::sort(line.begin() + lo, line.begin() + hi);
    auto gap = [&](int i) { return line[i].first - line[i - 1].first; };
    float gmax = 0.0f;
    for (int i = lo; i <= hi; ++i) gmax = std::max(gmax, gap(i));
    int cut = n / 2;
    for (int d = 0; d <= w; ++d) {
      bool found = false;
      for (int i : {n / 2 - d, n / 2 + d})
        if (!found && i >= lo && i <= hi && gap(i) >= 0.5f * gmax) {
          cut = i;
          found = true;
        }
      if (found) break;
    }
    for (int i = 0; i < n; ++i) set[i] = line[i].second;
    for (int i = 0; i < n; ++i) side[set[i]] = i < cut ? 0 : 1;
    // A vertex whose entries all end before the cut touches nothing beyond.
    const float first = line[cut].first, last = line[cut - 1].first;
    auto touches = [&](int v, int other) {
      const float x = pos[3 * v + axis];
      if (other == 1 ? x + reach[3 * v + axis] < first : x - reach[3 * v + axis] > last)
        return false;
      for (int k = rows[v]; k < rows[v + 1]; ++k)
        if (side[cols[k]] == other) return true;
      return false;
    };
    std::vector<int> s0, s1;
    for (int i = 0; i < cut; ++i)
      if (touches(set[i], 1)) s0.push_back(set[i]);
    for (int i = cut; i < n; ++i)
      if (touches(set[i], 0)) s1.push_back(set[i]);
    sep = s0.size() < s1.size() ? s0 : s1;
    for (int v : sep) side[v] = 2;
    a.clear();
    b.clear();
    for (int v : set) {
      if (side[v] == 0) a.push_back(v);
      if (side[v] == 1) b.push_back(v);
    }
    for (int v : set) side[v] = -1;
  }

  // Two bisections per tree level: own = both cuts' separators, up to four
  // children.
  void dissect(std::vector<int> set, int parent, int slot, int level, int leaf) {
    const int me = (int)regions.size();
    regions.push_back({{}, parent, slot, level});
    if ((int)set.size() <= leaf) {
      regions[me].own = std::move(set);
      return;
    }
    std::vector<int> half[2], own;
    bisect(set, half[0], half[1], own);
    std::vector<std::vector<int>> parts;
    for (auto& h : half) {
      if ((int)h.size() <= leaf) {
        if (!h.empty()) parts.push_back(std::move(h));
        continue;
      }
      std::vector<int> x, y, s;
      bisect(h, x, y, s);
      own.insert(own.end(), s.begin(), s.end());
      for (auto* p : {&x, &y})
        if (!p->empty()) parts.push_back(std::move(*p));
    }
    set = std::vector<int>();
    regions[me].own = std::move(own);
    for (int i = 0; i < (int)parts.size(); ++i)
      dissect(std::move(parts[i]), me, i, level + 1, leaf);
  }
};

}  // namespace

bool build_direct_plan(int nv, const std::vector<int>& rows, const std::vector<int>& cols,
                       const std::vector<float>& pos, DirectPlan& P) {
  P = DirectPlan{};
  if (nv <= 0) return false;
  Builder B{nv, rows, cols, pos, std::vector<int>(nv, -1), {}, {}, {}};
  B.reach.assign(3 * (size_t)nv, 0.0f);
  for (int v = 0; v < nv; ++v)
    for (int d = 0; d < 3; ++d) {
      float far = 0.0f;
      for (int k = rows[v]; k < rows[v + 1]; ++k)
        far = std::max(far, std::fabs(pos[3 * cols[k] + d] - pos[3 * v + d]));
      B.reach[3 * v + d] = far + 1e-5f * (far + std::fabs(pos[3 * v + d]));
    }
  {
    std::vector<int> all(nv);
    for (int i = 0; i < nv; ++i) all[i] = i;
    B.dissect(std::move(all), -1, 0, 0, leaf_limit(nv));
  }
  const int nr = (int)B.regions.size();
  int levels = 0;
  for (auto& r : B.regions) levels = std::max(levels, r.level + 1);
  // Elimination order: children before their parent (regions are listed
  // parent first, so the reverse of that list is one).
  std::vector<int> order(nv), owner(nv), vertex(nv);
  int next = 0;
  for (int k = nr - 1; k >= 0; --k) {
    std::sort(B.regions[k].own.begin(), B.regions[k].own.end());
    for (int v : B.regions[k].own) {
      vertex[next] = v;
      order[v] = next++;
      owner[v] = k;
    }
  }
  // Boundaries in elimination order, children first: every later vertex that
  // the own vertices or the children's boundaries touch.
  std::vector<std::vector<int>> bnd(nr), kids(nr);
  for (int k = 1; k < nr; ++k) kids[B.regions[k].parent].push_back(k);
  std::vector<int> mark(nv, -1);
  for (int k = nr - 1; k >= 0; --k) {
    auto add = [&](int v) {
      if (mark[v] == k || owner[v] >= k) return;  // own, or inside the region
      mark[v] = k;
      bnd[k].push_back(order[v]);
    };
    for (int v : B.regions[k].own)
      for (int q = rows[v]; q < rows[v + 1]; ++q) add(cols[q]);
    for (int c : kids[k])
      for (int v : bnd[c]) add(v);
    std::sort(bnd[k].begin(), bnd[k].end());
    for (int& v : bnd[k]) v = vertex[v];
  }
  // Nodes by level.
  std::vector<int> index(nr);
  P.level_off.assign(1, 0);
  for (int l = 0; l < levels; ++l) {
    int64_t front = 0;
    int panel = 0;
    for (int k = 0; k < nr; ++k) {
      if (B.regions[k].level != l) continue;
      index[k] = (int)P.nodes.size();
      DirectNode n;
      n.m = (int)B.regions[k].own.size();
      n.b = (int)bnd[k].size();
      n.level = l;
      n.parent = B.regions[k].parent < 0 ? -1 : index[B.regions[k].parent];
      n.slot = B.regions[k].slot;
      n.ids = (int)P.ids.size();
      n.u = P.u_total;
      n.front = front;
      n.panel = panel;
      n.ms = (n.m + 3) / 4 * 4;
      n.bs = (n.b + 3) / 4 * 4;
      n.g = P.g_total;
      n.t = P.t_total;
      const int64_t N = n.m + n.b;
      if (N > kMaxFront) {
        P = DirectPlan{};
        return false;
      }
      front += N * N;
      panel += (int)N;
      P.u_total += n.b;
      P.g_total += (int64_t)n.m * n.bs;
      P.t_total += N * n.ms;
      P.ids.insert(P.ids.end(), B.regions[k].own.begin(), B.regions[k].own.end());
      P.ids.insert(P.ids.end(), bnd[k].begin(), bnd[k].end());
      P.nodes.push_back(n);
    }
    P.level_off.push_back((int)P.nodes.size());
    P.level_front.push_back(front);
    P.level_panel.push_back(panel);
    if (front >= (int64_t(1) << 31) - 1 ||
        P.t_total + P.g_total > (int64_t)kMaxEntriesPerVertex * nv) {
      P = DirectPlan{};
      return false;
    }
  }
  // Positions of boundaries in the parents' fronts, and what is summed where:
  // a front entry receives at most one update of each of its (up to four)
  // children.
  P.cmap.assign(P.u_total, 0);
  P.gat.assign(4 * P.ids.size(), -1);
  std::vector<int> place(nv, -1);
  std::vector<std::vector<int>> children(P.nodes.size());
  for (int i = 1; i < (int)P.nodes.size(); ++i) children[P.nodes[i].parent].push_back(i);
  for (int i = 0; i < (int)P.nodes.size(); ++i) {
    const DirectNode& n = P.nodes[i];
    for (int q = 0; q < n.m + n.b; ++q) place[P.ids[n.ids + q]] = q;
    for (int c : children[i]) {
      const DirectNode& ch = P.nodes[c];
      for (int j = 0; j < ch.b; ++j) {
        const int at = place[P.ids[ch.ids + ch.m + j]];
        P.cmap[ch.u + j] = at;
        int* g = &P.gat[4 * (size_t)(n.ids + at)];
        while (*g >= 0) ++g;
        *g = ch.u + j;
      }
    }
  }
  P.ent_src.reserve(cols.size() / 2 + nv);
  P.ent_dst.reserve(cols.size() / 2 + nv);
  P.diag_id.reserve(nv);
  P.diag_dst.reserve(nv);
  // Matrix entries: row of an own vertex, the columns at or after it in the
  // front (upper triangle); each entry of A falls in exactly one front.
  P.ent_off.assign(1, 0);
  P.diag_off.assign(1, 0);
  for (int l = 0; l < levels; ++l) {
    for (int i = P.level_off[l]; i < P.level_off[l + 1]; ++i) {
      const DirectNode& n = P.nodes[i];
      const int64_t N = n.m + n.b;
      const int first = n.m ? order[P.ids[n.ids]] : 0;
      for (int q = 0; q < n.m + n.b; ++q) place[P.ids[n.ids + q]] = q;
      for (int q = 0; q < n.m; ++q) {
        const int v = P.ids[n.ids + q];
        for (int k = rows[v]; k < rows[v + 1]; ++k) {
          const int c = cols[k];
          if (order[c] < first || place[c] < q) continue;
          P.ent_src.push_back(k);
          P.ent_dst.push_back((int)(n.front + q * N + place[c]));
        }
        P.diag_id.push_back(v);
        P.diag_dst.push_back((int)(n.front + q * N + q));
      }
    }
    P.ent_off.push_back((int)P.ent_src.size());
    P.diag_off.push_back((int)P.diag_id.size());
  }
  return true;
}

}  // namespace silkb
