// dof_schedule.cu — host-side builder of the level schedule that the LM kernel uses to
// factor J^T J + damp I over the DOF tree (br_tree_t.dof_sched; layout in br_b200.h).
//
// The reference solves each LM step with a dense Cholesky of the full nv x nv normal
// matrix (src/better_robot/optim/optimizers/levenberg_marquardt.py:95-97 through
// optim/solvers/cholesky.py:14-18).  J^T J of a kinematic tree is sparse: columns c and c'
// interact only when one is an ancestor of the other in the DOF tree, so eliminating
// leaves first creates no fill-in.  This file lays that elimination out in levels of
// independent DOFs so that one team of lanes runs a whole level between two
// synchronisations (13 levels instead of 36 pivots for a floating-base humanoid).  The kernel reads
// the row schedule: a row's entries are consecutive, and every entry of row i that DOF k updates takes
// the same factor l_ki, so a task is four entries of one row (humanoid: 211 tasks
// in 10 passes of 32 lanes below the trunk, then its 27 entries, instead of 977 and 621 further
// contributions in 37).
#include <stdint.h>

#include <algorithm>
#include <unordered_map>
#include <vector>

#include "../../include/br_b200.h"

namespace {

struct Contrib {
  uint32_t a, b, d;
};

}  // namespace

extern "C" int64_t br_dof_schedule(const int32_t* dof_parent, int32_t nv, uint32_t* out, int64_t capacity) {
  if (nv < 0 || nv > BR_MAX_NV || (nv > 0 && !dof_parent) || capacity < 0) return BR_EINVAL;
  std::vector<int> dep(nv), rowoff(nv + 1), height(nv, 0);
  std::vector<std::vector<int>> anc(nv);  // ancestors of c by depth (root first)
  int nl = 0;
  for (int c = 0; c < nv; ++c) {
    const int p = dof_parent[c];
    if (p < -1 || p >= c) return BR_EINVAL;
    dep[c] = p < 0 ? 0 : dep[p] + 1;
    if (p >= 0) {
      anc[c] = anc[p];
      anc[c].push_back(p);
    }
    rowoff[c] = nl;
    nl += dep[c] + 1;
  }
  rowoff[nv] = nl;
  if (nl + nv > 0xffff) return BR_ETOOBIG;
  for (int c = nv - 1; c >= 0; --c)
    if (dof_parent[c] >= 0) height[dof_parent[c]] = std::max(height[dof_parent[c]], height[c] + 1);
  int levels = 0, depth_levels = 0;
  for (int c = 0; c < nv; ++c) {
    levels = std::max(levels, height[c] + 1);
    depth_levels = std::max(depth_levels, dep[c] + 1);
  }
  const uint32_t zoff = (uint32_t)nl;  // right-hand-side slots follow the packed rows

  std::vector<uint32_t> starts;
  std::vector<uint32_t> tasks;   // 4 words each
  std::vector<uint32_t> extras;  // 2 words each
  for (int lev = 0; lev < levels; ++lev) {
    starts.push_back((uint32_t)(tasks.size() / 4));
    std::vector<std::pair<uint32_t, std::vector<Contrib>>> groups;
    std::unordered_map<uint32_t, size_t> where;
    auto add = [&](uint32_t dst, Contrib c) {
      auto it = where.find(dst);
      if (it == where.end()) {
        where.emplace(dst, groups.size());
        groups.push_back({dst, {c}});
      } else {
        groups[it->second].second.push_back(c);
      }
    };
    for (int k = nv - 1; k >= 0; --k) {  // descending DOF index: the one-at-a-time order
      if (height[k] != lev) continue;
      const uint32_t rk = (uint32_t)rowoff[k], d = (uint32_t)k;
      for (int a = 0; a < dep[k]; ++a)
        for (int b = 0; b <= a; ++b) add((uint32_t)(rowoff[anc[k][a]] + b), {rk + a, rk + b, d});
      for (int a = 0; a < dep[k]; ++a) add(zoff + (uint32_t)anc[k][a], {rk + a, zoff + (uint32_t)k, d});
    }
    // entries with several contributions first, so that they spread over the lanes
    std::stable_sort(groups.begin(), groups.end(),
                     [](const auto& x, const auto& y) { return x.second.size() > y.second.size(); });
    for (const auto& g : groups) {
      const uint32_t n_extra = (uint32_t)g.second.size() - 1, first = (uint32_t)(extras.size() / 2);
      if (n_extra > 0xffff || first + n_extra > 0xffff) return BR_ETOOBIG;
      const Contrib& c0 = g.second[0];
      tasks.insert(tasks.end(), {g.first | (n_extra << 16), c0.a | (c0.b << 16), c0.d | (first << 16), 0u});
      for (size_t e = 1; e < g.second.size(); ++e) {
        const Contrib& c = g.second[e];
        extras.insert(extras.end(), {c.a | (c.b << 16), c.d});
      }
    }
  }
  const uint32_t n_tasks = (uint32_t)(tasks.size() / 4);
  starts.push_back(n_tasks);
  // the last task that updates DOF k's diagonal finalises its pivot: flag it (word 3 = k + 1)
  // so that the lane running it also stores 1 / (pivot + damp) for the levels above
  std::vector<int64_t> last(nv, -1);
  for (uint32_t p = 0; p < n_tasks; ++p) {
    const int dst = (int)(tasks[4 * p] & 0xffff);
    if (dst >= nl) continue;
    const int k = (int)(std::upper_bound(rowoff.begin(), rowoff.begin() + nv, dst) - rowoff.begin()) - 1;
    if (dst == rowoff[k] + dep[k]) last[k] = p;
  }
  for (int k = 0; k < nv; ++k)
    if (last[k] >= 0) tasks[4 * last[k] + 3] = (uint32_t)k + 1;
  // the last further contribution is no contribution but the mark of a table with a row section, and the
  // table's length (filled in below)
  extras.insert(extras.end(), {BR_DOF_SCHED_MARK, 0u});
  const int64_t toff = ((5 + (int64_t)levels) + 3) & ~(int64_t)3;
  const int64_t entry_words = toff + (int64_t)tasks.size() + (int64_t)extras.size();

  // ---- the row schedule: the same levels, one task per four entries of an updated row ----
  std::vector<int> ro(nv + 1);  // row c: right-hand side, then its entries by depth, padded to pairs
  int nr = 0;
  for (int c = 0; c < nv; ++c) {
    ro[c] = nr;
    nr += (dep[c] + 3) & ~1;
  }
  ro[nv] = nr;
  // trunk: the largest n <= 6 such that DOFs 0..n-1 form a chain from the root and every other DOF
  // descends from DOF n - 1.  Its rows are updated by every other DOF and are read by none of them: they
  // wait until the levels below are done, then take all their contributions in one sweep (trunk_from, in
  // the levels' order) and are eliminated in registers.
  int ntr = 0;
  for (int n = std::min(nv, 6); n >= 2 && ntr == 0; --n) {
    bool ok = true;
    for (int c = 0; c < nv && ok; ++c) ok = c < n ? dep[c] == c : (dep[c] >= n && anc[c][n - 1] == n - 1);
    if (ok) ntr = n;
  }
  const int blevels = levels - ntr;
  std::vector<uint32_t> rstarts, rtasks, rextras, trunk_from;
  for (int lev = 0; lev < blevels; ++lev) {
    for (int k = nv - 1; k >= ntr && ntr > 0; --k)
      if (height[k] == lev) trunk_from.push_back((uint32_t)ro[k] | ((uint32_t)k << 16));
    rstarts.push_back((uint32_t)(rtasks.size() / 4));
    struct Chunk {
      int row, p0;
      std::vector<uint32_t> from;  // soff | k << 16, descending k: the one-at-a-time order
    };
    std::vector<Chunk> chunks;
    std::unordered_map<int, size_t> where;  // first entry of the chunk -> its index
    for (int k = nv - 1; k >= 0; --k) {
      if (height[k] != lev) continue;
      for (int a = ntr; a < dep[k]; ++a) {
        const int row = anc[k][a];
        for (int p0 = 0; p0 < a + 2; p0 += 4) {
          const int dst = ro[row] + p0;
          auto it = where.find(dst);
          if (it == where.end()) {
            it = where.emplace(dst, chunks.size()).first;
            chunks.push_back({row, p0, {}});
          }
          chunks[it->second].from.push_back((uint32_t)(ro[k] + 1 + a) | ((uint32_t)k << 16));
        }
      }
    }
    std::stable_sort(chunks.begin(), chunks.end(),
                     [](const Chunk& x, const Chunk& y) { return x.from.size() > y.from.size(); });
    for (const Chunk& c : chunks) {
      const int a = dep[c.row];
      const uint32_t delta = (uint32_t)(1 + a - c.p0);          // the row's diagonal, from the chunk's start
      const bool two = c.p0 + 2 < a + 2;                        // a second pair of entries
      const bool last = delta < 4 && height[c.row] == lev + 1;  // the diagonal's last update
      const uint32_t first = (uint32_t)rextras.size();
      if (first > 0xffff || c.from.size() > 0xff) return BR_ETOOBIG;
      rtasks.insert(rtasks.end(), {(uint32_t)(ro[c.row] + c.p0) | (delta << 16) | ((uint32_t)c.from.size() << 24),
                                   c.from[0], first | ((last ? (uint32_t)c.row + 1 : 0u) << 16) | (two ? 1u << 31 : 0u),
                                   c.from.size() > 1 ? c.from[1] : 0u});
      for (size_t e = 2; e < c.from.size(); ++e) rextras.push_back(c.from[e]);
      if (rextras.size() & 1) rextras.push_back(0u);            // read in pairs
    }
  }
  rstarts.push_back((uint32_t)(rtasks.size() / 4));
  const int64_t roff = (entry_words + 3) & ~(int64_t)3, rtoff = roff + toff;
  const int64_t words = rtoff + (int64_t)(rtasks.size() + rextras.size() + trunk_from.size());
  extras.back() = (uint32_t)words;
  if (out && capacity >= words) {
    std::fill(out, out + toff, 0u);
    out[0] = (uint32_t)levels;
    out[1] = n_tasks;
    out[2] = (uint32_t)(extras.size() / 2);
    out[3] = (uint32_t)depth_levels;
    std::copy(starts.begin(), starts.end(), out + 4);
    std::copy(tasks.begin(), tasks.end(), out + toff);
    std::copy(extras.begin(), extras.end(), out + toff + tasks.size());
    std::fill(out + entry_words, out + rtoff, 0u);
    out[roff] = (uint32_t)(rtasks.size() / 4);
    out[roff + 1] = (uint32_t)rextras.size();
    out[roff + 2] = (uint32_t)blevels | ((uint32_t)ntr << 16);
    out[roff + 3] = (uint32_t)nr;
    std::copy(rstarts.begin(), rstarts.end(), out + roff + 4);
    std::copy(rtasks.begin(), rtasks.end(), out + rtoff);
    std::copy(rextras.begin(), rextras.end(), out + rtoff + rtasks.size());
    std::copy(trunk_from.begin(), trunk_from.end(), out + rtoff + rtasks.size() + rextras.size());
  }
  return words;
}
