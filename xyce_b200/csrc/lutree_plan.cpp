// Elimination-tree plan (lutree.h), built once per pivot order on the host.
#include "lutree.h"

#include <algorithm>
#include <climits>
#include <functional>
#include <queue>

namespace {

// A subtree with at most this many updates is a bottom subtree. Larger: fewer and shorter chains and
// fewer joins, but taller subtrees, whose levels cost a block barrier each. Refactorization + solve in
// us at 3,000 / 10,000 / 30,000 / 100,000 updates:
//     2.8k unknowns,  74k updates in all    90+60    90+65   102+82   188+149
//     7.8k           252k                  131+97   110+92   143+138  193+156
//     4.5k (any net) 413k                  164+82   162+84   139+83   170+106
//     12k            518k                  202+134  148+112  176+152  242+193
//     24k            1.2M                  367+225  265+175  254+185  319+230
//     41k            2.0M                  398+237  281+181  275+211  348+246
//     200k           12.6M                1732+916 1350+740 1088+630 1085+638
// A matrix with few updates has no use for tall subtrees. The line at 300k is right for what lies below
// it and for netlists wired any to any; placed ones between it and a million updates would be up to a
// fifth faster with the smaller limit.
constexpr double kTopWork = 30000, kTopWorkSmall = 10000, kSmallMatrix = 300000, kNoPlan = 5000;
constexpr int kTopHeight = 64;  // nor with more levels than this
constexpr size_t kLongRow = 256;  // entries of a bottom row that one warp sums in a solve
constexpr int kGroups = 296;  // two blocks for each of 148 SMs walk the bottom subtrees

}  // namespace

bool xd_tree_plan(int n, const std::vector<int> &mp, const std::vector<int> &mi, const std::vector<int> &mdiag,
                  XdTreePlan *plan) {
  XdTreePlan &t = *plan;
  t = XdTreePlan();
  t.n = n;
  const int nnz = mp[n];
  // L's columns (rows below each pivot, ascending, with positions) and U's column counts.
  std::vector<int> lcp(n + 1, 0), ucc(n, 0);
  for (int i = 0; i < n; ++i)
    for (int e = mp[i]; e < mp[i + 1]; ++e) {
      if (mi[e] < i) ++lcp[mi[e] + 1];
      if (mi[e] > i) ++ucc[mi[e]];
    }
  for (int k = 0; k < n; ++k) lcp[k + 1] += lcp[k];
  std::vector<int> lci(lcp[n]), lcpos(lcp[n]);
  {
    std::vector<int> fl(lcp.begin(), lcp.end() - 1);
    for (int i = 0; i < n; ++i)
      for (int e = mp[i]; e < mdiag[i]; ++e) {
        lci[fl[mi[e]]] = i;
        lcpos[fl[mi[e]]++] = e;
      }
  }
  auto lcount = [&](int k) { return lcp[k + 1] - lcp[k]; };
  auto ucount = [&](int k) { return mp[k + 1] - mdiag[k] - 1; };
  // Fronts: struct(k) = k's own adjacency and its children's, ascending. An update-free pivot's own
  // adjacency may be left out where solving needs no order for it: with an empty U row and an empty
  // L row its solved value is known from the start, whoever reads it; with an empty L column and an
  // empty U column nobody reads its value, and its row can be solved last.
  auto loose = [&](int k) {
    return (ucount(k) == 0 && mdiag[k] == mp[k]) || (lcount(k) == 0 && ucc[k] == 0);
  };
  std::vector<std::vector<int>> st(n);
  std::vector<int> parent(n, -1), height(n, 0), mark(n, -1);
  std::vector<double> work(n, 0.0);
  std::vector<int> child(n, -1), sibling(n, -1);
  long long total = 0;
  for (int k = 0; k < n; ++k) {
    std::vector<int> &s = st[k];
    auto add = [&](int j) {
      if (j != k && mark[j] != k) {
        mark[j] = k;
        s.push_back(j);
      }
    };
    if (!loose(k)) {
      for (int e = lcp[k]; e < lcp[k + 1]; ++e) add(lci[e]);
      for (int e = mdiag[k] + 1; e < mp[k + 1]; ++e) add(mi[e]);
      work[k] += (double)lcount(k) * ucount(k);
    }
    for (int c = child[k]; c >= 0; c = sibling[c]) {
      for (int j : st[c]) add(j);
      height[k] = std::max(height[k], height[c] + 1);
      work[k] += work[c];
    }
    std::sort(s.begin(), s.end());
    total += (long long)s.size();
    if (2 * total > (long long)nnz + nnz / 2 + 64) return false;  // the symmetrised pattern fills in
    if (!s.empty()) {
      parent[k] = s[0];
      sibling[k] = child[s[0]];
      child[s[0]] = k;
    }
  }
  auto in_front = [&](int k, int j) { return std::binary_search(st[k].begin(), st[k].end(), j); };
  std::vector<char> last(n, 0);
  for (int k = 0; k < n; ++k)
    if (loose(k))
      for (int e = mdiag[k] + 1; e < mp[k + 1]; ++e)
        if (!in_front(k, mi[e])) last[k] = 1;
  std::vector<char> top(n, 0);
  double all = 0.0;
  for (int k = 0; k < n; ++k)
    if (parent[k] < 0) all += work[k];
  // A few thousand updates in all: one block of level lists is as fast (1.1k unknowns, 2.2k updates:
  // 58.6 + 42.2 us a refactorization and solve, 58.2 + 46.7 us over the plan).
  if (all < kNoPlan) return false;
  const double top_work = all < kSmallMatrix ? kTopWorkSmall : kTopWork;
  for (int k = 0; k < n; ++k) {
    top[k] = work[k] > top_work || height[k] >= kTopHeight;
    t.ntop += top[k];
    if (top[k] && (int)st[k].size() >= kMaxFrame) return false;
  }
  t.nbot = n - t.ntop;

  // Bottom groups: subtrees dealt to the least loaded group, heaviest first.
  std::vector<int> roots, size(n, 1);
  for (int k = 0; k < n; ++k)
    if (parent[k] >= 0) size[parent[k]] += size[k];
  for (int k = 0; k < n; ++k)
    if (!top[k] && (parent[k] < 0 || top[parent[k]])) roots.push_back(k);
  std::vector<int> group(n, -1);
  {
    auto weight = [&](int k) { return work[k] + 8.0 * size[k]; };
    std::vector<int> by(roots);
    std::sort(by.begin(), by.end(), [&](int a, int b) { return weight(a) != weight(b) ? weight(a) > weight(b) : a < b; });
    t.ngroups = std::min((int)by.size(), kGroups);
    std::priority_queue<std::pair<double, int>, std::vector<std::pair<double, int>>, std::greater<std::pair<double, int>>> q;
    for (int g = 0; g < t.ngroups; ++g) q.push({0.0, g});
    for (int r : by) {
      auto least = q.top();
      q.pop();
      group[r] = least.second;
      q.push({least.first + weight(r), least.second});
    }
    for (int k = n - 1; k >= 0; --k)
      if (!top[k] && group[k] < 0) group[k] = group[parent[k]];
  }
  std::vector<int> bottom;
  for (int k = 0; k < n; ++k)
    if (!top[k]) bottom.push_back(k);
  std::stable_sort(bottom.begin(), bottom.end(), [&](int a, int b) {
    return group[a] != group[b] ? group[a] < group[b] : height[a] < height[b];
  });
  t.order = bottom;
  t.glev.assign(1, 0);
  t.lrow.assign(1, 0);
  for (int b = 0, g = 0; g < t.ngroups; ++g) {
    while (b < t.nbot && group[bottom[b]] == g) {
      const int h = height[bottom[b]];
      while (b < t.nbot && group[bottom[b]] == g && height[bottom[b]] == h) ++b;
      t.lrow.push_back(b);
    }
    t.glev.push_back((int)t.lrow.size() - 1);
  }

  // Chains: each top pivot continues the chain of its tallest top child; chains in the order of their
  // last pivots' heights, so that a chain comes after those that join it.
  std::vector<int> heavy(n, -1), panel(n, -1);
  for (int k = 0; k < n; ++k)
    if (top[k] && parent[k] >= 0) {
      int &h = heavy[parent[k]];
      if (h < 0 || height[k] > height[h]) h = k;
    }
  std::vector<int> ends;
  for (int k = 0; k < n; ++k)
    if (top[k] && (parent[k] < 0 || heavy[parent[k]] != k)) ends.push_back(k);
  std::sort(ends.begin(), ends.end(), [&](int a, int b) { return height[a] != height[b] ? height[a] < height[b] : a < b; });
  t.nchains = (int)ends.size();
  t.cptr.assign(1, 0);
  std::vector<int> chain_of(n, -1), nodes;
  for (int c = 0; c < t.nchains; ++c) {
    const size_t b = nodes.size();
    for (int k = ends[c]; k >= 0; k = heavy[k]) {
      nodes.push_back(k);
      chain_of[k] = c;
    }
    std::reverse(nodes.begin() + b, nodes.end());
    t.cptr.push_back((int)nodes.size());
  }
  for (int p = 0; p < t.ntop; ++p) panel[nodes[p]] = p;
  t.order.insert(t.order.end(), nodes.begin(), nodes.end());
  // Slots: a variable takes the lowest free slot when its chain's front first holds it and keeps it
  // to the end of its own block. slot[p]: the pivot's; sl[p]: those of struct(nodes[p]), aligned with it.
  std::vector<int> slot(t.ntop), where(n, -1);
  std::vector<std::vector<unsigned char>> sl(t.ntop);
  std::vector<XdPos2> left;  // (slot, variable) of each chain's border
  std::vector<int> left_ptr(1, 0);
  t.bptr.assign(1, 0);
  int frame = 0;
  for (int c = 0; c < t.nchains; ++c) {
    std::priority_queue<int, std::vector<int>, std::greater<int>> free_slots, used;
    for (int s = 0; s < kMaxFrame; ++s) free_slots.push(s);
    std::vector<int> live;
    auto enter = [&](int j) {
      if (where[j] < 0) {
        if (free_slots.empty()) return -1;
        where[j] = free_slots.top();
        free_slots.pop();
        live.push_back(j);
      }
      return where[j];
    };
    for (int p = t.cptr[c]; p < t.cptr[c + 1]; p += kBlockPivots) {
      const int pe = std::min(p + kBlockPivots, t.cptr[c + 1]);
      for (int x = p; x < pe; ++x) {
        if ((slot[x] = enter(nodes[x])) < 0) return false;
        for (int j : st[nodes[x]]) {
          const int s = enter(j);
          if (s < 0) return false;
          sl[x].push_back((unsigned char)s);
        }
      }
      int r = 0;
      for (int j : live) r = std::max(r, where[j] + 1);
      frame = std::max(frame, r);
      for (int x = p; x < p + kBlockPivots; ++x) t.blocks.push_back(x < pe ? slot[x] : kNoPivot);
      t.blocks.insert(t.blocks.end(), {r, 0, 0, 0});
      size_t kept = 0;
      for (int j : live) {
        if (chain_of[j] == c && panel[j] < pe) {
          free_slots.push(where[j]);
          where[j] = -1;
        } else {
          live[kept++] = j;
        }
      }
      live.resize(kept);
    }
    for (int j : live) {
      left.push_back({where[j], j});
      where[j] = -1;
    }
    left_ptr.push_back((int)left.size());
    t.bptr.push_back((int)t.blocks.size() / kBlockInts);
  }
  t.F = std::max(16, (frame + 15) / 16 * 16);
  // Panels hold whole frames: a matrix of long thin paths (a tridiagonal one) would waste them.
  if (2.0 * t.F * t.ntop > 16.0 * nnz + 65536.0) return false;
  // Joins, at the start of the block that holds the child's parent pivot.
  t.jmap.assign((size_t)t.nchains * t.F, (unsigned char)kJoinNone);
  auto block_of = [&](int p) { return t.bptr[chain_of[nodes[p]]] + (p - t.cptr[chain_of[nodes[p]]]) / kBlockPivots; };
  {
    const int nblocks = t.bptr[t.nchains];
    std::vector<int> jptr(nblocks + 1, 0);
    for (int c = 0; c < t.nchains; ++c)
      if (parent[ends[c]] >= 0) ++jptr[block_of(panel[parent[ends[c]]]) + 1];
    for (int x = 0; x < nblocks; ++x) {
      jptr[x + 1] += jptr[x];
      t.blocks[(size_t)x * kBlockInts + kBlockPivots + 1] = jptr[x];
      t.blocks[(size_t)x * kBlockInts + kBlockPivots + 2] = jptr[x + 1];
    }
    t.jchild.assign(jptr[nblocks], 0);
    for (int c = 0; c < t.nchains; ++c) {
      const int e = ends[c], k = parent[e];
      if (k < 0) continue;
      const int p = panel[k], pe = panel[e];
      t.jchild[jptr[block_of(p)]++] = c;
      for (size_t x = 0; x < st[e].size(); ++x) {
        const int j = st[e][x];
        int ps = slot[p];
        if (j != k) {
          const size_t y = std::lower_bound(st[k].begin(), st[k].end(), j) - st[k].begin();
          if (y >= st[k].size() || st[k][y] != j) return false;
          ps = sl[p][y];
        }
        t.jmap[(size_t)c * t.F + ps] = sl[pe][x];
      }
    }
  }

  // Positions in V.
  std::vector<int> place(n);
  for (int x = 0; x < n; ++x) place[t.order[x]] = x;
  t.border.assign((size_t)t.nchains * t.F, -1);
  for (int c = 0; c < t.nchains; ++c)
    for (int x = left_ptr[c]; x < left_ptr[c + 1]; ++x) t.border[(size_t)c * t.F + left[x].x] = place[left[x].y];
  auto panel_slot = [&](int k, int j) {  // slot of j at pivot k, or -1 outside its front
    if (j == k) return slot[panel[k]];
    const size_t y = std::lower_bound(st[k].begin(), st[k].end(), j) - st[k].begin();
    return y < st[k].size() && st[k][y] == j ? (int)sl[panel[k]][y] : -1;
  };
  t.pos.assign(nnz, -1);
  t.diag.assign(n, -1);
  const int *pi = mi.data();
  auto in_panel = [&](int i, int j) {
    const int k = std::min(i, j);
    return top[k] && panel_slot(k, std::max(i, j)) >= 0;
  };
  // Bottom rows' entries by pass: rows of a level by length, so that a pass's rows take about as many
  // rounds; lanes a power of two near the rows' lengths, more where few rows are left.
  auto build_passes = [&](XdPasses &ps, int off, bool upper) {
    ps.gptr.assign(1, 0);
    std::vector<std::vector<int>> ents(t.nbot);
    for (int x = 0; x < t.nbot; ++x) {
      const int i = t.order[x];
      if (upper && last[i]) continue;
      const int b = upper ? mdiag[i] + 1 : mp[i], e = upper ? mp[i + 1] : mdiag[i];
      for (int k = b; k < e; ++k)
        if (upper || !in_panel(i, pi[k])) ents[x].push_back(k);
    }
    for (int g = 0; g < t.ngroups; ++g) {
      for (int s = 0; s < t.glev[g + 1] - t.glev[g]; ++s) {
        const int l = upper ? t.glev[g + 1] - 1 - s : t.glev[g] + s;
        std::vector<int> rows;
        for (int x = t.lrow[l]; x < t.lrow[l + 1]; ++x)
          if (upper ? !last[t.order[x]] : !ents[x].empty()) rows.push_back(x);
        std::stable_sort(rows.begin(), rows.end(), [&](int a, int b) { return ents[a].size() < ents[b].size(); });
        for (size_t r = 0; r < rows.size();) {
          int lg = 0;
          while (lg < 5 && (1u << lg) < ents[rows[r]].size()) ++lg;
          // A long row takes up to the whole block, in passes with its like (a hub's row of 6,000 entries
          // by 32 lanes: 78 us a solve; by 512: 24).
          const bool longer = ents[rows[r]].size() > kLongRow;
          while (longer && (1u << lg) < (unsigned)kPassThreads && ents[rows[r]].size() > (8u << lg)) ++lg;
          size_t count = std::min(rows.size() - r, (size_t)(kPassThreads >> lg));
          while (!longer && ents[rows[r + count - 1]].size() > kLongRow) --count;
          size_t most = ents[rows[r + count - 1]].size();
          while (lg < 5 && most > (1u << lg) && (count << (lg + 1)) <= (size_t)kPassThreads) ++lg;
          const int lanes = 1 << lg, rounds = std::max(1, (int)((most + lanes - 1) / lanes)), width = (int)count * lanes;
          const bool end = r + count == rows.size();
          ps.pass.push_back({(int)ps.rows.size(), (int)count | lg << 16 | (int)end << 24, off + (int)ps.col.size(), rounds});
          const int base = (int)ps.col.size();
          ps.col.resize(ps.col.size() + (size_t)rounds * width, -1);
          for (size_t y = 0; y < count; ++y) {
            const int x = rows[r + y];
            ps.rows.push_back(x);
            for (size_t z = 0; z < ents[x].size(); ++z) {
              const int at = base + (int)(z / lanes) * width + (int)y * lanes + (int)(z % lanes);
              ps.col[at] = place[pi[ents[x][z]]];
              t.pos[ents[x][z]] = off + at;
            }
          }
          r += count;
        }
      }
      ps.gptr.push_back((int)ps.pass.size());
    }
    return off + (int)ps.col.size();
  };
  t.l0 = build_passes(t.fwd, 0, false);
  t.lptr.assign(1, 0);
  for (int x = t.nbot; x < n; ++x) {
    const int i = t.order[x];
    for (int e = mp[i]; e < mdiag[i]; ++e)
      if (!in_panel(i, pi[e])) {
        t.pos[e] = t.l0 + (int)t.lcol.size();
        t.lcol.push_back(place[pi[e]]);
      }
    t.lptr.push_back((int)t.lcol.size());
  }
  t.u0 = t.l0 + (int)t.lcol.size();
  t.t0 = build_passes(t.bwd, t.u0, true);
  t.tptr.assign(1, 0);
  for (int x = 0; x < n; ++x) {
    const int i = t.order[x];
    if (!last[i]) continue;
    t.tail.push_back(x);
    for (int e = mdiag[i] + 1; e < mp[i + 1]; ++e)
      if (!in_panel(i, pi[e])) {
        t.pos[e] = t.t0 + (int)t.tcol.size();
        t.tcol.push_back(place[pi[e]]);
      }
    t.tptr.push_back((int)t.tcol.size());
  }
  t.d0 = t.t0 + (int)t.tcol.size();
  t.p0 = (t.d0 + t.nbot + 15) / 16 * 16;  // panels start on 128 bytes
  t.nv = (long long)t.p0 + xd_panel_size(t.F) * t.bptr[t.nchains];
  if (t.nv > INT_MAX) return false;
  for (int i = 0; i < n; ++i) {
    for (int e = mp[i]; e < mp[i + 1]; ++e) {
      if (t.pos[e] >= 0) continue;
      const int j = pi[e];
      if (i == j && !top[i]) {
        t.pos[e] = t.d0 + place[i];
      } else {
        const int k = std::min(i, j), s = panel_slot(k, std::max(i, j));
        if (!top[k] || s < 0) return false;
        const int p = panel[k], row = (p - t.cptr[chain_of[k]]) % kBlockPivots + (j >= i ? 0 : kBlockPivots);
        t.pos[e] = t.p0 + (int)xd_panel_size(t.F) * block_of(p) + row * t.F + s;
      }
    }
    t.diag[i] = t.pos[mdiag[i]];
  }

  // Bottom divisions and updates, level by level; updates of top entries aside.
  t.ldiv.assign(1, 0);
  t.ldst.assign(1, 0);
  std::vector<int> slot_of(nnz, -1), touched, upd, su;
  std::vector<XdPos4> lv;
  std::vector<int> cnt, start;
  std::vector<XdPos2> sv;
  for (size_t l = 0; l + 1 < t.lrow.size(); ++l) {
    touched.clear();
    upd.clear();
    lv.clear();
    for (int x = t.lrow[l]; x < t.lrow[l + 1]; ++x) {
      const int k = t.order[x];
      for (int e = lcp[k]; e < lcp[k + 1]; ++e) {
        const int i = lci[e], lp = t.pos[lcpos[e]];
        t.div.push_back({lp, t.diag[k]});
        const int *rb = pi + mp[i], *re = pi + mp[i + 1];
        for (int u = mdiag[k] + 1; u < mp[k + 1]; ++u) {
          const int j = pi[u];
          rb = std::lower_bound(rb, re, j);
          if (rb == re || *rb != j) return false;
          const int d = (int)(rb - pi);
          if (top[std::min(i, j)]) {
            su.push_back(d);
            sv.push_back({lp, t.pos[u]});
            continue;
          }
          if (slot_of[d] < 0) {
            slot_of[d] = (int)touched.size();
            touched.push_back(d);
          }
          upd.push_back(slot_of[d]);
          lv.push_back({lp, t.pos[u], t.diag[k], 0});
        }
      }
    }
    cnt.assign(touched.size() + 1, 0);
    for (int s : upd) ++cnt[s + 1];
    start = cnt;
    for (size_t d = 0; d < touched.size(); ++d) start[d + 1] += start[d];
    std::vector<XdPos4> sorted(lv.size());
    {
      std::vector<int> f(start.begin(), start.end());
      for (size_t x = 0; x < lv.size(); ++x) sorted[f[upd[x]]++] = lv[x];
    }
    std::vector<XdPos4> longer;
    for (size_t d = 0; d < touched.size(); ++d) {
      const int b = start[d], c = cnt[d + 1], dp = t.pos[touched[d]];
      slot_of[touched[d]] = -1;
      if (c > kLongPairs) {
        longer.push_back({dp, (int)t.pairs.size(), c, -1});
        t.pairs.insert(t.pairs.end(), sorted.begin() + b, sorted.begin() + b + c);
      } else if (c == 1) {
        t.dst.push_back({dp, sorted[b].x, sorted[b].y, sorted[b].z});
      } else {
        t.dst.push_back({dp, (int)t.pairs.size(), c, -1});
        t.pairs.insert(t.pairs.end(), sorted.begin() + b, sorted.begin() + b + c);
      }
    }
    t.llong.push_back((int)t.dst.size());
    t.any_long = t.any_long || !longer.empty();
    t.dst.insert(t.dst.end(), longer.begin(), longer.end());
    t.ldiv.push_back((int)t.div.size());
    t.ldst.push_back((int)t.dst.size());
    if (t.pairs.size() > (size_t)INT_MAX || sv.size() > (size_t)INT_MAX) return false;
  }
  // Top destinations (in the order of their positions), each with its pairs in the order of the levels.
  {
    std::vector<int> count(nnz, 0);
    for (int d : su) ++count[d];
    std::vector<XdPos2> by;  // (position in V, M entry)
    for (int d = 0; d < nnz; ++d)
      if (count[d] > 0) by.push_back({t.pos[d], d});
    std::sort(by.begin(), by.end(), [](const XdPos2 &a, const XdPos2 &b) { return a.x < b.x; });
    std::vector<int> fill(nnz, 0);
    t.sptr.assign(1, 0);
    for (const XdPos2 &d : by) {
      t.sdst.push_back(d.x);
      fill[d.y] = t.sptr.back();
      t.sptr.push_back(t.sptr.back() + count[d.y]);
    }
    t.spairs.resize(sv.size());
    for (size_t x = 0; x < su.size(); ++x) t.spairs[fill[su[x]]++] = sv[x];
  }
  for (int p = 0; p < t.ntop; ++p) {
    const int k = nodes[p];
    for (int e = lcp[k]; e < lcp[k + 1]; ++e)
      if (panel_slot(k, lci[e]) < 0) t.tdiv.push_back({t.pos[lcpos[e]], t.diag[k]});
  }
  return true;
}
