// Host part of the nested subspace products: the tree of subspaces, the program of the mult, and the
// chunks of the multTranspose (nest_plan.h), with a host evaluation of both programs for the tests.
#include "nest_plan.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>

#include "../../include/sgmev_tools.h"

namespace sgmev {
namespace {
int64_t round_up32(int64_t x) { return (x + 31) / 32 * 32; }
}  // namespace

bool nest_plan(NestTables* p, int dim, int64_t n, const double* level_pow2, const double* index,
               std::string* err) {
  *p = NestTables{};
  if (dim < 1 || dim > 32 || n < 1 || n > (int64_t(1) << 27)) {
    *err = "nested kernels need 1 <= dim <= 32 and a non-empty grid";
    return false;
  }
  // ---- group the grid points by level vector (open-addressed hash of the level rows) ----
  std::vector<uint8_t> lev;       // [nodes][dim]
  std::vector<int> node_of(static_cast<size_t>(n));
  std::vector<int> slots(1024, -1);
  std::vector<uint64_t> node_hash;
  int n_nodes = 0;
  auto hash_row = [&](const uint8_t* r) {
    uint64_t h = 1469598103934665603ull;  // FNV-1a
    for (int t = 0; t < dim; ++t) h = (h ^ r[t]) * 1099511628211ull;
    return h ^ (h >> 29);
  };
  auto find = [&](const uint8_t* r, bool insert) -> int {
    const uint64_t h = hash_row(r);
    for (size_t s = h & (slots.size() - 1);; s = (s + 1) & (slots.size() - 1)) {
      const int id = slots[s];
      if (id < 0) {
        if (!insert) return -1;
        slots[s] = n_nodes;
        lev.insert(lev.end(), r, r + dim);
        node_hash.push_back(h);
        ++n_nodes;
        if (static_cast<size_t>(n_nodes) * 2 > slots.size()) {
          slots.assign(slots.size() * 4, -1);
          for (int k = 0; k < n_nodes; ++k) {
            size_t q = node_hash[k] & (slots.size() - 1);
            while (slots[q] >= 0) q = (q + 1) & (slots.size() - 1);
            slots[q] = k;
          }
        }
        return n_nodes - 1;
      }
      if (node_hash[id] == h && std::memcmp(&lev[static_cast<size_t>(id) * dim], r, dim) == 0) return id;
    }
  };
  std::vector<uint8_t> row(dim, 1);
  const int root = find(row.data(), true);
  p->lmax.assign(dim, 1);
  for (int64_t g = 0; g < n; ++g) {
    for (int t = 0; t < dim; ++t) {
      uint64_t b;
      std::memcpy(&b, &level_pow2[g * dim + t], 8);
      const int l = static_cast<int>((b >> 52) & 0x7FF) - 1023;
      if (l < 1 || l > 20) {
        *err = "nested kernels need levels in [1, 20]";
        return false;
      }
      row[t] = static_cast<uint8_t>(l);
      p->lmax[t] = std::max(p->lmax[t], l);
    }
    node_of[g] = find(row.data(), true);
  }
  std::vector<char> real(n_nodes, 0);
  for (int64_t g = 0; g < n; ++g) real[node_of[g]] = 1;
  p->n_sub = static_cast<int>(std::count(real.begin(), real.end(), 1));
  // ---- the tree: parents (without the last active dimension), missing ones added ----
  std::vector<int> parent, fac, last, excess, ent(dim + 1, 1);
  for (int t = 0; t < dim; ++t) ent[t + 1] = ent[t] + p->lmax[t] - 1;
  p->n_ent = ent[dim];
  if (p->n_ent > 1000 || 64 * (8 * p->n_ent + 4 * dim) > 128 * 1024) {
    *err = "nested kernels: the table of a data point is too long";
    return false;
  }
  for (int id = 0; id < n_nodes; ++id) {  // grows while it runs
    std::copy(&lev[static_cast<size_t>(id) * dim], &lev[static_cast<size_t>(id) * dim] + dim, row.begin());
    int t = dim - 1, ex = 0;
    for (int u = 0; u < dim; ++u) ex += row[u] - 1;
    while (t >= 0 && row[t] == 1) --t;
    excess.push_back(ex);
    last.push_back(t);
    if (t < 0) {
      parent.push_back(-1);
      fac.push_back(kFacH1);
      continue;
    }
    if (ex > 9) {  // 2^9 = kNestMaxCells
      *err = "nested kernels need subspaces of at most 512 cells";
      return false;
    }
    const int l = row[t];
    fac.push_back(make_fac(ent[t] + l - 2, t, l - 1, p->lmax[t] - l));
    row[t] = 1;
    const int par = find(row.data(), true);
    if (static_cast<size_t>(n_nodes) > real.size()) real.resize(n_nodes, 0);
    parent.push_back(par);
  }
  std::vector<std::vector<int>> kids(n_nodes);
  for (int id = 0; id < n_nodes; ++id)
    if (parent[id] >= 0) kids[parent[id]].push_back(id);
  for (auto& k : kids)
    std::sort(k.begin(), k.end(), [&](int a, int b) { return fac_e(fac[a]) < fac_e(fac[b]); });
  auto inner = [&](int id) { return id == root || !kids[id].empty(); };
  // ---- mult program ----
  std::vector<int> dfs{root}, order;
  while (!dfs.empty()) {
    const int id = dfs.back();
    dfs.pop_back();
    order.push_back(id);
    for (size_t k = kids[id].size(); k-- > 0;) dfs.push_back(kids[id][k]);
  }
  // a node of budget b has in every later dimension, and no others, children of levels 2 .. b + 1, that
  // of level l of budget b + 1 - l (in the last dimension: a leaf). The kernels evaluate budgets 1
  // (run), 2 (tree) and 3 (forest) whole (nest_plan.h).
  std::vector<int> budget(n_nodes, 0);
  auto block_of = [&](int id, int b) -> int64_t {
    const int k = dim - 1 - last[id];
    const int64_t c = int64_t(1) << excess[id];
    return b == 1 ? c * nest_run_row(k) : b == 2 ? c * nest_tree_row(k) : (c + 3) / 4 * 4 + c * nest_forest_at(k);
  };
  if (dim <= kNestMacroDim) {
    for (size_t at = order.size(); at-- > 0;) {  // children before parents
      const int id = order[at], k = dim - 1 - last[id], nk = static_cast<int>(kids[id].size());
      if (k == 0 || nk % k != 0 || nk / k < 1 || nk / k > 3) continue;
      const int b = nk / k;
      bool all = block_of(id, b) <= kNestBlockCells;
      for (int i = 0; i < nk; ++i) {  // ordered by (dimension, level)
        const int c = kids[id][i], t = last[id] + 1 + i / b, l = 2 + i % b;
        all = all && last[c] == t && fac_k(fac[c]) == l - 1 &&
              (l == b + 1 || t == dim - 1 ? kids[c].empty() : budget[c] == b + 1 - l);
      }
      if (all) budget[id] = b;
    }
  }
  // where the coefficient of cell c of a node lies: base + (c >> hs) hi + ((c >> ms) & mm) mid + (c & lm)
  struct Place { int64_t base = -1, hi = 0; int hs = 31, ms = 31, mm = 0, mid = 0, lm = 0; };
  std::vector<Place> place(n_nodes);
  std::vector<NestOp4> qops;
  std::vector<NestOp2> lops;
  std::vector<int> facs, q_work, q_group;
  std::vector<int64_t> q_coef;  // first position of an inner node's coefficients
  std::vector<NestOp2> groups;  // first and end factor
  int64_t total = 0;
  auto plain = [&](int id) {  // cells in order
    place[id].base = total;
    place[id].lm = (1 << excess[id]) - 1;
    total += int64_t(1) << excess[id];
  };
  auto add_q = [&](int id) {
    q_coef.push_back(total);
    q_group.push_back(static_cast<int>(groups.size()) - 1);
    const int k = dim - 1 - last[id], t0 = last[id] + 1;
    if (budget[id] > 0) {
      const int64_t b = total;
      auto put = [&](int c, int64_t base, int64_t hi, int hs, int ms, int mm, int mid, int lm) {
        place[c].base = base;
        place[c].hi = hi;
        place[c].hs = hs;
        place[c].ms = ms;
        place[c].mm = mm;
        place[c].mid = mid;
        place[c].lm = lm;
      };
      auto run = [&](int n, int64_t at) {  // the node's rows from `at` on
        const int row = nest_run_row(dim - 1 - last[n]);
        put(n, at, row, 0, 31, 0, 0, 0);
        for (int c : kids[n]) put(c, at + 1 + 2 * (dim - 1 - last[c]), row, 1, 31, 0, 0, 1);
      };
      auto tree = [&](int n, int64_t at) {
        const int row = nest_tree_row(dim - 1 - last[n]);
        put(n, at, row, 0, 31, 0, 0, 0);
        for (int c : kids[n]) {
          const int kt = dim - 1 - last[c], rr = nest_run_row(kt);
          const int64_t sec = at + nest_tree_at(kt);
          if (fac_k(fac[c]) == 2) {  // the level-3 leaf
            put(c, sec + 2 * rr, row, 2, 31, 0, 0, 3);
          } else {
            put(c, sec, row, 1, 0, 1, rr, 0);
            for (int g : kids[c]) put(g, sec + 1 + 2 * (dim - 1 - last[g]), row, 2, 1, 1, rr, 1);
          }
        }
      };
      int param = budget[id] == 1 ? nest_run_row(k) : nest_tree_row(k);
      if (budget[id] == 1) {
        run(id, b);
      } else if (budget[id] == 2) {
        tree(id, b);
      } else {
        const int64_t c0 = int64_t(1) << excess[id], b0 = b + (c0 + 3) / 4 * 4;
        param = excess[id];
        put(id, b, 0, 31, 31, 0, 0, (1 << excess[id]) - 1);
        for (int c : kids[id]) {
          const int kt = dim - 1 - last[c], l = fac_k(fac[c]) + 1;
          const int64_t at = b0 + c0 * nest_forest_at(kt);
          if (l == 2) tree(c, at);
          else if (l == 3) run(c, at + 2 * c0 * nest_tree_row(kt));
          else put(c, at + 2 * c0 * nest_tree_row(kt) + 4 * c0 * nest_run_row(kt), 0, 31, 31, 0, 0, (1 << excess[c]) - 1);
        }
      }
      qops.push_back(NestOp4{static_cast<int>(b), -(1 + 4 * t0 + (budget[id] - 1)), param, fac[id]});
      int units = 6 + 2 * k;
      if (budget[id] == 2) units = 8 + k * (k + 5);
      if (budget[id] == 3)
        for (int i = 0; i < k; ++i) units += 14 + i * (i + 5);
      q_work.push_back(units);
      total += (block_of(id, budget[id]) + 3) / 4 * 4;
      return;
    }
    int b = -1, l0 = static_cast<int>(lops.size());
    if (real[id]) {
      b = static_cast<int>(total);
      plain(id);
    }
    auto flush = [&] {
      const int l1 = static_cast<int>(lops.size());
      qops.push_back(NestOp4{b, l0, l1, fac[id]});
      q_work.push_back(6 + 3 * (l1 - l0));
      l0 = l1;
      b = -1;
    };
    for (int c : kids[id]) {
      if (inner(c)) continue;
      if (total - q_coef.back() + (int64_t(1) << excess[c]) > kNestBlockCells ||
          static_cast<int>(lops.size()) - l0 == kNestLeaves) {
        flush();  // the rest of the leaves under the same node, in a window of their own if need be
        q_coef.push_back(total);
        q_group.push_back(q_group.back());
      }
      lops.push_back(NestOp2{static_cast<int>(total), fac[c]});
      plain(c);
    }
    flush();
  };
  p->whole = budget[root] > 0;
  groups.push_back(NestOp2{0, 0});
  add_q(root);  // the root by itself: its factor is H_1
  for (int id : order) {
    if (budget[id] > 0) continue;
    const int f0 = static_cast<int>(facs.size());
    bool any = false;
    for (int c : kids[id]) any = any || inner(c);
    if (!any) continue;
    facs.push_back(kFacH1);
    for (int a = id; a != root; a = parent[a]) facs.push_back(fac[a]);
    std::reverse(facs.begin() + f0 + 1, facs.end());  // cells are built from the first dimension on
    groups.push_back(NestOp2{f0, static_cast<int>(facs.size())});
    for (int c : kids[id])
      if (inner(c)) add_q(c);
  }
  q_coef.push_back(total);
  if (total > kNestMaxPositions) {
    *err = "nested kernels: too many coefficient positions";
    return false;
  }
  // windows: runs of inner nodes whose coefficients and program fit shared memory together; a list
  // for S CTAs per tile of points asks for a multiple of S of them, with about the same work each
  const int n_q = static_cast<int>(qops.size());
  const int64_t all_work = std::accumulate(q_work.begin(), q_work.end(), int64_t(0));
  auto opens = [&](int q, int q0) { return q == q0 || q_group[q - 1] != q_group[q]; };
  std::vector<int> q_head(static_cast<size_t>(n_q)), q_words(static_cast<size_t>(n_q));
  int64_t least_words = 0;  // of all windows
  for (int q = 0; q < n_q; ++q) {
    const NestOp2& g = groups[q_group[q]];
    q_head[q] = 1 + (g.y - g.x + 3) / 4;
    q_words[q] = 2 + (qops[q].y >= 0 ? qops[q].z - qops[q].y : 0);
    least_words += q_words[q] + (opens(q, 0) ? q_head[q] : 0);
  }
  if (least_words > kNestMaxWords) {
    *err = "nested kernels: too many subspaces";
    return false;
  }
  // the end of window number `made` that begins with node q0, with `want` of them asked for
  auto window_end = [&](int q0, int64_t cap, int64_t want, int64_t made, int64_t* done) {
    int64_t words = 0;
    int q = q0;
    for (; q < n_q; ++q) {
      const int64_t more = q_words[q] + (opens(q, q0) ? q_head[q] : 0);
      // (a window ends where the work so far, with half of the next node's, passes its share)
      if (q > q0 && (q_coef[q + 1] - q_coef[q0] > cap || words + more > kNestProgram ||
                     (2 * *done + q_work[q]) * want >= 2 * all_work * (made + 1)))
        break;
      words += more;
      *done += q_work[q];
    }
    return q;
  };
  for (int list = 0; list < kNestLists; ++list) {
    const int64_t cap = nest_list_cap(list), ctas = nest_list_ctas(list);
    // The fewest windows that the nodes divide into: asked for fewer, they fill up and make more. No
    // fewer than the coefficients or the words need, and in larger steps while far off (one count after
    // the other from S on took 6 s for 230,230 subspaces, this 0.3 s); the kernels take any number.
    int64_t want = std::max((total + cap - 1) / cap, (least_words + kNestProgram - 1) / kNestProgram);
    want = std::max<int64_t>(1, (want + ctas - 1) / ctas) * ctas;
    const size_t prog0 = p->prog.size(), win0 = p->windows.size();
    int64_t widest = 0, longest = 0, made = 0, done = 0;
    auto build = [&] {
      p->prog.resize(prog0);
      p->windows.resize(win0);
      widest = longest = made = done = 0;
      for (int q = 0; q < n_q; ++made) {
        const int p0 = static_cast<int>(p->prog.size()), q0 = q, c0 = static_cast<int>(q_coef[q0]);
        const int q1 = window_end(q0, cap, want, made, &done);
        size_t header = 0;
        for (; q < q1; ++q) {
          const NestOp4& o = qops[q];
          const NestOp2& g = groups[q_group[q]];
          const int nl = o.y >= 0 ? o.z - o.y : 0;
          if (opens(q, q0)) {
            header = p->prog.size();
            p->prog.push_back(NestOp4{0, g.y - g.x, 0, 0});
            for (int i = g.x; i < g.y; i += 4) {
              auto f = [&](int k) { return k < g.y ? facs[k] : 0; };
              p->prog.push_back(NestOp4{f(i), f(i + 1), f(i + 2), f(i + 3)});
            }
          }
          ++p->prog[header].x;
          p->prog.push_back(NestOp4{o.x >= 0 ? o.x - c0 : -1, o.y >= 0 ? nl : o.y, o.z, 0});
          p->prog.push_back(NestOp4{fac_e(o.w), fac_t(o.w), fac_k(o.w), fac_shift(o.w)});
          for (int i = 0; i < nl; ++i) {
            const NestOp2& u = lops[o.y + i];
            p->prog.push_back(NestOp4{u.x - c0, fac_e(u.y) | (fac_t(u.y) << 16), fac_k(u.y), fac_shift(u.y)});
          }
        }
        const int p1 = static_cast<int>(p->prog.size());
        widest = std::max(widest, q_coef[q] - q_coef[q0]);
        longest = std::max<int64_t>(longest, p1 - p0);
        p->windows.push_back(NestOp4{p0, p1, c0, static_cast<int>(q_coef[q])});
      }
    };
    build();
    if (made > want && want < 2 * n_q) {  // (count before the next one is built)
      for (int tries = 0; tries < 32 && made > want && want < 2 * n_q; ++tries) {
        want += std::max<int64_t>(1, (made - want) / (4 * ctas)) * ctas;
        made = done = 0;
        for (int q = 0; q < n_q; ++made) q = window_end(q, cap, want, made, &done);
      }
      build();
    }
    p->list_begin.push_back(static_cast<int>(win0));
    p->list_cells.push_back(static_cast<int>(widest));
    p->list_words.push_back(static_cast<int>(longest));
  }
  p->list_begin.push_back(static_cast<int>(p->windows.size()));
  std::vector<int> inv(static_cast<size_t>(total), -1);
  std::vector<int> cell_of(static_cast<size_t>(n));
  for (int64_t g = 0; g < n; ++g) {
    const uint8_t* l = &lev[static_cast<size_t>(node_of[g]) * dim];
    int c = 0;
    for (int t = 0; t < dim; ++t)
      if (l[t] > 1) c = (c << (l[t] - 1)) | ((static_cast<int>(index[g * dim + t]) - 1) / 2);
    cell_of[g] = c;
    const Place& pl = place[node_of[g]];
    int& at = inv[pl.base + (c >> pl.hs) * pl.hi + ((c >> pl.ms) & pl.mm) * pl.mid + (c & pl.lm)];
    if (at >= 0) {  // a position holds one grid point; the dense kernels add both
      *err = "nested kernels: a grid point occurs twice";
      return false;
    }
    at = static_cast<int>(g);
  }
  // ---- multTranspose program: subspaces by cell count, then tree order, in chunks ----
  std::vector<int> subs;
  for (int id : order)
    if (real[id]) subs.push_back(id);
  std::stable_sort(subs.begin(), subs.end(), [&](int a, int b) { return excess[a] > excess[b]; });
  for (int id : subs) {
    p->cells += int64_t(1) << excess[id];
    p->cmax = std::max(p->cmax, 1 << excess[id]);
  }
  std::vector<NestOp4> chunks;
  std::vector<NestOp2> cq, cs, cwarp;
  std::vector<int> clev, ccell, local(n_nodes, -1), depth(n_nodes, 0);
  for (int id : order) depth[id] = parent[id] < 0 ? 0 : depth[parent[id]] + 1;
  for (int id : subs) p->n_act += depth[id];
  std::vector<int64_t> tpos(n_nodes, -1);
  int64_t row_total = 0;
  for (size_t at = 0; at < subs.size();) {
    const int cells = 1 << excess[subs[at]];
    int threads = static_cast<int>(std::min<size_t>(256, kNestAccBudget / sizeof(double) / cells / 32 * 32));
    threads = std::max(32, threads);
    threads = std::min<int>(threads, static_cast<int>(round_up32(static_cast<int64_t>(subs.size() - at))));
    // the class takes the following subspaces too, until they have so few cells that a class of
    // their own would run blocks of four times the threads
    NestClass c;
    c.threads = threads;
    c.chunk_begin = static_cast<int>(chunks.size());
    c.row_begin = row_total;
    while (at < subs.size()) {
      const int cc = 1 << excess[subs[at]];
      if (threads < 128 && cc * 4 <= cells && subs.size() - at > 64) break;
      const int cnt = static_cast<int>(std::min<size_t>(threads, subs.size() - at));
      // inner nodes of the chunk: the parents of its subspaces and their ancestors, by depth
      std::vector<int> need;
      for (int k = 0; k < cnt; ++k)
        for (int a = parent[subs[at + k]]; a >= 0 && local[a] < 0; a = parent[a]) {
          local[a] = 0;
          need.push_back(a);
        }
      if (local[root] < 0) need.push_back(root);
      std::sort(need.begin(), need.end(), [&](int a, int b) {
        return depth[a] != depth[b] ? depth[a] < depth[b] : a < b;
      });
      for (size_t k = 0; k < need.size(); ++k) local[need[k]] = static_cast<int>(k);
      const int lev0 = static_cast<int>(clev.size()), q0 = static_cast<int>(cq.size());
      int nlev = 0;
      for (size_t k = 0; k < need.size(); ++k) {
        const int a = need[k];
        if (k > 0 && depth[a] != depth[need[k - 1]]) {
          clev.push_back(static_cast<int>(k));
          ++nlev;
        }
        cq.push_back(NestOp2{parent[a] >= 0 ? local[parent[a]] : 0, fac[a]});
      }
      clev.push_back(static_cast<int>(need.size()));
      chunks.push_back(NestOp4{q0, static_cast<int>(need.size()), lev0, nlev});
      for (int k = 0; k < threads; ++k) {
        if (k >= cnt) {
          cs.push_back(NestOp2{0, kFacH1});
          ccell.push_back(0);
          continue;
        }
        const int id = subs[at + k];
        // the root itself: v_j H_1 times the 1 behind the table row
        cs.push_back(id == root ? NestOp2{0, make_fac(p->n_ent, 0, 0, 31)}
                                : NestOp2{local[parent[id]], fac[id]});
        ccell.push_back(1 << excess[id]);
      }
      // a warp's sums: [most cells of its subspaces][32], in the chunk's shared memory and in the rows
      int sums = 0;
      for (int w = 0; w < threads / 32; ++w) {
        int most = 0;
        for (int k = 32 * w; k < std::min(cnt, 32 * w + 32); ++k) {
          most = std::max(most, 1 << excess[subs[at + k]]);
          tpos[subs[at + k]] = row_total + c.row_len + sums + (k - 32 * w);
        }
        cwarp.push_back(NestOp2{sums, static_cast<int>(c.row_len) + sums});
        sums += 32 * most;
      }
      c.sums = std::max(c.sums, sums);
      c.row_len += sums;
      if (row_total + c.row_len > kNestMaxPositions) {
        *err = "nested kernels: too many cell sums";
        return false;
      }
      c.nq = std::max(c.nq, static_cast<int>(need.size()));
      for (int a : need) local[a] = -1;
      at += cnt;
    }
    c.chunks = static_cast<int>(chunks.size()) - c.chunk_begin;
    if (c.smem(sizeof(double), p->n_ent, dim) > kNestSmem) {
      *err = "nested kernels: a chunk of subspaces does not fit shared memory";
      return false;
    }
    row_total += c.row_len;
    p->classes.push_back(c);
  }
  std::vector<int> tinv(static_cast<size_t>(row_total), -1);
  for (int64_t g = 0; g < n; ++g)
    tinv[tpos[node_of[g]] + static_cast<int64_t>(cell_of[g]) * 32] = static_cast<int>(g);
  p->dim = dim;
  p->n = n;
  p->inv = std::move(inv);
  p->chunks = std::move(chunks);
  p->cq = std::move(cq);
  p->cs = std::move(cs);
  p->cwarp = std::move(cwarp);
  p->clev = std::move(clev);
  p->ccell = std::move(ccell);
  p->tinv = std::move(tinv);
  return true;
}

}  // namespace sgmev

// ---- host evaluation --------------------------------------------------------------------------------
extern "C" SGMEV_API int sgmev_nest_host(int dim, int64_t n_grid, const double* level_pow2,
                                         const double* index, int modlinear, int64_t n_data,
                                         const double* data, const double* alpha,
                                         const double* source, double* mult_out,
                                         double* multt_out) {
  using namespace sgmev;
  NestTables p;
  std::string err;
  if (!nest_plan(&p, dim, n_grid, level_pow2, index, &err)) return 1;
  // every access goes through at(): an index outside its array ends the evaluation with status 2
  bool bad = false;
  auto at = [&](const auto& v, int64_t i) {
    using V = typename std::decay<decltype(v[0])>::type;
    if (i < 0 || i >= static_cast<int64_t>(v.size())) {
      bad = true;
      return V{};
    }
    return v[static_cast<size_t>(i)];
  };
  std::vector<double> coef(p.inv.size(), 0.0);
  for (size_t k = 0; k < p.inv.size(); ++k)
    if (p.inv[k] >= 0) coef[k] = alpha[p.inv[k]];
  std::vector<double> sums(p.tinv.size(), 0.0), tab(static_cast<size_t>(p.n_ent) + 1), prod, inner;
  std::vector<uint32_t> xc(static_cast<size_t>(dim)), cell;
  for (int64_t j = 0; j < n_data && !bad; ++j) {
    const double* x = data + j * dim;
    bool inside = true;
    for (int t = 0; t < dim; ++t)
      inside = inside && (modlinear ? x[t] >= 0.0 && x[t] <= 1.0 : x[t] > 0x1p-1000 && x[t] < 1.0);
    tab[0] = inside ? 1.0 : 0.0;
    tab[p.n_ent] = 1.0;
    int e = 1;
    for (int t = 0; t < dim; ++t) {
      const double xt = inside ? x[t] : 0.5;
      const int bits = p.lmax[t] - 1;
      const uint32_t last = (1u << bits) - 1u;
      xc[t] = std::min(static_cast<uint32_t>(xt * static_cast<double>(1u << bits)), last);
      double h = 2.0 * (xt > 0.5 ? 1.0 - xt : xt);
      const double h1 = h;
      if (!modlinear) tab[0] *= h1;
      for (int l = 2; l <= bits + 1; ++l, ++e) {
        const double y = std::ldexp(xt, l);
        const uint32_t k = xc[t] >> (bits - (l - 1)), top = (1u << (l - 1)) - 1u;
        h = 2.0 * (h > 0.5 ? 1.0 - h : h);
        if (modlinear && k == 0u) tab[e] = 2.0 - y;
        else if (modlinear && k == top) tab[e] = y - (std::ldexp(1.0, l) - 2.0);
        else tab[e] = modlinear ? 1.0 - std::fabs(y - (2.0 * k + 1.0)) : h / h1;
      }
    }
    auto step = [&](uint32_t c, int f) {
      return (c << fac_k(f)) | (at(xc, fac_t(f)) >> fac_shift(f));
    };
    // mult: the windows of a list, another list for another point
    double acc = 0.0;
    const int list = static_cast<int>(j % kNestLists);
    for (int w = at(p.list_begin, list); w < at(p.list_begin, list + 1); ++w) {
      const NestOp4 win = at(p.windows, w);
      if (win.w - win.z > p.list_cells[list] || win.w - win.z > nest_list_cap(list) ||
          win.y - win.x > p.list_words[list] || win.y - win.x > kNestProgram)
        bad = true;
      auto co = [&](int64_t i) {  // a window's coefficients only
        if (i < 0 || i >= win.w - win.z) bad = true;
        return at(coef, win.z + i);
      };
      for (int at_op = win.x; at_op < win.y && !bad;) {
        const NestOp4 head = at(p.prog, at_op++);
        double pr = 1.0, ar = 0.0;
        uint32_t cr = 0;
        for (int i = 0; i < head.y; ++i) {
          const NestOp4 f4 = at(p.prog, at_op + i / 4);
          const int f = i % 4 == 0 ? f4.x : i % 4 == 1 ? f4.y : i % 4 == 2 ? f4.z : f4.w;
          pr *= at(tab, fac_e(f));
          cr = step(cr, f);
        }
        at_op += (head.y + 3) / 4;
        for (int q = 0; q < head.x; ++q) {
          const NestOp4 qo = at(p.prog, at_op++), qf = at(p.prog, at_op++);
          const int qfac = make_fac(qf.x, qf.y, qf.z, qf.w);
          const uint32_t c = step(cr, qfac);
          double sum = 0.0;
          if (qo.y >= 0) {
            sum = qo.x >= 0 ? co(static_cast<int64_t>(qo.x) + c) : 0.0;
            for (int i = 0; i < qo.y; ++i) {
              const NestOp4 l4 = at(p.prog, at_op++);
              const NestOp2 lo{l4.x, make_fac(l4.y & 0xFFFF, l4.y >> 16, l4.z, l4.w)};
              sum += at(tab, fac_e(lo.y)) * co(static_cast<int64_t>(lo.x) + step(c, lo.y));
            }
          } else {
            const int kind = -qo.y - 1, t0 = kind >> 2;
            auto cell_at = [&](int t, int l) { return xc[t] >> (p.lmax[t] - l); };
            auto entry = [&](int t, int l) {
              int e0 = 1;
              for (int u = 0; u < t; ++u) e0 += p.lmax[u] - 1;
              return at(tab, e0 + l - 2);
            };
            auto run = [&](int64_t r0, int t1) {
              double sr = co(r0);
              for (int t = t1; t < dim; ++t)
                sr += entry(t, 2) * co(r0 + 1 + 2 * (dim - 1 - t) + cell_at(t, 2));
              return sr;
            };
            auto tree = [&](int64_t row, int t1) {
              double st = co(row);
              for (int t = t1; t < dim; ++t) {
                const int kt = dim - 1 - t;
                const int64_t sec = row + nest_tree_at(kt);
                st += entry(t, 2) * run(sec + static_cast<int64_t>(cell_at(t, 2)) * nest_run_row(kt), t + 1);
                st += entry(t, 3) * co(sec + 2 * nest_run_row(kt) + cell_at(t, 3));
              }
              return st;
            };
            if ((kind & 3) == 0) {
              sum = run(qo.x + static_cast<int64_t>(c) * qo.z, t0);
            } else if ((kind & 3) == 1) {
              sum = tree(qo.x + static_cast<int64_t>(c) * qo.z, t0);
            } else {
              const int64_t c0 = int64_t(1) << qo.z, b0 = qo.x + (c0 + 3) / 4 * 4;
              sum = co(qo.x + c);
              for (int t = t0; t < dim; ++t) {
                const int kt = dim - 1 - t;
                const int64_t at_t = b0 + c0 * nest_forest_at(kt), at_r = at_t + 2 * c0 * nest_tree_row(kt),
                              at_l = at_r + 4 * c0 * nest_run_row(kt);
                sum += entry(t, 2) * tree(at_t + static_cast<int64_t>((c << 1) | cell_at(t, 2)) * nest_tree_row(kt), t + 1);
                sum += entry(t, 3) * run(at_r + static_cast<int64_t>((c << 2) | cell_at(t, 3)) * nest_run_row(kt), t + 1);
                sum += entry(t, 4) * co(at_l + ((c << 3) | cell_at(t, 4)));
              }
            }
          }
          ar += at(tab, fac_e(qfac)) * sum;
        }
        acc += pr * ar;
      }
    }
    mult_out[j] = acc;
    // multTranspose
    int64_t cs_at = 0;
    for (const NestClass& c : p.classes) {
      if (c.threads < 32 || c.threads > 256 || c.threads % 32 || c.smem(8, p.n_ent, dim) > kNestSmem) bad = true;
      for (int k = 0; k < c.chunks; ++k) {
        const NestOp4 ch = at(p.chunks, c.chunk_begin + k);
        if (ch.y > c.nq || at(p.clev, ch.z + ch.w) != ch.y) bad = true;
        prod.assign(static_cast<size_t>(c.nq), 0.0);
        cell.assign(static_cast<size_t>(c.nq), 0u);
        prod[0] = source[j] * tab[0];
        for (int q = at(p.clev, ch.z); q < ch.y; ++q) {
          const NestOp2 o = at(p.cq, ch.x + q);
          if (o.x >= q) bad = true;  // a parent comes before its children
          prod[q] = at(prod, o.x) * at(tab, fac_e(o.y));
          cell[q] = step(at(cell, o.x), o.y);
          if (cell[q] > 0xFFFFu) bad = true;
        }
        for (int d = 0; d < ch.w; ++d)  // parents lie in earlier depths
          for (int q = at(p.clev, ch.z + d); q < at(p.clev, ch.z + d + 1); ++q)
            if (at(p.cq, ch.x + q).x >= at(p.clev, ch.z + d)) bad = true;
        for (int t = 0; t < c.threads; ++t) {
          const int cells = at(p.ccell, cs_at + static_cast<int64_t>(k) * c.threads + t);
          if (cells == 0) continue;
          const NestOp2 o = at(p.cs, cs_at + static_cast<int64_t>(k) * c.threads + t);
          const uint32_t cl = step(at(cell, o.x), o.y);
          const NestOp2 wp = at(p.cwarp, cs_at / 32 + (k * c.threads + t) / 32);
          const int64_t in_chunk = wp.x + static_cast<int64_t>(cl) * 32 + t % 32;
          if (cl >= static_cast<uint32_t>(cells) || in_chunk >= c.sums) bad = true;
          const int64_t pos = c.row_begin + wp.y + static_cast<int64_t>(cl) * 32 + t % 32;
          if (pos >= c.row_begin + c.row_len || pos >= static_cast<int64_t>(sums.size())) bad = true;
          else sums[pos] += at(prod, o.x) * at(tab, fac_e(o.y));
        }
      }
      cs_at += static_cast<int64_t>(c.chunks) * c.threads;
    }
  }
  std::vector<int> seen(static_cast<size_t>(n_grid), 0), seen_m(seen);
  for (size_t k = 0; k < p.tinv.size(); ++k)
    if (p.tinv[k] >= 0) {
      multt_out[p.tinv[k]] = sums[k];
      ++seen[p.tinv[k]];
    }
  for (size_t k = 0; k < p.inv.size(); ++k)
    if (p.inv[k] >= 0) ++seen_m[p.inv[k]];
  for (int64_t g = 0; g < n_grid; ++g)
    if (seen[g] != 1 || seen_m[g] != 1) bad = true;
  return bad ? 2 : 0;
}
