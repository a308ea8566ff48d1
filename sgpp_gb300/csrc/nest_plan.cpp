// Host part of the nested subspace products: the tree of subspaces, the program of the mult, and the
// chunks of the multTranspose (nest_plan.h), with a host evaluation of both programs for the tests.
#include "nest_plan.h"

#include <algorithm>
#include <cmath>
#include <cstring>

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
  if (p->n_ent > 1000 || sizeof(double) * kNestMultThreads * p->n_ent +
                                 sizeof(uint32_t) * kNestMultThreads * dim > kNestSmem) {
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
  std::vector<NestOp4> rops, qops;
  std::vector<NestOp2> lops;
  std::vector<int> facs, base(n_nodes, -1), work;
  int64_t total = 0;
  auto place = [&](int id) {
    if (real[id]) {
      base[id] = static_cast<int>(total);
      total += int64_t(1) << excess[id];
    }
    return base[id];
  };
  auto add_q = [&](int id, int& units) {
    const int b = place(id), l0 = static_cast<int>(lops.size());
    for (int c : kids[id])
      if (!inner(c)) lops.push_back(NestOp2{place(c), fac[c]});
    qops.push_back(NestOp4{b, l0, static_cast<int>(lops.size()), fac[id]});
    units += 3 + static_cast<int>(lops.size()) - l0;
  };
  {
    int units = 0;
    add_q(root, units);  // the root by itself: its factor is H_1
    rops.push_back(NestOp4{0, 1, 0, 0});
    work.push_back(units);
  }
  std::vector<int> dfs{root}, order;
  while (!dfs.empty()) {
    const int id = dfs.back();
    dfs.pop_back();
    order.push_back(id);
    for (size_t k = kids[id].size(); k-- > 0;) dfs.push_back(kids[id][k]);
  }
  for (int id : order) {
    const int q0 = static_cast<int>(qops.size()), f0 = static_cast<int>(facs.size());
    int units = 2 + excess[id];
    for (int c : kids[id])
      if (inner(c)) add_q(c, units);
    if (static_cast<int>(qops.size()) == q0) continue;
    facs.push_back(kFacH1);
    for (int a = id; a != root; a = parent[a]) facs.push_back(fac[a]);
    std::reverse(facs.begin() + f0 + 1, facs.end());  // cells are built from the first dimension on
    rops.push_back(NestOp4{q0, static_cast<int>(qops.size()), f0, static_cast<int>(facs.size())});
    work.push_back(units);
  }
  if (lops.empty()) lops.push_back(NestOp2{0, kFacH1});
  if (facs.empty()) facs.push_back(kFacH1);
  const int n_r = static_cast<int>(rops.size());
  // group boundaries for 1 .. kNestSplits CTAs per tile, by work
  std::vector<int64_t> cum(n_r + 1, 0);
  for (int r = 0; r < n_r; ++r) cum[r + 1] = cum[r] + work[r];
  p->cuts.assign(kNestSplits * (kNestSplits + 1), n_r);
  for (int s = 1; s <= kNestSplits; ++s)
    for (int k = 0; k < s; ++k)
      p->cuts[(s - 1) * (kNestSplits + 1) + k] = static_cast<int>(
          std::lower_bound(cum.begin(), cum.end(), cum.back() * k / s) - cum.begin());
  std::vector<int> inv(static_cast<size_t>(total), -1);
  std::vector<int> cell_of(static_cast<size_t>(n));
  for (int64_t g = 0; g < n; ++g) {
    const uint8_t* l = &lev[static_cast<size_t>(node_of[g]) * dim];
    int c = 0;
    for (int t = 0; t < dim; ++t)
      if (l[t] > 1) c = (c << (l[t] - 1)) | ((static_cast<int>(index[g * dim + t]) - 1) / 2);
    cell_of[g] = c;
    inv[base[node_of[g]] + c] = static_cast<int>(g);
  }
  // ---- multTranspose program: subspaces by cell count, then tree order, in chunks ----
  std::vector<int> subs;
  for (int id : order)
    if (real[id]) subs.push_back(id);
  std::stable_sort(subs.begin(), subs.end(), [&](int a, int b) { return excess[a] > excess[b]; });
  std::vector<NestOp4> chunks;
  std::vector<NestOp2> cq, cs;
  std::vector<int> clev, ccell, local(n_nodes, -1), depth(n_nodes, 0);
  for (int id : order) depth[id] = parent[id] < 0 ? 0 : depth[parent[id]] + 1;
  std::vector<int64_t> tpos(n_nodes, -1);
  std::vector<int> tstep(n_nodes, 0);
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
    c.cells = cells;
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
        tpos[id] = row_total + static_cast<int64_t>(chunks.size() - 1 - c.chunk_begin) * cells * threads + k;
        tstep[id] = threads;
      }
      c.nq = std::max(c.nq, static_cast<int>(need.size()));
      for (int a : need) local[a] = -1;
      at += cnt;
    }
    c.chunks = static_cast<int>(chunks.size()) - c.chunk_begin;
    c.row_len = static_cast<int64_t>(c.chunks) * cells * threads;
    c.smem = sizeof(double) * static_cast<size_t>(cells) * threads +
             NestTileLayout(c.nq, p->n_ent, dim).bytes();
    if (c.smem > kNestSmem) {
      *err = "nested kernels: a chunk of subspaces does not fit shared memory";
      return false;
    }
    row_total += c.row_len;
    p->classes.push_back(c);
  }
  std::vector<int> tinv(static_cast<size_t>(row_total), -1);
  for (int64_t g = 0; g < n; ++g)
    tinv[tpos[node_of[g]] + static_cast<int64_t>(cell_of[g]) * tstep[node_of[g]]] = static_cast<int>(g);
  p->dim = dim;
  p->n = n;
  p->rops = std::move(rops);
  p->qops = std::move(qops);
  p->lops = std::move(lops);
  p->facs = std::move(facs);
  p->inv = std::move(inv);
  p->chunks = std::move(chunks);
  p->cq = std::move(cq);
  p->cs = std::move(cs);
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
  const int n_r = static_cast<int>(p.rops.size());
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
    // mult: the groups of every split, and the whole program the same whatever the split
    double acc = 0.0;
    const int splits = 1 + static_cast<int>(j % kNestSplits);
    for (int y = 0; y < splits; ++y) {
      const int r_end = at(p.cuts, (splits - 1) * (kNestSplits + 1) + y + 1);
      for (int r = at(p.cuts, (splits - 1) * (kNestSplits + 1) + y); r < r_end; ++r) {
        const NestOp4 ro = at(p.rops, r);
        double pr = 1.0, ar = 0.0;
        uint32_t cr = 0;
        for (int i = ro.z; i < ro.w; ++i) {
          pr *= at(tab, fac_e(at(p.facs, i)));
          cr = step(cr, at(p.facs, i));
        }
        for (int q = ro.x; q < ro.y; ++q) {
          const NestOp4 qo = at(p.qops, q);
          const uint32_t c = step(cr, qo.w);
          double sum = qo.x >= 0 ? at(coef, static_cast<int64_t>(qo.x) + c) : 0.0;
          for (int i = qo.y; i < qo.z; ++i) {
            const NestOp2 lo = at(p.lops, i);
            sum += at(tab, fac_e(lo.y)) * at(coef, static_cast<int64_t>(lo.x) + step(c, lo.y));
          }
          ar += at(tab, fac_e(qo.w)) * sum;
        }
        acc += pr * ar;
      }
    }
    if (at(p.cuts, (splits - 1) * (kNestSplits + 1)) != 0 ||
        at(p.cuts, (splits - 1) * (kNestSplits + 1) + splits) != n_r)
      bad = true;
    mult_out[j] = acc;
    // multTranspose
    int64_t cs_at = 0;
    for (const NestClass& c : p.classes) {
      if (c.threads < 32 || c.threads > 256 || c.threads % 32 || c.smem > kNestSmem) bad = true;
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
          if (cl >= static_cast<uint32_t>(cells) || cells > c.cells) bad = true;
          const int64_t pos = c.row_begin + (static_cast<int64_t>(k) * c.cells + cl) * c.threads + t;
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
