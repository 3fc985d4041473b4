// block_plan.cpp — see block_plan.h.
#include "block_plan.h"

#include <algorithm>
#include <cmath>
#include <numeric>

namespace dfem {
namespace {

// Cost model (microseconds), from measurements on the B200: a dependent phase
// of the solve is a grid-wide barrier and the latency of its loads; products
// stream from L2; a pivot of a rebuild is one pivot inverse, two tile
// products and a barrier; a rebuild is shared by kSolvesPerBuild solves.
constexpr double kPhaseUs = 2.4, kBytesPerUs = 6.0e6, kPivotUs = 6.5, kFlopsPerUs = 20.0e6, kSolvesPerBuild = 100.0;

struct Tree {
  std::vector<int> size;  // columns of every supernode's subtree
};

Tree subtree(const SupernodalFactor& F) {
  Tree t;
  t.size.assign(F.nsuper, 0);
  for (int q = 0; q < F.nsuper; ++q) {  // children precede parents
    t.size[q] += F.sn_w[q];
    if (F.sn_parent[q] >= 0) t.size[F.sn_parent[q]] += t.size[q];
  }
  return t;
}

// tier and block root (topmost supernode of the same tier) of every supernode
void tiers_of(const SupernodalFactor& F, const Tree& t, const std::vector<int>& taus, std::vector<int>& tier,
              std::vector<int>& root) {
  const int ns = F.nsuper;
  tier.assign(ns, 0);
  root.assign(ns, 0);
  for (int q = 0; q < ns; ++q) {
    int k = 0;
    while (k < (int)taus.size() && t.size[q] > taus[k]) ++k;
    tier[q] = k;
  }
  for (int q = ns - 1; q >= 0; --q) {
    const int p = F.sn_parent[q];
    root[q] = (p >= 0 && tier[p] == tier[q]) ? root[p] : q;
  }
}

// model cost; the tiers that hold blocks are counted (a limit may leave one empty)
struct CostModel {
  const SupernodalFactor& F;
  const Tree& t;
  std::vector<int> tier, root, n;  // scratch: the search asks a few hundred times
  double operator()(const std::vector<int>& taus) {
    tiers_of(F, t, taus, tier, root);
    const int ns = F.nsuper;
    n.assign(ns, 0);
    for (int q = 0; q < ns; ++q) n[root[q]] += F.sn_w[q];
    double bytes = 0, flops = 0;
    int piv[4] = {0, 0, 0, 0};  // at most three limits
    for (int q = 0; q < ns; ++q)
      if (root[q] == q) {
        const double a = n[q], r = F.sn_r[q];
        bytes += 8.0 * (a * a + 2 * a * r);
        flops += 1.5 * (a + r) * (a + r) * a;
        piv[tier[q]] = std::max(piv[tier[q]], (n[q] + kBlkPivot - 1) / kBlkPivot);
      }
    int used = 0, steps = 0;
    for (int p : piv) { used += p > 0; steps += p; }
    return (2 * used - 1) * kPhaseUs + bytes / kBytesPerUs + (steps * kPivotUs + flops / kFlopsPerUs) / kSolvesPerBuild;
  }
};

int even(int v) { return (v + 1) & ~1; }

}  // namespace

bool plan_blocks_with(const SupernodalFactor& F, const SparseSym& Hs, const std::vector<int>& taus, int64_t max_doubles,
                      BlockPlan& P) {
  P = BlockPlan();
  const int ns = F.nsuper, N = F.n;
  if (ns == 0) return false;
  const Tree t = subtree(F);
  std::vector<int> tier, root;
  tiers_of(F, t, taus, tier, root);
  // empty tiers drop out
  std::vector<int> used(taus.size() + 1, 0), tid(taus.size() + 1, 0);
  for (int q = 0; q < ns; ++q) used[tier[q]] = 1;
  for (size_t k = 0; k < used.size(); ++k)
    if (used[k]) tid[k] = P.tiers++;
  std::vector<int> n(ns, 0);
  for (int q = 0; q < ns; ++q) n[root[q]] += F.sn_w[q];
  std::vector<int> roots;
  for (int q = 0; q < ns; ++q)
    if (root[q] == q) roots.push_back(q);
  std::stable_sort(roots.begin(), roots.end(), [&](int a, int b) {
    if (tier[a] != tier[b]) return tier[a] < tier[b];
    return (n[a] + kBlkPivot - 1) / kBlkPivot > (n[b] + kBlkPivot - 1) / kBlkPivot;
  });
  const int nb = (int)roots.size();
  std::vector<int> bid(ns, -1);
  for (int b = 0; b < nb; ++b) bid[roots[b]] = b;
  P.N = N;
  P.blk.resize(nb);
  P.tier_ptr.assign(P.tiers + 1, 0);
  P.vblk.assign(N, 0);
  for (int q = 0; q < ns; ++q)
    for (int c = 0; c < F.sn_w[q]; ++c) P.vblk[F.sn_c0[q] + c] = bid[root[q]];
  int64_t cof = 0, rof = 0, fr = 0, pa = 0, so = 0;
  for (int b = 0; b < nb; ++b) {
    const int q = roots[b];
    BlockInfo& B = P.blk[b];
    B.n = n[q];
    B.r = F.sn_r[q];
    B.np = (B.n + kBlkPivot - 1) / kBlkPivot;
    const int64_t m = (int64_t)B.np * kBlkPivot + B.r;
    if (m > 30000) return false;  // a front's offsets and tile counts stay within 32 bits
    B.M = (int)((m + kBlkTile - 1) / kBlkTile) * kBlkTile;
    B.tier = tid[tier[q]];
    B.parent = F.sn_parent[q] >= 0 ? bid[root[F.sn_parent[q]]] : -1;
    B.cofs = (int)cof;
    B.rofs = (int)rof;
    B.ldx = even(B.n);
    B.ldr = even(B.r);
    B.front = fr;
    B.panel = pa;
    B.xp = so;
    B.pt = so + (int64_t)(B.n + B.r) * B.ldx;
    B.pivofs = b;
    cof += B.n;
    rof += B.r;
    fr += (int64_t)B.M * B.M;
    pa += 2 * (int64_t)B.M * kBlkPivot;
    so = B.pt + (int64_t)B.n * B.ldr;
    P.tier_ptr[B.tier + 1] = b + 1;
  }
  P.front_doubles = fr;
  P.panel_doubles = pa;
  P.solve_doubles = so;
  if (fr + pa + so > max_doubles || rof > INT32_MAX / 4) return false;
  // columns (ascending vertex ids) and rows
  P.cols.resize(N);
  P.rows.resize(rof);
  P.rmap.assign(rof, 0);
  std::vector<int> fill(nb, 0), cpos(N, 0);
  for (int i = 0; i < N; ++i) {
    const int b = P.vblk[i];
    cpos[i] = fill[b];
    P.cols[P.blk[b].cofs + fill[b]++] = i;
  }
  for (int b = 0; b < nb; ++b)
    std::copy(F.rowidx.begin() + F.sn_rofs[roots[b]], F.rowidx.begin() + F.sn_rofs[roots[b]] + P.blk[b].r,
              P.rows.begin() + P.blk[b].rofs);
  auto index_in = [&](int b, int v) -> int {  // vertex v in block b's padded front
    const BlockInfo& B = P.blk[b];
    if (P.vblk[v] == b) return cpos[v];
    const int* R = P.rows.data() + B.rofs;
    const int* p = std::lower_bound(R, R + B.r, v);
    if (p == R + B.r || *p != v) return -1;
    return B.np * kBlkPivot + (int)(p - R);
  };
  for (int b = 0; b < nb; ++b) {
    const BlockInfo& B = P.blk[b];
    for (int a = 0; a < B.r; ++a) {
      const int k = B.parent >= 0 ? index_in(B.parent, P.rows[B.rofs + a]) : -1;
      if (k < 0) return false;  // (cannot happen for a valid tree)
      P.rmap[B.rofs + a] = k;
    }
  }
  // contributions: slots grouped by destination vertex, blocks in order
  P.vptr.assign(N + 1, 0);
  for (int v : P.rows) P.vptr[v + 1]++;
  for (int i = 0; i < N; ++i) P.vptr[i + 1] += P.vptr[i];
  P.cslot.resize(rof);
  {
    std::vector<int> f(P.vptr.begin(), P.vptr.end() - 1);
    for (size_t k = 0; k < P.rows.size(); ++k) P.cslot[k] = f[P.rows[k]]++;
  }
  // tiles
  P.tier_tile.assign(P.tiers + 1, 0);
  std::vector<int> tile0(nb, 0);
  for (int b = 0; b < nb; ++b) {
    const int nt = P.blk[b].M / kBlkTile;
    tile0[b] = (int)P.tiles.size();
    for (int I = 0; I < nt; ++I)
      for (int J = 0; J <= I; ++J) P.tiles.push_back(BlockTile{b, I, J, 0, 0, 0, 0});
    P.tier_tile[P.blk[b].tier + 1] = (int)P.tiles.size();
  }
  // entries of Hs: (i, j) with j eliminated first (or in the same block, both halves of a diagonal tile)
  // in the order of their tiles, within a tile in their own order
  const size_t nnz = (size_t)Hs.ptr[N], nt = P.tiles.size();
  std::vector<int> at(nnz, -1), loc(nnz), hp(nt + 1, 0);
  for (int i = 0; i < N; ++i)
    for (int64_t k = Hs.ptr[i]; k < Hs.ptr[i + 1]; ++k) {
      const int j = Hs.col[k];
      const int b = P.vblk[std::min(i, j)];
      const int fi = index_in(b, i), fj = index_in(b, j);
      if (fi < 0 || fj < 0) return false;
      const int I = fi / kBlkTile, J = fj / kBlkTile;
      if (I < J) continue;  // the other half of the symmetric matrix
      at[k] = tile0[b] + I * (I + 1) / 2 + J;
      loc[k] = (fi % kBlkTile) * kBlkTile + fj % kBlkTile;
      hp[at[k] + 1]++;
    }
  for (size_t q = 0; q < nt; ++q) hp[q + 1] += hp[q];
  P.hs_idx.resize(hp[nt]);
  P.hs_loc.resize(hp[nt]);
  {
    std::vector<int> f(hp.begin(), hp.end() - 1);
    for (size_t k = 0; k < nnz; ++k)
      if (at[k] >= 0) {
        P.hs_idx[f[at[k]]] = (int)k;
        P.hs_loc[f[at[k]]++] = loc[k];
      }
  }
  std::vector<std::vector<int>> kids(nb);
  for (int b = 0; b < nb; ++b)
    if (P.blk[b].parent >= 0) kids[P.blk[b].parent].push_back(b);
  for (size_t q = 0; q < P.tiles.size(); ++q) {
    BlockTile& T = P.tiles[q];
    T.hs0 = hp[q];
    T.hs1 = hp[q + 1];
    T.kid0 = (int)P.kids.size();
    for (int d : kids[T.blk]) {
      const int* m = P.rmap.data() + P.blk[d].rofs;
      const int r = P.blk[d].r;
      auto lo = [&](int v) { return (int)(std::lower_bound(m, m + r, v) - m); };  // rmap ascends with the rows
      const BlockKid K{d, lo(T.I * kBlkTile), lo((T.I + 1) * kBlkTile), lo(T.J * kBlkTile), lo((T.J + 1) * kBlkTile)};
      if (K.i1 > K.i0 && K.j1 > K.j0) P.kids.push_back(K);
    }
    T.kid1 = (int)P.kids.size();
  }
  return true;
}

bool plan_blocks(const SupernodalFactor& F, const SparseSym& Hs, int64_t max_doubles, BlockPlan& P) {
  const Tree t = subtree(F);
  std::vector<int> cand;
  for (int c = 48; c < F.n; c = c * 4 / 3 + 1) cand.push_back(c);
  // thin the candidates of scenes with very many supernodes (the search is per candidate tuple and supernode)
  std::vector<int> best;
  CostModel cost{F, t, {}, {}, {}};
  double bc = cost({});
  auto consider = [&](const std::vector<int>& v) {
    const double c = cost(v);
    if (c < bc) { bc = c; best = v; }
  };
  const size_t nc = cand.size(), step = F.nsuper > 4000 ? 2 : 1;
  for (size_t a = 0; a < nc; ++a) consider({cand[a]});
  for (size_t a = 0; a < nc; a += step)
    for (size_t b = a + 1; b < nc; b += step) consider({cand[a], cand[b]});
  if (F.n > 4096)
    for (size_t a = 0; a < nc; a += 2)
      for (size_t b = a + 2; b < nc; b += 2)
        for (size_t c = b + 2; c < nc; c += 2) consider({cand[a], cand[b], cand[c]});
  return plan_blocks_with(F, Hs, best, max_doubles, P);
}

void block_shares(const BlockPlan& P, int G, std::vector<BlockChunk>& chunks, std::vector<int>& ptr) {
  chunks.clear();
  const int phases = 2 * P.tiers - 1;
  ptr.assign((size_t)phases * (G + 1), 0);
  for (int p = 0; p < phases; ++p) {
    const bool fwd = p < P.tiers;
    const int tier = fwd ? p : 2 * P.tiers - 2 - p, b0 = P.tier_ptr[tier], b1 = P.tier_ptr[tier + 1], nb = b1 - b0;
    // a row costs its products and a fixed part (reduction, epilogue)
    auto rows = [&](const BlockInfo& B) { return fwd ? B.n + B.r : B.n; };
    auto width = [&](const BlockInfo& B) { return (fwd ? B.n : B.r) + 64; };
    std::vector<double> cost(nb);
    std::vector<std::vector<BlockChunk>> mine(G);
    for (int k = 0; k < nb; ++k) cost[k] = (double)rows(P.blk[b0 + k]) * width(P.blk[b0 + k]);
    if (nb <= G) {
      // whole CTAs per block, given one by one to the block with the largest
      // share: a CTA with parts of two blocks would stage twice, and every
      // phase ends with its slowest CTA
      std::vector<int> ctas(nb, 1);
      for (int left = G - nb; left > 0; --left) {
        int best = -1;
        for (int k = 0; k < nb; ++k)
          if (ctas[k] < rows(P.blk[b0 + k]) && (best < 0 || cost[k] / ctas[k] > cost[best] / ctas[best])) best = k;
        if (best < 0) break;
        ++ctas[best];
      }
      int c = 0;
      for (int k = 0; k < nb; ++k) {
        const int R = rows(P.blk[b0 + k]), m = ctas[k];
        for (int q = 0; q < m; ++q, ++c) {
          const int r0 = (int)((int64_t)R * q / m), r1 = (int)((int64_t)R * (q + 1) / m);
          if (r1 > r0) mine[c].push_back(BlockChunk{b0 + k, r0, r1 - r0});
        }
      }
    } else {  // whole blocks, the largest first, each to the CTA with the least
      std::vector<int> order(nb);
      std::iota(order.begin(), order.end(), 0);
      std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return cost[x] > cost[y]; });
      std::vector<double> load(G, 0.0);
      for (int k : order) {
        const int c = (int)(std::min_element(load.begin(), load.end()) - load.begin());
        load[c] += cost[k];
        if (rows(P.blk[b0 + k]) > 0) mine[c].push_back(BlockChunk{b0 + k, 0, rows(P.blk[b0 + k])});
      }
    }
    for (int c = 0; c < G; ++c) {
      ptr[(size_t)p * (G + 1) + c] = (int)chunks.size();
      chunks.insert(chunks.end(), mine[c].begin(), mine[c].end());
    }
    ptr[(size_t)p * (G + 1) + G] = (int)chunks.size();
  }
}

}  // namespace dfem
