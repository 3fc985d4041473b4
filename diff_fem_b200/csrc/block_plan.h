// block_plan.h — plan of the block-inverse form of the global solve (the
// "dense" solve form), for single scenes.
//
// The elimination tree's supernodes are merged into a few tiers of blocks:
// tier 0 the subtrees of at most tau_0 columns, tier t the connected rest of
// the subtrees of at most tau_t columns, the last tier what is left at the
// top.  A block B has its columns C_B and the rows R_B below them (the row
// structure of its topmost supernode, all in blocks of later tiers).  With
//   X_B = L_BB^-T L_BB^-1,   P_B = L_RB L_BB^-1
// (dense; the zeros inside a block are kept) a solve of Hs x = b is
//   tier 0, 1, ...:  t_B = b_B - sum over blocks D below B of (P_D t_D)_B,  y_B = X_B t_B
//   ... 1, 0:        x_B = y_B - P_B^T x_R
// — 2 tiers - 1 dependent phases of independent dense products instead of two
// sweeps over the elimination tree's levels.  One tier is X = Hs^-1 itself.
//
// X_B, P_B and the update passed on to the parent come from symmetric
// Gauss-Jordan sweeps of the block's front [A_CC A_CR; A_RC 0] plus its
// children's updates (multifrontal, block_inverse.cuh).
#pragma once
#include <cstdint>
#include <vector>

#include "cholesky.h"

namespace dfem {

constexpr int kBlkTile = 64;    // output tile of a sweep
constexpr int kBlkPivot = 32;   // columns swept at once

struct BlockInfo {
  int n, r;              // columns, rows below
  int np, M;             // pivots of kBlkPivot columns; padded front size (columns to np kBlkPivot, then rows)
  int tier, parent;
  int cofs, rofs;        // cols[cofs .. + n), rows[rofs .. + r): internal vertex ids, ascending
  int ldx, ldr;          // row lengths of [X; P] (n, even) and P^T (r, even)
  int64_t front;         // M x M, row-major
  int64_t panel;         // two M x kBlkPivot panels
  int64_t xp;            // [X; P]: (n + r) x ldx, row-major
  int64_t pt;            // P^T: n x ldr, row-major
  int pivofs;            // first pivot inverse (two slots of kBlkPivot^2 per block)
};

// lower tile (I, J) of a front and what is assembled into it
struct BlockTile {
  int blk, I, J;
  int hs0, hs1;          // entries of Hs: hs_idx / hs_loc [hs0, hs1)
  int kid0, kid1;        // children's update ranges: kids [kid0, kid1)
};
struct BlockKid {
  int blk;               // the child
  int i0, i1, j0, j1;    // its rows (positions in R) that land in the tile's rows / columns
};
// rows [row0, row0 + rows) of a block's product in one phase of the solve, done by one CTA
struct BlockChunk {
  int blk, row0, rows;
};

struct BlockPlan {
  int N = 0, tiers = 0;
  std::vector<BlockInfo> blk;                   // by tier; within a tier the most pivots first
  std::vector<int> tier_ptr;                    // tiers + 1
  std::vector<int> cols, rows, rmap;            // rmap: a row's index in the parent's padded front
  std::vector<int> vblk;                        // block of every vertex
  // contributions (P_D t_D): row a of block D writes slot cslot[rofs + a]; vertex i sums slots
  // [vptr[i], vptr[i + 1]) in order
  std::vector<int> cslot, vptr;
  // fronts
  std::vector<BlockTile> tiles;                 // by tier, blocks in order
  std::vector<int> tier_tile;                   // tiers + 1 into tiles
  std::vector<BlockKid> kids;
  std::vector<int> hs_idx, hs_loc;              // entry of Hs (index into its values), place in the tile (row * kBlkTile + col)
  int64_t front_doubles = 0, panel_doubles = 0, solve_doubles = 0;
};

// Chooses the tiers by the cost model and lays the blocks out.
// max_doubles: limit of the stored doubles (fronts, panels and products).
bool plan_blocks(const SupernodalFactor& F, const SparseSym& Hs, int64_t max_doubles, BlockPlan& P);

// The same with given tier limits (ascending; empty: one block).
bool plan_blocks_with(const SupernodalFactor& F, const SparseSym& Hs, const std::vector<int>& taus, int64_t max_doubles,
                      BlockPlan& P);

// Shares of every phase for G CTAs (phase p: tier p forward for p < tiers, else tier 2 tiers - 2 - p
// backward): chunks ptr[p * (G + 1) + c] .. ptr[p * (G + 1) + c + 1) of CTA c.
void block_shares(const BlockPlan& P, int G, std::vector<BlockChunk>& chunks, std::vector<int>& ptr);

}  // namespace dfem
