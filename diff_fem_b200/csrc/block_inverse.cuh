// block_inverse.cuh — the block-inverse form of the global solve: building
// X_B and P_B of every block (block_plan.h) and solving with them.
//
// Build (k_block_factor, one cooperative launch): tier by tier, the blocks'
// fronts are assembled (entries of Hs, the children's updates in order) and
// swept: a symmetric Gauss-Jordan sweep of the pivot columns K,
//   D = F_KK^-1;  F_ij -= F_iK D F_Kj;  F_iK = F_iK D;  F_KK = -D,
// which after the block's n columns leaves -X, P and the update U = F_RR in
// place.  With Z_i = F_iK outside K and -e_i inside it, every element of the
// swept matrix is (F_ij, 0 where i or j is in K) - (Z_i D) Z_j^T, so a sweep
// is the same two products (FP64 tensor cores) for every 64 x 64 tile of the
// lower half.  A tile belongs to one CTA, which keeps it in shared memory
// (its first kBfRes tiles; the others in the front's own storage) for all
// sweeps of the tier; between sweeps only the panel Z of the next pivot and
// its inverse D go through global memory, and one grid-wide barrier separates
// sweeps.  The CTA of the tile that holds the next pivot inverts it before
// the barrier.  All values have one writer and a fixed order: the result is
// deterministic.  A pivot that is not positive (or not finite) raises bit 0 of
// the failure word, as the supernodal factor does; the host retries with the
// next regularisation.  A barrier that gave up raises bit 1 (kBuildGaveUp).
// Invalid materials (the word after it) leave everything as it was.  12,800-tet beam (10 blocks of up to 373 columns and a top
// one of 693): 34 pivots of 11.1 us, 0.38 ms (a first version: 16 us each).
//
// Solve: 2 tiers - 1 phases of row products, see block_solve.
#pragma once

// (included by engine.cu after pd_kernels.cu and factor_kernels.cuh)
#include "block_plan.h"
#include "factor_kernels.cuh"

namespace dfem {

struct BlockDev {
  int N, tiers, nblk, G;          // G: CTAs of the solve's shares
  const BlockInfo* blk;
  const BlockTile* tiles;
  const int* tier_tile;
  const BlockKid* kids;
  const int* hs_idx;
  const int* hs_loc;
  const int* cols;
  const int* rows;
  const int* rmap;
  const int* cslot;
  const int* vptr;
  const BlockChunk* chunks;
  const int* share;               // (2 tiers - 1) x (G + 1)
  double* front;                  // lower tiles of every front (assembled there past kBfRes tiles; updates U)
  double* panel;                  // two panels Z (M x kBlkPivot) per block
  double* sol;                    // [X; P] and P^T of every block
  double* piv;                    // two pivot inverses per block
  double* contrib;                // 3 per row of every block
  unsigned* bar;                  // grid barrier: arrivals, CTAs done
  int* status;
  int spin_tries;                 // polls of a grid barrier before it gives up
  int vec;                        // doubles of one staged component (largest n or r, even)
};

// ------------------------------------------------------------- barriers ----
//
// Barrier over a cooperative launch (every CTA resident): arrivals counted in
// global memory, thread 0 polls (acquire) until all CTAs of this round have
// come, at most `tries` times.  1.2 us on 148 CTAs; a barrier of one
// cluster takes 0.25 us.  sync() is false, in every thread of the CTA, when
// the wait gave up (status 6, wait kWaitGrid): the caller returns.  The
// counters are then left as they are until the host has seen the status and
// cleared both (reset_barriers): a launch that finds the status so on entry
// returns at once (gave_up).
constexpr int kWaitGrid = 14;

struct GridBarrier {
  unsigned* c;
  int* status;
  int tries;
  unsigned target = 0;
  __device__ GridBarrier(unsigned* c_, int* s_, int t_) : c(c_), status(s_), tries(t_) {}
  __device__ static bool gave_up(const int* s) {
    return __syncthreads_or(threadIdx.x == 0 && *(const volatile int*)(s + 2) == kWaitGrid) != 0;
  }
  __device__ static int cta() { return blockIdx.x; }
  __device__ static int ctas() { return gridDim.x; }
  __device__ bool sync() {
    __syncthreads();
    int ok = 1;
    if (threadIdx.x == 0) {
      target += gridDim.x;
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(c) : "memory");
      ok = 0;
#pragma unroll 1
      for (int k = 0; k < tries; ++k) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(c) : "memory");
        if ((int)(v - target) >= 0) { ok = 1; break; }
      }
      if (!ok) {
        status[0] = 6;
        status[2] = kWaitGrid;
        atomicAdd(status + 3, 1);
      }
    }
    return __syncthreads_and(ok) != 0;
  }
  // after the last barrier: the last CTA to leave readies the counters for the next launch
  __device__ void leave() {
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      if (atomicAdd(c + 1, 1u) == gridDim.x - 1) {
        c[0] = 0u;
        c[1] = 0u;
      }
    }
  }
};

// The same over one thread-block cluster (the grid is one cluster).
struct ClusterBarrier {
  __device__ ClusterBarrier(unsigned*, int*, int) {}
  __device__ static bool gave_up(const int*) { return false; }
  __device__ static int cta() { return (int)cluster_rank(); }
  __device__ static int ctas() { return gridDim.x; }
  __device__ bool sync() {
    cluster_sync_all();
    return true;
  }
  __device__ void leave() {}
};

// ---------------------------------------------------------------- build ----

constexpr int kBuildGaveUp = 2;
constexpr int kBfThreads = 512;   // one CTA per SM: sixteen warps, 16 x 16 of a tile's output each
constexpr int kBfOwn = 32;        // tiles of a CTA whose descriptors are kept in shared memory
constexpr int kBfRes = 4;         // tiles of a CTA kept in shared memory
constexpr int kBfLd = kBlkPivot + 4;  // shared row of a 32-wide operand: the DMMA fragments read 16 banks at once
constexpr int kBfTld = kBlkTile + 8;  // shared row of a tile: the fragments' 16-byte accesses touch distinct banks
struct BfTile {
  BlockTile t;
  BlockInfo b;
};
constexpr int kBfOps = 3 * kBlkTile * kBfLd + kBlkPivot * kBfLd;  // Z_I, Z_J, G, D
constexpr size_t kBfSmem = sizeof(double) * (kBfOps + 2 * 4 * kBlkPivot + (size_t)kBfRes * kBlkTile * kBfTld) +
                           sizeof(BfTile) * kBfOwn;
static_assert(3 * kBlkTile * kBfLd >= kBlkTile * kBfTld, "a tile past the resident ones is assembled in the operands' space");

// D = A^-1 of the symmetric positive definite A (32 x 32 at A, row length ld,
// lower half) by sweeps of 2 x 2 pivots, to out (32 x 32).  Warp w holds rows
// 2 w and 2 w + 1, a lane two columns of one of them, in registers; the warp
// that owns a step's pivot rows publishes them, and their products with the
// inverse of the pivot, through shared memory (zz: 2 x 4 x 32 doubles, used
// in turn): sixteen dependent steps of one barrier each, 0.33 K cycles a step
// (with every warp reading the whole matrix from shared memory and forming
// the pivot's inverse itself: 0.8 K).  True when a pivot is not positive.
__device__ __forceinline__ bool invert_pivot(const double* A, int ld, double* zz, double* out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, i = 2 * warp + (lane >> 4), j0 = 2 * (lane & 15);
  bool bad = false;
  double a0 = i >= j0 ? A[i * ld + j0] : A[j0 * ld + i], a1 = i >= j0 + 1 ? A[i * ld + j0 + 1] : A[(j0 + 1) * ld + i];
  auto publish = [&](int k) {  // by warp k / 2: rows k, k + 1 with -I in the pivot's place, and their products
    double* z = zz + ((k >> 1) & 1) * 4 * kBlkPivot;
    const int src = k >> 1;
    const double p = __shfl_sync(0xffffffffu, a0, src), q = __shfl_sync(0xffffffffu, a1, src),
                 r = __shfl_sync(0xffffffffu, a1, 16 + src);
    const double det = fma(p, r, -q * q), id = 1.0 / det;
    bad |= !(p > 0.0) || !(det > 0.0) || !isfinite(det) || !(id > 0.0) || !isfinite(id);
    const bool mine = (lane & 15) == src;
    const double z0 = mine ? (lane < 16 ? -1.0 : 0.0) : a0, z1 = mine ? (lane < 16 ? 0.0 : -1.0) : a1;
    // row k in lanes 0 .. 15, row k + 1 in lanes 16 .. 31
    const double o0 = __shfl_xor_sync(0xffffffffu, z0, 16), o1 = __shfl_xor_sync(0xffffffffu, z1, 16);
    const double m = lane < 16 ? r * id : p * id, n = -q * id;
    double2* row = reinterpret_cast<double2*>(z + (lane >> 4) * kBlkPivot + j0);
    double2* prd = reinterpret_cast<double2*>(z + (2 + (lane >> 4)) * kBlkPivot + j0);
    *row = make_double2(z0, z1);
    *prd = make_double2(fma(z0, m, o0 * n), fma(z1, m, o1 * n));
  };
  if (warp == 0) publish(0);
#pragma unroll 1
  for (int k = 0; k < kBlkPivot; k += 2) {
    __syncthreads();
    const double* z = zz + ((k >> 1) & 1) * 4 * kBlkPivot;
    const double2 y0 = *reinterpret_cast<const double2*>(z + j0), y1 = *reinterpret_cast<const double2*>(z + kBlkPivot + j0);
    const double g0 = z[2 * kBlkPivot + i], g1 = z[3 * kBlkPivot + i];
    const bool in = warp == (k >> 1) || (lane & 15) == (k >> 1);
    a0 = fma(-g1, y1.x, fma(-g0, y0.x, in ? 0.0 : a0));
    a1 = fma(-g1, y1.y, fma(-g0, y0.y, in ? 0.0 : a1));
    if (k + 2 < kBlkPivot && warp == (k >> 1) + 1) publish(k + 2);
  }
  *reinterpret_cast<double2*>(out + i * kBlkPivot + j0) = make_double2(-a0, -a1);
  return bad;
}

// Tile (I, J) (ld kBfTld, shared or ld in global memory) into the panel of the
// pivot [32 s, 32 s + 32), if it holds its columns (J = s / 2: Z of row tile
// I) or rows (I = s / 2 > J: Z of row tile J, transposed).
__device__ __forceinline__ void write_panel(const double* Tl, int ld, int I, int J, int s, double* panel) {
  const int K0 = s * kBlkPivot, Kt = s / 2, o = K0 - Kt * kBlkTile;
  if (J == Kt) {
#pragma unroll
    for (int u = 0; u < kBlkTile * kBlkPivot / 2 / kBfThreads; ++u) {
      const int q = threadIdx.x + kBfThreads * u, r = q >> 4, c = 2 * (q & 15), g = I * kBlkTile + r;
      double2 v = *reinterpret_cast<const double2*>(Tl + (size_t)r * ld + o + c);
      if (g >= K0 && g < K0 + kBlkPivot) v = make_double2(g == K0 + c ? -1.0 : 0.0, g == K0 + c + 1 ? -1.0 : 0.0);
      *reinterpret_cast<double2*>(panel + (size_t)g * kBlkPivot + c) = v;
    }
  } else if (I == Kt) {
    for (int q = threadIdx.x; q < kBlkTile * kBlkPivot; q += kBfThreads) {
      const int r = q & (kBlkTile - 1), c = q / kBlkTile;
      panel[(size_t)(J * kBlkTile + r) * kBlkPivot + c] = Tl[(size_t)(o + c) * ld + r];
    }
  }
}

__global__ void __launch_bounds__(kBfThreads, 1) k_block_factor(BlockDev b, const double* __restrict__ hs_val,
                                                                 const double* __restrict__ reg_p, int* fail) {
  extern __shared__ __align__(16) double bfsh[];
  double* ZI = bfsh;
  double* ZJ = ZI + kBlkTile * kBfLd;
  double* Gs = ZJ + kBlkTile * kBfLd;
  double* Ds = Gs + kBlkTile * kBfLd;
  double* zz = bfsh + kBfOps;
  double* res = zz + 2 * 4 * kBlkPivot;
  BfTile* own = reinterpret_cast<BfTile*>(res + (size_t)kBfRes * kBlkTile * kBfTld);
  if (fail[1]) return;  // uniform, before any barrier
  if (GridBarrier::gave_up(b.status)) {
    if (threadIdx.x == 0) atomicOr(fail, kBuildGaveUp);
    return;
  }
  GridBarrier bar(b.bar, b.status, b.spin_tries);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double reg = reg_p[0];
  bool bad = false;
  for (int t = 0; t < b.tiers; ++t) {
    const int q0 = b.tier_tile[t], q1 = b.tier_tile[t + 1];
    const int nown = q0 + (int)blockIdx.x < q1 ? (q1 - q0 - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    __syncthreads();
    for (int k = tid; k < min(nown, kBfOwn); k += kBfThreads) {
      own[k].t = b.tiles[q0 + blockIdx.x + k * gridDim.x];
      own[k].b = b.blk[own[k].t.blk];
    }
    // assembly: identity padding, entries of Hs, children's updates; the first pivot's panel and inverse
    for (int k = 0; k < nown; ++k) {
      const BlockTile T = b.tiles[q0 + blockIdx.x + k * gridDim.x];
      const BlockInfo B = b.blk[T.blk];
      double* S = k < kBfRes ? res + (size_t)k * kBlkTile * kBfTld : bfsh;
      __syncthreads();
      for (int e = tid; e < kBlkTile * kBlkTile; e += kBfThreads) {
        const int g = T.I * kBlkTile + (e >> 6);
        S[(e >> 6) * kBfTld + (e & 63)] =
            (T.I == T.J && (e >> 6) == (e & 63) && g >= B.n && g < B.np * kBlkPivot) ? 1.0 : 0.0;
      }
      __syncthreads();
      for (int e = T.hs0 + tid; e < T.hs1; e += kBfThreads) {
        const int r = b.hs_loc[e] >> 6, c = b.hs_loc[e] & 63;
        S[r * kBfTld + c] += hs_val[b.hs_idx[e]] + ((T.I == T.J && r == c) ? reg : 0.0);
      }
      for (int c = T.kid0; c < T.kid1; ++c) {
        const BlockKid C = b.kids[c];
        const BlockInfo D = b.blk[C.blk];
        const double* U = b.front + D.front;
        const int* map = b.rmap + D.rofs;
        const int p0 = D.np * kBlkPivot, nj = C.j1 - C.j0, cnt = (C.i1 - C.i0) * nj;
        __syncthreads();
        for (int e = tid; e < cnt; e += kBfThreads) {
          const int i = C.i0 + e / nj, j = C.j0 + e % nj;
          const double u = __ldcg(U + (size_t)(p0 + max(i, j)) * D.M + p0 + min(i, j));
          S[(map[i] - T.I * kBlkTile) * kBfTld + map[j] - T.J * kBlkTile] += u;
        }
      }
      __syncthreads();
      if (k >= kBfRes) {
        double* F = b.front + B.front + (size_t)T.I * kBlkTile * B.M + T.J * kBlkTile;
        for (int e = tid; e < kBlkTile * kBlkTile; e += kBfThreads)
          F[(size_t)(e >> 6) * B.M + (e & 63)] = S[(e >> 6) * kBfTld + (e & 63)];
      }
      write_panel(S, kBfTld, T.I, T.J, 0, b.panel + B.panel);
      if (T.I == 0) bad |= invert_pivot(S, kBfTld, zz, b.piv + (size_t)2 * B.pivofs * kBlkPivot * kBlkPivot);
    }
    if (!bar.sync()) {
      if (tid == 0) atomicOr(fail, kBuildGaveUp);
      return;
    }
    int steps = 0;
    if (q0 < q1) steps = b.blk[b.tiles[q0].blk].np;  // the tier's first block has the most pivots
    for (int s = 0; s < steps; ++s) {
      const int K0 = s * kBlkPivot;
      const int nt = (s + 1) / 2;  // tile of the next pivot
      // own tiles: those holding a next pivot first (their CTA inverts it), then the others
      for (int pass = 0; pass < 2; ++pass)
        for (int k = 0; k < nown; ++k) {
          BlockTile T;
          BlockInfo B;
          if (k < kBfOwn) {
            T = own[k].t;
            B = own[k].b;
          } else {
            T = b.tiles[q0 + blockIdx.x + k * gridDim.x];
            B = b.blk[T.blk];
          }
          if (s >= B.np) break;  // blocks are ordered by their pivots
          const bool last = s == B.np - 1, next = !last && T.I == nt && T.J == nt;
          if (next != (pass == 0)) continue;
          const double* Z = b.panel + B.panel + (size_t)(s & 1) * B.M * kBlkPivot;
          const double* D = b.piv + (size_t)(2 * B.pivofs + (s & 1)) * kBlkPivot * kBlkPivot;
          const double2* zi = reinterpret_cast<const double2*>(Z + (size_t)T.I * kBlkTile * kBlkPivot);
          const double2* zj = reinterpret_cast<const double2*>(Z + (size_t)T.J * kBlkTile * kBlkPivot);
          const double2 dv = __ldcg(reinterpret_cast<const double2*>(D) + tid);
          const double2 i0 = __ldcg(zi + tid), i1 = __ldcg(zi + tid + kBfThreads);
          const double2 j0 = __ldcg(zj + tid), j1 = __ldcg(zj + tid + kBfThreads);
          __syncthreads();  // the operands' readers of the tile before
          {
            const int r = tid >> 4, c = 2 * (tid & 15);
            *reinterpret_cast<double2*>(Ds + r * kBfLd + c) = dv;
            *reinterpret_cast<double2*>(ZI + r * kBfLd + c) = i0;
            *reinterpret_cast<double2*>(ZI + (r + 32) * kBfLd + c) = i1;
            *reinterpret_cast<double2*>(ZJ + r * kBfLd + c) = j0;
            *reinterpret_cast<double2*>(ZJ + (r + 32) * kBfLd + c) = j1;
          }
          __syncthreads();
          {  // G = -Z_I D (rows 8 (warp & 7) .., columns 16 (warp >> 3) ..)
            double g[2][2];
            g[0][0] = g[0][1] = g[1][0] = g[1][1] = 0.0;
            const int gr = 8 * (warp & 7) + (lane >> 2), gc = 16 * (warp >> 3);
#pragma unroll
            for (int kk = 0; kk < kBlkPivot; kk += 4) {
              const double av = ZI[gr * kBfLd + kk + (lane & 3)];
#pragma unroll
              for (int j = 0; j < 2; ++j)
                dmma_8x8x4(g[j][0], g[j][1], av, Ds[(gc + 8 * j + (lane >> 2)) * kBfLd + kk + (lane & 3)]);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
              *reinterpret_cast<double2*>(Gs + gr * kBfLd + gc + 8 * j + 2 * (lane & 3)) = make_double2(-g[j][0], -g[j][1]);
          }
          // the tile's own values in the layout of the products: rows 16 (warp & 3) + 8 i + (lane >> 2),
          // columns 16 (warp >> 2) + 8 j + 2 (lane & 3) + {0, 1}
          const int r0 = 16 * (warp & 3) + (lane >> 2), c0 = 16 * (warp >> 2) + 2 * (lane & 3);
          const bool inres = k < kBfRes;
          double* Tl = inres ? res + (size_t)k * kBlkTile * kBfTld
                             : b.front + B.front + (size_t)T.I * kBlkTile * B.M + T.J * kBlkTile;
          const int tld = inres ? kBfTld : B.M;
          double d[2][2][2];
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const int gi = T.I * kBlkTile + r0 + 8 * i, gj = T.J * kBlkTile + c0 + 8 * j;
              const double2 v = *reinterpret_cast<const double2*>(Tl + (size_t)(r0 + 8 * i) * tld + c0 + 8 * j);
              const bool in = (gi >= K0 && gi < K0 + kBlkPivot) || (gj >= K0 && gj < K0 + kBlkPivot);
              d[i][j][0] = in ? 0.0 : v.x;
              d[i][j][1] = in ? 0.0 : v.y;
            }
          __syncthreads();
#pragma unroll
          for (int kk = 0; kk < kBlkPivot; kk += 4) {
            double av[2], bv[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) av[i] = Gs[(r0 + 8 * i) * kBfLd + kk + (lane & 3)];
#pragma unroll
            for (int j = 0; j < 2; ++j) bv[j] = ZJ[(16 * (warp >> 2) + 8 * j + (lane >> 2)) * kBfLd + kk + (lane & 3)];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
              for (int j = 0; j < 2; ++j) dmma_8x8x4(d[i][j][0], d[i][j][1], av[i], bv[j]);
          }
          if (!last) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
              for (int j = 0; j < 2; ++j)
                *reinterpret_cast<double2*>(Tl + (size_t)(r0 + 8 * i) * tld + c0 + 8 * j) =
                    make_double2(d[i][j][0], d[i][j][1]);
            if (T.J == nt || T.I == nt) {  // the next pivot's panel (and its inverse)
              __syncthreads();
              double* Zn = b.panel + B.panel + (size_t)((s + 1) & 1) * B.M * kBlkPivot;
              if (next) {
                const int o = (s + 1) * kBlkPivot - nt * kBlkTile;
                bad |= invert_pivot(Tl + (size_t)o * tld + o, tld, zz,
                                    b.piv + (size_t)(2 * B.pivofs + ((s + 1) & 1)) * kBlkPivot * kBlkPivot);
              }
              write_panel(Tl, tld, T.I, T.J, s + 1, Zn);
            }
            continue;
          }
          // the block is done: -X, P, U
          const int npad = B.np * kBlkPivot;
          double* X = b.sol + B.xp;
          double* PT = b.sol + B.pt;
          double* U = b.front + B.front;
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const int gi = T.I * kBlkTile + r0 + 8 * i, gj = T.J * kBlkTile + c0 + 8 * j + e;
                const double v = d[i][j][e];
                if (gi < B.n) {
                  if (gj <= gi) {
                    X[(size_t)gi * B.ldx + gj] = -v;
                    X[(size_t)gj * B.ldx + gi] = -v;
                  }
                } else if (gi >= npad && gi - npad < B.r) {
                  const int a = gi - npad;
                  if (gj < B.n) {
                    X[(size_t)(B.n + a) * B.ldx + gj] = v;
                    PT[(size_t)gj * B.ldr + a] = v;
                  } else if (gj >= npad && gj <= gi) {
                    U[(size_t)gi * B.M + gj] = v;
                  }
                }
              }
        }
      if (!bar.sync()) {
        if (tid == 0) atomicOr(fail, kBuildGaveUp);
        return;
      }
    }
  }
  if (bad) atomicOr(fail, 1);
  bar.leave();
}

// ---------------------------------------------------------------- solve ----
//
// Phase p < tiers (forward): rows of [X_B; P_B] times t_B = rhs_B minus the
// contributions pushed to B's vertices by the blocks below (each vertex sums
// its own in a fixed order); a row of X_B gives y, a row of P_B the
// contribution to its vertex.  The other phases (backward): y_B -= P_B^T x_R.
// A CTA's share of a phase is a few row ranges of blocks (block_shares): it
// stages the block's vector as x / y / z planes in shared memory; a warp
// takes two rows at a time (each staged value then serves two products: the
// planes are three times the bytes of a row) and, where a share has fewer
// row pairs than warps, a segment of their columns; eight 16-byte loads of
// each row are in flight.  Segments, lanes and the reduction tree are summed
// in a fixed order.  done(v, value) is called once per vertex, by one thread,
// with its solution.
constexpr int kBsThreads = 512;
constexpr int kBsRows = 256;  // rows of a share handled at once
__host__ __device__ inline size_t block_solve_doubles(int vec) { return 3 * (size_t)vec + 3 * 2 * kBsRows; }

__device__ __forceinline__ void row_pair(const double2* __restrict__ r0, const double2* __restrict__ r1, const double2* bx,
                                         const double2* by, const double2* bz, int q0, int q1, double o[2][3]) {
  const int lane = threadIdx.x & 31;
  double a[2][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
  for (int q = q0 + lane; q < q1; q += 256) {
    double2 u[8], w[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int p = q + 32 * k;
      u[k] = p < q1 ? __ldcg(r0 + p) : make_double2(0.0, 0.0);
      w[k] = p < q1 ? __ldcg(r1 + p) : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int p = q + 32 * k;
      if (p < q1) {
        const double2 x = bx[p], y = by[p], z = bz[p];
        a[0][0] += u[k].x * x.x + u[k].y * x.y;
        a[0][1] += u[k].x * y.x + u[k].y * y.y;
        a[0][2] += u[k].x * z.x + u[k].y * z.y;
        a[1][0] += w[k].x * x.x + w[k].y * x.y;
        a[1][1] += w[k].x * y.x + w[k].y * y.y;
        a[1][2] += w[k].x * z.x + w[k].y * z.y;
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) o[r][c] = warp_sum(a[r][c]);
}

template <class BAR, class DONE>
__device__ __forceinline__ bool block_solve(const BlockDev& b, BAR& bar, const double* rhs, double* y, double* sh,
                                            DONE done) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
  double* sx = sh;
  double* sy = sx + b.vec;
  double* sz = sy + b.vec;
  double* part = sz + b.vec;  // 3 x (row, segment): at most 2 kBsRows
  const int phases = 2 * b.tiers - 1;
  for (int p = 0; p < phases; ++p) {
    const bool fwd = p < b.tiers;
    const int* share = b.share + (size_t)p * (b.G + 1) + BAR::cta();
    for (int k = share[0]; k < share[1]; ++k) {
      const BlockChunk C = b.chunks[k];
      const BlockInfo B = b.blk[C.blk];
      const int w = fwd ? B.n : B.r, ld = fwd ? B.ldx : B.ldr;
      __syncthreads();  // the planes' and partials' readers of the chunk before
      for (int i = tid; i < ld; i += blockDim.x) {
        Vec3<double> v = mk3(0.0, 0.0, 0.0);
        if (i < w) {
          if (fwd) {
            const int g = b.cols[B.cofs + i];
            v = ld3(rhs, g);
            if (B.tier > 0)
              for (int q = b.vptr[g]; q < b.vptr[g + 1]; ++q) v = v - ld3(b.contrib, q);
          } else {
            v = ld3(y, b.rows[B.rofs + i]);
          }
        }
        sx[i] = v.x; sy[i] = v.y; sz[i] = v.z;
      }
      __syncthreads();
      const double* mat = b.sol + (fwd ? B.xp : B.pt);
      const int w2 = ld / 2;
      for (int base = 0; base < C.rows; base += kBsRows) {
        const int nr = min(kBsRows, C.rows - base), pairs = (nr + 1) / 2;
        int seg = 1;  // column segments: power of two, up to one per warp and no shorter than 32 pairs of columns
        while (2 * seg * pairs <= nwarp && 64 * seg <= w2) seg *= 2;
        const int len = (w2 + seg - 1) / seg;
        if (base > 0) __syncthreads();
        for (int u = warp; u < pairs * seg; u += nwarp) {
          const int pr = u / seg, sg = u % seg;
          const int ra = C.row0 + base + 2 * pr, rb = min(ra + 1, C.row0 + C.rows - 1);
          const double2* m0 = reinterpret_cast<const double2*>(mat + (size_t)ra * ld);
          const double2* m1 = reinterpret_cast<const double2*>(mat + (size_t)rb * ld);
          double o[2][3];
          row_pair(m0, m1, reinterpret_cast<const double2*>(sx), reinterpret_cast<const double2*>(sy),
                   reinterpret_cast<const double2*>(sz), sg * len, min(w2, (sg + 1) * len), o);
          if (lane == 0) {
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
              for (int c = 0; c < 3; ++c)
                if (2 * pr + r < nr) part[3 * ((2 * pr + r) * seg + sg) + c] = o[r][c];
          }
        }
        __syncthreads();
        for (int r = tid; r < nr; r += blockDim.x) {
          Vec3<double> v = ld3(part, r * seg);
          for (int sg = 1; sg < seg; ++sg) v = v + ld3(part, r * seg + sg);
          const int row = C.row0 + base + r;
          if (fwd && row >= B.n) {
            st3(b.contrib, b.cslot[B.rofs + row - B.n], v);
          } else {
            const int g = b.cols[B.cofs + row];
            if (!fwd) v = ld3(y, g) - v;
            if (!fwd || p == b.tiers - 1) done(g, v);
            else st3(y, g, v);
          }
        }
      }
    }
    if (p + 1 < phases && !bar.sync()) return false;
  }
  return true;
}

// The solve alone, for the paths that launch their kernels one by one.
template <class BAR>
__global__ void __launch_bounds__(kBsThreads, 1) k_block_solve(BlockDev b, Gate gate, const double* rhs, double* y) {
  extern __shared__ __align__(16) double bssh[];
  if (gate.skip(0) || BAR::gave_up(b.status)) return;  // uniform, before any barrier
  BAR bar(b.bar, b.status, b.spin_tries);
  if (!block_solve(b, bar, rhs, y, bssh, [&](int g, Vec3<double> v) { st3(y, g, v); })) return;
  bar.leave();
}

}  // namespace dfem
