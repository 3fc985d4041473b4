// step_kernels.cuh — whole time steps in one launch, for single scenes whose
// solve is the block-inverse form.
//
// k_pd_forward runs n time steps (gravity, right-hand side, the local-global
// iterations with their early exit, velocity update) and k_pd_adjoint their
// reverse, with barriers between the phases of an iteration instead of kernel
// boundaries: local step | slot gather | the solve's phases (the last ones
// update the iterate and its convergence sum).  The launches of the graph
// form cost a conditional node's 12 us per step and 6 us per iteration on the
// B200 besides the kernels themselves; a barrier of the whole grid takes
// 1.2 us, one of a 16-CTA cluster 0.25 us.  Two launch shapes:
//   grid     one CTA per SM, cooperative launch (GridBarrier);
//   cluster  16 CTAs of one thread-block cluster (ClusterBarrier), for scenes
//            small enough that sixteen SMs hold an element per thread and the
//            products stay within their L2 bandwidth (rule: engine.cu).
// A CTA's shares of the solve are the same in every iteration, so their rows
// are copied into shared memory once per launch (as many as fit; the others
// stream from L2), with the tables their staging reads.
//
// Every value has one writer and a fixed order of sums: results are
// deterministic, n steps in one call equal n calls of one step, and a replayed
// step equals the recorded one, bit for bit.
#pragma once

// (included by engine.cu after pd_kernels.cu and block_inverse.cuh)
#include <type_traits>

namespace dfem {

constexpr int kPsThreads = 512;
constexpr int kPsWarps = kPsThreads / 32;
constexpr int kPsChunks = 40;   // row ranges of a CTA over all phases of the solve
constexpr int kPsPair = kPsThreads / 2;  // tets of a CTA in flight (two threads each)
constexpr int kPsXch = 20;               // doubles a pair of threads exchanges

struct PdSteps {
  int n, s0;                    // steps, index of the first
  const int* step;              // when set: n = 1 and the step index is *step
  int K, end;                   // end: 0 leaves out the step's end (contact follows)
  int zero;                     // clear the status word (and the adjoint's accumulators) first
  int ckpt_every;
  double* xt;                   // state, internal order
  double* vt;
  double* qn;
  double* c0;
  double* xk;                   // the iterate (the step's result)
  double* xk2;                  // its other buffer (alternate steps)
  double* rhs;
  double* y;
  double* slot;
  double* hist;
  long long hist_step;
  double* ckpt_x;
  double* ckpt_v;
  const double* act_all;
  double* partial;              // two per CTA
  int* iters;
  int* status;
  double* vwc;
  double* traj;
  const int* to_user;
  const double* x_in;           // user order, device memory (null: the state is in xt / vt)
  const double* v_in;
  double* x_out;                // user order, device memory (null: stays in xt / vt)
  double* v_out;
  const double* X;              // mixed form: Hs^-1, N_p x N_p (dense_solve.cuh)
  int Np;
  int res_doubles;              // shared memory for the solve's rows
  int tab_ints;                 // ... and for its index tables
  // adjoint
  double* xkb;
  double* xtb;
  double* bb;
  double* gE;
  double* gnu;
  double* mg;                   // 2 (M + S): this iteration's activation terms, their sum over the step
  double* gact;
  double* io_a;                 // cotangents of x, v (internal order)
  double* io_b;
  int tape_warps;               // warps of a CTA that run the adjoint local step (the tape's size)
  double* gE_out;               // copies of the accumulators (device memory; may be null)
  double* gnu_out;
  double* gact_out;
};

// A row range of the solve in this CTA's hands.
struct PsChunk {
  int n, r, ld, tier, row0, rows, cofs, rofs;
  const double* mat;            // its rows: shared memory, or the stored products
  const int* idx;               // vertices of the staged vector
  const int* v0;                // forward, tiers > 0: their contribution ranges [v0, v1)
  const int* v1;
  const int* out;               // a row's vertex, or -1 - its contribution slot
};

struct PsShared {
  PsChunk ch[kPsChunks];
  int first[2 * 16];            // chunks of phase p: ch[first[p]] .. ch[first[p + 1]]
  double ws[kPsWarps];
};

// Shared memory: PsShared | staged planes (3 vec) | partial products | the
// local step's exchange | tables | tape (adjoint) | rows.
__host__ __device__ inline size_t ps_fixed_doubles(int vec) {
  return (sizeof(PsShared) + 15) / 16 * 2 + 3 * (size_t)vec + 3 * kBsRows + kPsXch * kPsPair;
}

// The CTA's chunks, index tables and rows (once per launch).
template <class BAR>
__device__ __forceinline__ void ps_setup(const BlockDev& b, PsShared& S, int* tab, int tab_ints, double* res,
                                         int res_doubles) {
  const int phases = 2 * b.tiers - 1, tid = threadIdx.x;
  int nc = 0, ti = 0, rd = 0;
  for (int p = 0; p < phases; ++p) {
    const bool fwd = p < b.tiers;
    const int* share = b.share + (size_t)p * (b.G + 1) + BAR::cta();
    if (tid == 0) S.first[p] = nc;
    for (int k = share[0]; k < share[1]; ++k, ++nc) {
      const BlockChunk C = b.chunks[k];
      const BlockInfo B = b.blk[C.blk];
      PsChunk P;
      P.n = B.n; P.r = B.r; P.ld = fwd ? B.ldx : B.ldr; P.tier = B.tier;
      P.row0 = C.row0; P.rows = C.rows; P.cofs = B.cofs; P.rofs = B.rofs;
      const int w = fwd ? B.n : B.r, size = C.rows * P.ld;
      const double* src = b.sol + (fwd ? B.xp : B.pt) + (size_t)C.row0 * P.ld;
      if (rd + size <= res_doubles) {
        const double2* s2 = reinterpret_cast<const double2*>(src);
        double2* d2 = reinterpret_cast<double2*>(res + rd);
        for (int q = tid; q < size / 2; q += blockDim.x) d2[q] = __ldcg(s2 + q);
        P.mat = res + rd;
        rd += size;
      } else {
        P.mat = src;
      }
      const int* gi = fwd ? b.cols + B.cofs : b.rows + B.rofs;
      const bool ptr = fwd && B.tier > 0;
      const int need = (ptr ? 3 : 1) * w + C.rows;
      P.out = nullptr;
      if (ti + need <= tab_ints) {
        int* o = tab + ti;
        for (int q = tid; q < w; q += blockDim.x) {
          const int g = gi[q];
          o[q] = g;
          if (ptr) { o[w + q] = b.vptr[g]; o[2 * w + q] = b.vptr[g + 1]; }
        }
        P.idx = o;
        P.v0 = ptr ? o + w : nullptr;
        P.v1 = ptr ? o + 2 * w : nullptr;
        o += (ptr ? 3 : 1) * w;
        for (int q = tid; q < C.rows; q += blockDim.x) {
          const int row = C.row0 + q;
          o[q] = row < B.n ? b.cols[B.cofs + row] : -1 - b.cslot[B.rofs + row - B.n];
        }
        P.out = o;
        ti += need;
      } else {
        P.idx = gi;
        P.v0 = P.v1 = nullptr;  // read through the vertex
      }
      if (tid == 0) S.ch[nc] = P;
    }
  }
  if (tid == 0) S.first[phases] = nc;
  __syncthreads();
}

// R rows (2 or 4; ld apart, the last `valid` - 1 repeated) of a chunk times
// the staged planes, columns [2 q0, 2 q1): each staged value serves R
// products.  The warp's sums are folded R values at a time, so that lane group
// lane / (32 / R) ends with its row's three.
template <int R>
__device__ __forceinline__ void ps_rows(const double* mat, int ld, int valid, const double2* bx, const double2* by,
                                        const double2* bz, int q0, int q1, double o[3]) {
  const int lane = threadIdx.x & 31;
  const double2* row[R];
#pragma unroll
  for (int r = 0; r < R; ++r) row[r] = reinterpret_cast<const double2*>(mat + (size_t)min(r, valid - 1) * ld);
  double a[R][3];
#pragma unroll
  for (int r = 0; r < R; ++r) a[r][0] = a[r][1] = a[r][2] = 0.0;
#pragma unroll 2
  for (int q = q0 + lane; q < q1; q += 32) {
    double2 u[R];
#pragma unroll
    for (int r = 0; r < R; ++r) u[r] = row[r][q];
    const double2 x = bx[q], y = by[q], z = bz[q];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      a[r][0] = fma(u[r].y, x.y, fma(u[r].x, x.x, a[r][0]));
      a[r][1] = fma(u[r].y, y.y, fma(u[r].x, y.x, a[r][1]));
      a[r][2] = fma(u[r].y, z.y, fma(u[r].x, z.x, a[r][2]));
    }
  }
  double v[R / 2][3];
  const bool h16 = lane & 16;
#pragma unroll
  for (int r = 0; r < R / 2; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double keep = h16 ? a[r + R / 2][c] : a[r][c], send = h16 ? a[r][c] : a[r + R / 2][c];
      v[r][c] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
  if (R == 4) {
    const bool h8 = lane & 8;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double keep = h8 ? v[R / 2 - 1][c] : v[0][c], send = h8 ? v[0][c] : v[R / 2 - 1][c];
      v[0][c] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
  }
#pragma unroll
  for (int s = R == 4 ? 4 : 8; s > 0; s >>= 1)
#pragma unroll
    for (int c = 0; c < 3; ++c) v[0][c] += __shfl_xor_sync(0xffffffffu, v[0][c], s);
#pragma unroll
  for (int c = 0; c < 3; ++c) o[c] = v[0][c];
}

// block_solve with the CTA's tables and rows in shared memory.  pre(v) loads
// what done(v, value, loaded) needs before the products, so that its latency
// is hidden.
template <class BAR, class PRE, class DONE>
__device__ __forceinline__ bool ps_solve(const BlockDev& b, BAR& bar, const PsShared& S, const double* rhs, double* y,
                                         double* planes, PRE pre, DONE done) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* sx = planes;
  double* sy = sx + b.vec;
  double* sz = sy + b.vec;
  double* part = sz + b.vec;
  const int phases = 2 * b.tiers - 1;
  for (int p = 0; p < phases; ++p) {
    const bool fwd = p < b.tiers, fin = !fwd || p == b.tiers - 1;
    for (int k = S.first[p]; k < S.first[p + 1]; ++k) {
      const PsChunk& C = S.ch[k];
      const int w = fwd ? C.n : C.r, ld = C.ld, w2 = ld / 2;
      __syncthreads();  // the planes' and partials' readers of the chunk before
      for (int i = tid; i < ld; i += kPsThreads) {
        Vec3<double> v = mk3(0.0, 0.0, 0.0);
        if (i < w) {
          const int g = C.idx[i];
          if (fwd) {
            v = ld3(rhs, g);
            if (C.tier > 0) {
              const int e = C.v0 ? C.v1[i] : b.vptr[g + 1];
              for (int q = C.v0 ? C.v0[i] : b.vptr[g]; q < e; q += 8) {  // eight in flight, subtracted in order
                Vec3<double> c[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) c[u] = q + u < e ? ld3(b.contrib, q + u) : mk3(0.0, 0.0, 0.0);
#pragma unroll
                for (int u = 0; u < 8; ++u) v = v - c[u];
              }
            }
          } else {
            v = ld3(y, g);
          }
        }
        sx[i] = v.x; sy[i] = v.y; sz[i] = v.z;
      }
      for (int base = 0; base < C.rows; base += kBsRows) {
        const int nr = min(kBsRows, C.rows - base);
        int out = 0;
        Vec3<double> yo = mk3(0.0, 0.0, 0.0);
        decltype(pre(0)) pl;
        if (tid < nr) {
          const int row = C.row0 + base + tid;
          out = C.out ? C.out[base + tid] : row < C.n ? b.cols[C.cofs + row] : -1 - b.cslot[C.rofs + row - C.n];
          if (out >= 0 && fin) {
            if (!fwd) yo = ld3(y, out);
            pl = pre(out);
          }
        }
        __syncthreads();
        const int R = nr > 2 ? 4 : 2, groups = nr > 2 ? (nr + 3) >> 2 : 1;
        int ls = 0;  // log2 of the column segments: up to one per warp and no shorter than 32 pairs of columns
        while ((2 << ls) * groups <= kPsWarps && (64 << ls) <= w2) ++ls;
        const int seg = 1 << ls, len = (w2 + seg - 1) >> ls;
        const double2* bx = reinterpret_cast<const double2*>(sx);
        const double2* by = reinterpret_cast<const double2*>(sy);
        const double2* bz = reinterpret_cast<const double2*>(sz);
        for (int u = warp; u < groups * seg; u += kPsWarps) {
          const int gr = u >> ls, sg = u & (seg - 1), q0 = sg * len, q1 = min(w2, q0 + len);
          const double* m = C.mat + (size_t)(base + gr * R) * ld;
          double o[3];
          if (R == 4) ps_rows<4>(m, ld, nr - 4 * gr, bx, by, bz, q0, q1, o);
          else ps_rows<2>(m, ld, nr - 2 * gr, bx, by, bz, q0, q1, o);
          const int r = gr * R + lane / (32 / R);
          if (lane % (32 / R) == 0 && r < nr) st3(part, r * seg + sg, mk3(o[0], o[1], o[2]));
        }
        __syncthreads();
        if (tid < nr) {
          Vec3<double> v = ld3(part, tid * seg);
          for (int sg = 1; sg < seg; ++sg) v = v + ld3(part, tid * seg + sg);
          if (out < 0) st3(b.contrib, -1 - out, v);
          else if (fin) done(out, fwd ? v : yo - v, pl);
          else st3(y, out, v);
        }
      }
    }
    if (p + 1 < phases && !bar.sync()) return false;
  }
  return true;
}

// The mixed form's solve: rows cta, cta + nc, ... of X times rhs, every row
// summed as in k_dense_solve (the same lanes, order and operations: the mixed
// form's results follow the solve's last bits).  A warp takes one row, or two
// side by side where the CTA has more rows than warps (each staged value then
// serves both).  res: the CTA's first nres rows in shared memory.
template <class DONE>
__device__ __forceinline__ void ps_dense_rows(const double* X, int Np, const double* res, int nres, int N, int cta, int nc,
                                              const double* rhs, double* planes, DONE done) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, np2 = Np / 2;
  double* sx = planes;
  double* sy = sx + Np;
  double* sz = sy + Np;
  for (int j = tid; j < Np; j += kPsThreads) {
    const Vec3<double> v = j < N ? ld3(rhs, j) : mk3(0.0, 0.0, 0.0);
    sx[j] = v.x; sy[j] = v.y; sz[j] = v.z;
  }
  __syncthreads();
  const double2* bx = reinterpret_cast<const double2*>(sx);
  const double2* by = reinterpret_cast<const double2*>(sy);
  const double2* bz = reinterpret_cast<const double2*>(sz);
  const int rows = (N - cta + nc - 1) / nc;
  auto run = [&](auto two, int r0, int r1) {
    constexpr bool kTwo = decltype(two)::value;
    const double2* m0 = reinterpret_cast<const double2*>(r0 < nres ? res + (size_t)r0 * Np : X + (size_t)(cta + r0 * nc) * Np);
    const double2* m1 = reinterpret_cast<const double2*>(r1 < nres ? res + (size_t)r1 * Np : X + (size_t)(cta + r1 * nc) * Np);
    double a[2][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
    for (int q0 = lane; q0 < np2; q0 += 256) {
      double2 u[8], w[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int q = q0 + 32 * k;
        u[k] = q < np2 ? m0[q] : make_double2(0.0, 0.0);
        if (kTwo) w[k] = q < np2 ? m1[q] : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int q = q0 + 32 * k;
        if (q < np2) {
          const double2 x = bx[q], y = by[q], z = bz[q];
          a[0][0] = __dadd_rn(a[0][0], __fma_rn(u[k].x, x.x, __dmul_rn(u[k].y, x.y)));
          a[0][1] = __dadd_rn(a[0][1], __fma_rn(u[k].y, y.y, __dmul_rn(u[k].x, y.x)));
          a[0][2] = __dadd_rn(a[0][2], __fma_rn(u[k].x, z.x, __dmul_rn(u[k].y, z.y)));
          if (kTwo) {
            a[1][0] = __dadd_rn(a[1][0], __fma_rn(w[k].x, x.x, __dmul_rn(w[k].y, x.y)));
            a[1][1] = __dadd_rn(a[1][1], __fma_rn(w[k].y, y.y, __dmul_rn(w[k].x, y.x)));
            a[1][2] = __dadd_rn(a[1][2], __fma_rn(w[k].x, z.x, __dmul_rn(w[k].y, z.y)));
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < (kTwo ? 2 : 1); ++r) {
#pragma unroll
      for (int c = 0; c < 3; ++c) a[r][c] = warp_sum(a[r][c]);
      if (lane == 0) done(cta + (r == 0 ? r0 : r1) * nc, mk3(a[r][0], a[r][1], a[r][2]));
    }
  };
  int r = warp;
  for (; r + kPsWarps < rows; r += 2 * kPsWarps) run(std::true_type{}, r, r + kPsWarps);
  if (r < rows) run(std::false_type{}, r, r);
}

// Local step of all constraints by a CTA's sixteen warps.  A tet is given to
// two threads, eight warps apart: one takes its rotation, the other its
// volume projection (the two iterations do not depend on one another and are
// the chain of dependent FP64 operations that bounds a scene with less than a
// warp per scheduler); the rotation passes through shared memory.
__device__ __forceinline__ void ps_give(double* xch, bool rot, int me, const Vec3<double> P[3]) {
  double* o = xch + (rot ? 0 : 9) * kPsPair + me;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    o[(3 * j) * kPsPair] = P[j].x;
    o[(3 * j + 1) * kPsPair] = P[j].y;
    o[(3 * j + 2) * kPsPair] = P[j].z;
  }
}
// P += the other half's (a sum of two: the same bits in both)
__device__ __forceinline__ void ps_take(const double* xch, bool rot, int me, Vec3<double> P[3]) {
  const double* o = xch + (rot ? 9 : 0) * kPsPair + me;
#pragma unroll
  for (int j = 0; j < 3; ++j)
    P[j] = rn_add(P[j], mk3(o[(3 * j) * kPsPair], o[(3 * j + 1) * kPsPair], o[(3 * j + 2) * kPsPair]));
}
// corners 0, 1 (rotation's thread) or 2, 3 of G P into their slots
__device__ __forceinline__ void ps_corners(const double G[4][3], const Vec3<double> P[3], int4 sl, bool rot, double* slot) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const double g0 = rot ? G[q][0] : G[q + 2][0], g1 = rot ? G[q][1] : G[q + 2][1], g2 = rot ? G[q][2] : G[q + 2][2];
    const int o = rot ? (q == 0 ? sl.x : sl.y) : (q == 0 ? sl.z : sl.w);
    st3(slot, o, rn_comb(g0, P[0], g1, P[1], g2, P[2]));
  }
}

template <class BAR>
__device__ __forceinline__ void ps_local(const SceneDev& d, const double* x, const double* act_row, double* slot,
                                         double* xch, int4 tv0, int first, int stride) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nc = BAR::ctas();
  const int me = tid & (kPsPair - 1);
  const bool rot = warp < kPsWarps / 2;
  for (int base = 0; base < d.T; base += kPsPair * nc) {
    const int t = base + 32 * ((warp & (kPsWarps / 2 - 1)) * nc + BAR::cta()) + lane;
    double G[4][3];
    Vec3<double> P[3];  // this half's part of wr md + wv md_volume
    int4 sl;
    if (t < d.T) {
      sl = d.tslot[t];
      const int4 v = base == 0 ? tv0 : d.tv[t];
      const Vec3<double> xv[4] = {ld3(x, v.x), ld3(x, v.y), ld3(x, v.z), ld3(x, v.w)};
      load_g(d.tinv, d.T, t, G);
      const double w = rot ? d.twr[t] : d.twv[t];
      const Mat3<double> F = deformation(G, xv);
      Mat3<double> m;
      if (rot) corot_rotation(F, m);
      else corot_volume(F, m);
#pragma unroll
      for (int j = 0; j < 3; ++j) P[j] = rn_scale(w, m.c[j]);
      ps_give(xch, rot, me, P);
    }
    __syncthreads();
    if (t < d.T) {  // two corners each
      ps_take(xch, rot, me, P);
      ps_corners(G, P, sl, rot, slot);
    }
    if (base + kPsPair * nc < d.T) __syncthreads();
  }
  for (int t = first; t < d.M + d.S + d.B; t += stride) local_rest(d, t, x, act_row, slot);
}

// Its VJP (with the Hs term of the next iterate x1), split the same way; the
// volume half's tape takes the threads of tape_warps warps.
template <class BAR>
__device__ __forceinline__ void ps_adj_local(const SceneDev& d, const double* x, const double* x1, const double* y,
                                             const double* act_row, double* slot, double* gE, double* gnu, double* mg,
                                             bool first_it, double* xch, double* tape, int tape_warps, int4 tv0, int first,
                                             int stride) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nc = BAR::ctas();
  const int me = tid & (kPsPair - 1), half = warp & (kPsWarps / 2 - 1);
  const bool rot = warp < kPsWarps / 2;
  for (int base = 0; base < d.T; base += 32 * tape_warps * nc) {
    const int t = half < tape_warps ? base + 32 * (half * nc + BAR::cta()) + lane : d.T;
    double G[4][3], yv = 0.0;
    Mat3<double> gF;
    int4 sl;
    if (t < d.T) {
      sl = d.tslot[t];
      const int4 v = base == 0 ? tv0 : d.tv[t];
      const int vi[4] = {v.x, v.y, v.z, v.w};
      Vec3<double> xv[4], yw[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) { xv[a] = ld3(x, vi[a]); yw[a] = ld3(y, vi[a]); }
      load_g(d.tinv, d.T, t, G);
      const Mat3<double> F = deformation(G, xv), Y = deformation(G, yw);
      if (rot) {
        double yr;
        corot_adjoint_rotation(F, Y, d.twr[t], yr, gF);
#pragma unroll
        for (int a = 0; a < 4; ++a) xv[a] = ld3(x1, vi[a]);
        xch[18 * kPsPair + me] = yr;
        xch[19 * kPsPair + me] = iterate_yh(G, Y, xv);
      } else {
        corot_adjoint_volume(F, Y, d.twv[t], yv, gF, tape + 32 * half + lane, 32 * tape_warps);
      }
      ps_give(xch, rot, me, gF.c);
    }
    __syncthreads();
    if (t < d.T) {
      ps_take(xch, rot, me, gF.c);
      ps_corners(G, gF.c, sl, rot, slot);
      if (!rot) {
        tet_moduli_grad(gE, gnu, t, d.tE[t], d.tnu[t], d.tvol[t], xch[18 * kPsPair + me], yv, xch[19 * kPsPair + me]);
      }
    }
    if (base + 32 * tape_warps * nc < d.T) __syncthreads();
  }
  const int nmg = d.M + (d.sch ? d.S : 0);
  for (int t = first; t < d.M + d.S + d.B; t += stride) {
    adj_local_rest(d, t, x, y, act_row, slot, mg);
    // activation terms: summed over the step's iterations by their constraint's thread
    if (t < nmg && (t < d.M || d.sch[t - d.M] >= 0)) mg[nmg + t] = first_it ? mg[t] : mg[nmg + t] + mg[t];
  }
}

// Sum of v over the grid: the CTA's part goes to partial; after the next
// barrier ps_total gives every warp of every CTA the same sum (two sets of
// partials, used in turn: a CTA is never two sums ahead of another).
__device__ __forceinline__ void ps_put(double v, double* ws, double* partial) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0;
#pragma unroll
    for (int w = 0; w < kPsWarps; ++w) s += ws[w];
    *partial = s;
  }
}
__device__ __forceinline__ double ps_total(const double* partial, int n) {
  double s = 0;
  for (int k = threadIdx.x & 31; k < n; k += 256) {  // eight loads in flight
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = k + 32 * u < n ? __ldcg(partial + k + 32 * u) : 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u) s += v[u];
  }
  return warp_sum(s);
}

// Sum of a vertex's slots by eight lanes (lane l adds slots l, l + 8, ..., then a fixed tree).
__device__ __forceinline__ Vec3<double> ps_sum_slots(const double* slot, int k0, int k1) {
  Vec3<double> a = mk3(0.0, 0.0, 0.0);
  for (int k = k0 + (int)(threadIdx.x & 7); k < k1; k += 32) {  // four loads in flight
    Vec3<double> v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const size_t q = 3 * (size_t)(k + 8 * u);
      v[u] = k + 8 * u < k1 ? mk3(slot[q], slot[q + 1], slot[q + 2]) : mk3(0.0, 0.0, 0.0);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) a = a + v[u];
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
    a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
    a.z += __shfl_xor_sync(0xffffffffu, a.z, o);
  }
  return a;
}

template <class BAR, bool MIXED>
__global__ void __launch_bounds__(kPsThreads, 1) k_pd_forward(const __grid_constant__ SceneDev d, BlockDev b, PdSteps a) {
  extern __shared__ __align__(16) double pssh[];
  PsShared& S = *reinterpret_cast<PsShared*>(pssh);
  double* planes = pssh + (sizeof(PsShared) + 15) / 16 * 2;
  // plain form: ps_fixed_doubles, tables, rows; mixed form: three planes of N_p, rows of X
  const int vec = MIXED ? a.Np : b.vec;
  int* tab = reinterpret_cast<int*>(pssh + ps_fixed_doubles(vec));
  double* res = pssh + ps_fixed_doubles(vec) + (MIXED ? 0 : a.tab_ints / 2);
  double* xch = planes + 3 * (size_t)vec + 3 * kBsRows;
  if (MIXED) res = xch;  // the mixed form exchanges nothing
  if (BAR::gave_up(b.status)) return;
  BAR bar(b.bar, b.status, b.spin_tries);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cta = BAR::cta(), nc = BAR::ctas();
  // items are dealt to the CTAs a warp's worth at a time
  const int first = 32 * (warp * nc + cta) + lane, stride = kPsThreads * nc;
  const bool lead = cta == 0 && tid == 0;
  const int s0 = a.step ? *a.step : a.s0;
  const int ncons = d.T + d.M + d.S + d.B;
  if (lead && a.zero)
    for (int q = 0; q < 4; ++q) a.status[q] = 0;
  // mixed form: the first of the CTA's rows cta, cta + nc, ... of X stay in shared memory
  const int xres = MIXED ? min((d.N - cta + nc - 1) / nc, a.res_doubles / a.Np) : 0;
  if (MIXED) {
    {
      for (int q = tid; q < xres * (a.Np / 2); q += kPsThreads) {
        const int r = q / (a.Np / 2), c = q % (a.Np / 2);
        reinterpret_cast<double2*>(res)[q] = __ldcg(reinterpret_cast<const double2*>(a.X + (size_t)(cta + r * nc) * a.Np) + c);
      }
    }
    __syncthreads();
  } else {
    ps_setup<BAR>(b, S, tab, a.tab_ints, res, a.res_doubles);
  }
  if (a.x_in) {
    for (int i = first; i < d.N; i += stride) {
      const int u = a.to_user[i];
      st3(a.xt, i, ld3(a.x_in, u));
      st3(a.vt, i, ld3(a.v_in, u));
    }
    if (!bar.sync()) return;
  }
  // this thread's first tet and vertex: their tables are read once, so that the first loads after a barrier are
  // the ones that wait for it
  const int t0 = 32 * ((warp & (kPsWarps / 2 - 1)) * nc + cta) + lane, g0 = min(first >> 3, d.N - 1);
  const int4 tv0 = t0 < d.T ? d.tv[t0] : make_int4(0, 0, 0, 0);
  const int vs0 = d.vslot_ptr[g0], vs1 = d.vslot_ptr[g0 + 1];
  int par = 0;
  double* xprev = a.xt;  // positions the step starts from, as every CTA reads them
  double* xk = a.xk;
  double* xo = a.xk2;
  for (int st = 0; st < a.n; ++st) {
    const int s = s0 + st;
    double* hist = a.hist + (size_t)s * a.hist_step;
    // begin (after the end of the step before): v_wc, q_n, x^0 = q_n, c0 = M/h^2 q_n - Hs x + J_att d_att
    double q2 = 0.0;
    for (int g = first >> 3; g < ((d.N + 3) & ~3); g += stride >> 3) {  // eight lanes per vertex: its row of Hs
      const int i = min(g, d.N - 1);
      Vec3<double> acc = mk3(0.0, 0.0, 0.0);
      if (!MIXED) {
        const int k1 = d.hs_ptr[i + 1];
        for (int k = d.hs_ptr[i] + (lane & 7); k < k1; k += 8) acc = acc + d.hs_val[k] * ld3(xprev, d.hs_col[k]);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
          acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
          acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
          acc.z += __shfl_xor_sync(0xffffffffu, acc.z, o);
        }
      }
      if ((lane & 7) != 0 || g >= d.N) continue;
      Vec3<double> x, v;
      if (st > 0) {
        x = ld3(xprev, i);
        v = (d.damping / d.h) * (x - ld3(a.xt, i));
        if (a.traj) st3(a.traj + (size_t)(s - 1) * 3 * d.N, a.to_user[i], x);
        st3(a.xt, i, x);
      } else {
        x = ld3(a.xt, i);
        v = ld3(a.vt, i);
      }
      if (a.ckpt_x && s % a.ckpt_every == 0) {
        const size_t o = (size_t)(s / a.ckpt_every) * 3 * d.N;
        st3(a.ckpt_x + o, i, x);
        st3(a.ckpt_v + o, i, v);
      }
      const Vec3<double> vwc = step_vwc(d, i, v);
      if (a.vwc) st3(a.vwc, i, vwc);
      const Vec3<double> q = x + d.h * vwc;
      st3(a.qn, i, q);
      st3(xk, i, q);
      st3(hist, i, q);
      if (!MIXED) st3(a.c0, i, (d.mass[i] / (d.h * d.h)) * q - acc + ld3(d.attach_jd, i));
      q2 += dot3(q, q);
    }
    ps_put(q2, S.ws, a.partial + par * nc + cta);
    if (!bar.sync()) return;
    double tot = ps_total(a.partial + par * nc, nc);
    par ^= 1;
    // iteration 0 of the reference compares q_n with a zero vector
    bool conv = sqrt(tot) / (3.0 * d.N) < kConvergenceEps;
    if (lead && !isfinite(tot)) a.status[0] = 4;
    const double* act_row = a.act_all + (size_t)s * d.nseg;
    int k = 0;
    for (; k < a.K && !conv; ++k) {
      if (MIXED)
        for (int t = first; t < ncons; t += stride) force_item(d, t, xk, act_row, reinterpret_cast<float*>(a.slot));
      else
        ps_local<BAR>(d, xk, act_row, a.slot, xch, tv0, first, stride);
      if (!bar.sync()) return;
      if (MIXED) {
        for (int i = first; i < d.N; i += stride) st3(a.rhs, i, force_rhs(d, i, reinterpret_cast<float*>(a.slot), a.qn, xk));
      } else {
        for (int g = first >> 3; g < ((d.N + 3) & ~3); g += stride >> 3) {  // eight lanes per vertex
          const int i = min(g, d.N - 1);
          const Vec3<double> c = ld3(a.c0, i);
          const Vec3<double> f = ps_sum_slots(a.slot, i == g0 ? vs0 : d.vslot_ptr[i], i == g0 ? vs1 : d.vslot_ptr[i + 1]);
          if ((lane & 7) == 0 && g < d.N) st3(a.rhs, i, c + f);
        }
      }
      if (!bar.sync()) return;
      double e2 = 0.0;
      double* h1 = hist + (size_t)(k + 1) * 3 * d.N;
      if (MIXED) {  // x^{k+1} = x^k + z
        ps_dense_rows(a.X, a.Np, res, xres, d.N, cta, nc, a.rhs, planes, [&](int g, Vec3<double> z) {
          const Vec3<double> xc = ld3(xk, g), xn = xc + z, dl = xn - xc;
          e2 += dot3(dl, dl);
          st3(xk, g, xn);
          st3(h1, g, xn);
        });
      } else {  // x^{k+1} = x_t + z (the reference's delta form)
        struct Pos { Vec3<double> xc, x0; };
        const bool ok = ps_solve(
            b, bar, S, a.rhs, a.y, planes, [&](int g) { return Pos{ld3(xk, g), ld3(a.xt, g)}; },
            [&](int g, Vec3<double> z, const Pos& p) {
              const Vec3<double> xn = p.x0 + z, dl = xn - p.xc;
              e2 += dot3(dl, dl);
              st3(xk, g, xn);
              st3(h1, g, xn);
              if (b.tiers > 1) st3(a.y, g, z);  // read by the blocks below
            });
        if (!ok) return;
      }
      ps_put(e2, S.ws, a.partial + par * nc + cta);
      if (!bar.sync()) return;
      tot = ps_total(a.partial + par * nc, nc);
      par ^= 1;
      conv = sqrt(tot) / (3.0 * d.N) < kConvergenceEps;
      if (!isfinite(tot)) {
        if (lead) a.status[0] = 4;
        conv = true;
      }
    }
    if (lead) a.iters[s] = k;
    xprev = xk;
    double* t = xk;
    xk = xo;
    xo = t;
  }
  if (a.end) {
    for (int i = first; i < d.N; i += stride) {
      const Vec3<double> x = ld3(xprev, i), v = (d.damping / d.h) * (x - ld3(a.xt, i));
      const int u = a.to_user[i];
      if (a.traj) st3(a.traj + (size_t)(s0 + a.n - 1) * 3 * d.N, u, x);
      st3(a.xt, i, x);
      st3(a.vt, i, v);
      if (a.x_out) {
        st3(a.x_out, u, x);
        st3(a.v_out, u, v);
      }
    }
  }
  bar.leave();
}

template <class BAR>
__global__ void __launch_bounds__(kPsThreads, 1) k_pd_adjoint(SceneDev d, BlockDev b, PdSteps a) {
  extern __shared__ __align__(16) double pssh[];
  PsShared& S = *reinterpret_cast<PsShared*>(pssh);
  double* planes = pssh + (sizeof(PsShared) + 15) / 16 * 2;
  int* tab = reinterpret_cast<int*>(pssh + ps_fixed_doubles(b.vec));
  double* tape = pssh + ps_fixed_doubles(b.vec) + a.tab_ints / 2;
  const int tstride = 32 * a.tape_warps;
  double* res = tape + (size_t)kVolTape * tstride;
  double* xch = planes + 3 * (size_t)b.vec + 3 * kBsRows;
  if (BAR::gave_up(b.status)) return;
  BAR bar(b.bar, b.status, b.spin_tries);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cta = BAR::cta(), nc = BAR::ctas();
  const int first = 32 * (warp * nc + cta) + lane, stride = kPsThreads * nc;
  const int nmg = d.M + (d.sch ? d.S : 0);
  ps_setup<BAR>(b, S, tab, a.tab_ints, res, a.res_doubles);
  if (a.zero) {
    if (cta == 0 && tid < 4) a.status[tid] = 0;
    for (int t = first; t < d.T; t += stride) { a.gE[t] = 0.0; a.gnu[t] = 0.0; }
    for (int q = first; q < a.n * d.nseg; q += stride) a.gact[(size_t)a.s0 * d.nseg + q] = 0.0;
  }
  const int t0 = 32 * ((warp & (kPsWarps / 2 - 1)) * nc + cta) + lane, g0 = min(first >> 3, d.N - 1);
  const int4 tv0 = (warp & (kPsWarps / 2 - 1)) < a.tape_warps && t0 < d.T ? d.tv[t0] : make_int4(0, 0, 0, 0);
  const int vs0 = d.vslot_ptr[g0], vs1 = d.vslot_ptr[g0 + 1];
  const double c = d.damping / d.h, ih2 = 1.0 / (d.h * d.h);
  for (int st = a.n - 1; st >= 0; --st) {
    const int s = a.s0 + st;
    const double* hist = a.hist + (size_t)s * a.hist_step;
    // the cotangents of the step's output: given, or those of the step after it
    for (int i = first; i < d.N; i += stride) {
      Vec3<double> gx, gv;
      if (st < a.n - 1) {
        const Vec3<double> qb = ld3(a.xkb, i) + (d.mass[i] * ih2) * ld3(a.bb, i);
        gx = ld3(a.xtb, i) + qb;
        gv = d.h * qb;
      } else if (a.x_in) {
        const int u = a.to_user[i];
        gx = ld3(a.x_in, u);
        gv = ld3(a.v_in, u);
      } else {
        gx = ld3(a.io_a, i);
        gv = ld3(a.io_b, i);
      }
      st3(a.xkb, i, gx + c * gv);
      st3(a.xtb, i, (-c) * gv);
      st3(a.bb, i, mk3(0.0, 0.0, 0.0));
    }
    const int nit = min(max(a.iters[s], 0), a.K);
    const double* act_row = a.act_all + (size_t)s * d.nseg;
    if (!bar.sync()) return;
    for (int k = nit - 1; k >= 0; --k) {
      const bool ok = ps_solve(
          b, bar, S, a.xkb, a.y, planes, [&](int g) { return ld3(a.bb, g); },
          [&](int g, Vec3<double> y, const Vec3<double>& bb) {
            st3(a.y, g, y);
            st3(a.bb, g, bb + y);
          });
      if (!ok || !bar.sync()) return;
      const double* x = hist + (size_t)k * 3 * d.N;
      const double* x1 = x + 3 * (size_t)d.N;
      ps_adj_local<BAR>(d, x, x1, a.y, act_row, a.slot, a.gE, a.gnu, a.mg, k == nit - 1, xch, tape, a.tape_warps, tv0,
                        first, stride);
      if (!bar.sync()) return;
      for (int g = first >> 3; g < ((d.N + 3) & ~3); g += stride >> 3) {
        const int i = min(g, d.N - 1);
        const Vec3<double> f = ps_sum_slots(a.slot, i == g0 ? vs0 : d.vslot_ptr[i], i == g0 ? vs1 : d.vslot_ptr[i + 1]);
        if ((lane & 7) == 0 && g < d.N) st3(a.xkb, i, f);
      }
      if (k == 0)  // the activation gradient of the step
        for (int q = first; q < d.nseg; q += stride) {
          double g = 0;
          for (int m = d.seg_ptr[q]; m < d.seg_ptr[q + 1]; ++m) g += a.mg[nmg + member_slot(d.M, d.seg_mus[m])];
          a.gact[(size_t)s * d.nseg + q] += g;
        }
      if (!bar.sync()) return;
    }
  }
  for (int i = first; i < d.N; i += stride) {
    const Vec3<double> qb = ld3(a.xkb, i) + (d.mass[i] * ih2) * ld3(a.bb, i);
    const Vec3<double> gx = ld3(a.xtb, i) + qb, gv = d.h * qb;
    if (a.x_out) {
      const int u = a.to_user[i];
      st3(a.x_out, u, gx);
      st3(a.v_out, u, gv);
    } else {
      st3(a.io_a, i, gx);
      st3(a.io_b, i, gv);
    }
  }
  // the accumulators, last written before the last barrier
  if (a.gE_out)
    for (int t = first; t < d.T; t += stride) a.gE_out[t] = a.gE[t];
  if (a.gnu_out)
    for (int t = first; t < d.T; t += stride) a.gnu_out[t] = a.gnu[t];
  if (a.gact_out)
    for (int q = first; q < a.n * d.nseg; q += stride) a.gact_out[q] = a.gact[(size_t)a.s0 * d.nseg + q];
  bar.leave();
}

}  // namespace dfem
