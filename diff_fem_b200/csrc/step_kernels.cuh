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

namespace dfem {

constexpr int kPsThreads = 512;
constexpr int kPsWarps = kPsThreads / 32;
constexpr int kPsChunks = 40;   // row ranges of a CTA over all phases of the solve

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
};

struct PsShared {
  PsChunk ch[kPsChunks];
  int first[2 * 16];            // chunks of phase p: ch[first[p]] .. ch[first[p + 1]]
  double ws[kPsWarps];
};

// Shared memory: PsShared | staged planes (3 vec) | partial products | tables
// | rows | tape (adjoint).
__host__ __device__ inline size_t ps_fixed_doubles(int vec) {
  return (sizeof(PsShared) + 15) / 16 * 2 + 3 * (size_t)vec + 3 * kBsRows;
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
      if (ti + (ptr ? 3 : 1) * w <= tab_ints) {
        int* o = tab + ti;
        for (int q = tid; q < w; q += blockDim.x) {
          const int g = gi[q];
          o[q] = g;
          if (ptr) { o[w + q] = b.vptr[g]; o[2 * w + q] = b.vptr[g + 1]; }
        }
        P.idx = o;
        P.v0 = ptr ? o + w : nullptr;
        P.v1 = ptr ? o + 2 * w : nullptr;
        ti += (ptr ? 3 : 1) * w;
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

// Two rows of a chunk times the staged planes, columns [2 q0, 2 q1).
__device__ __forceinline__ void ps_row_pair(const double2* r0, const double2* r1, const double2* bx, const double2* by,
                                            const double2* bz, int q0, int q1, double o[2][3]) {
  const int lane = threadIdx.x & 31;
  double a[2][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
  int q = q0 + lane;
  for (; q + 96 < q1; q += 128) {
    double2 u[4], w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) { u[k] = r0[q + 32 * k]; w[k] = r1[q + 32 * k]; }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double2 x = bx[q + 32 * k], y = by[q + 32 * k], z = bz[q + 32 * k];
      a[0][0] += u[k].x * x.x + u[k].y * x.y;
      a[0][1] += u[k].x * y.x + u[k].y * y.y;
      a[0][2] += u[k].x * z.x + u[k].y * z.y;
      a[1][0] += w[k].x * x.x + w[k].y * x.y;
      a[1][1] += w[k].x * y.x + w[k].y * y.y;
      a[1][2] += w[k].x * z.x + w[k].y * z.y;
    }
  }
  for (; q < q1; q += 32) {
    const double2 u = r0[q], w = r1[q], x = bx[q], y = by[q], z = bz[q];
    a[0][0] += u.x * x.x + u.y * x.y;
    a[0][1] += u.x * y.x + u.y * y.y;
    a[0][2] += u.x * z.x + u.y * z.y;
    a[1][0] += w.x * x.x + w.y * x.y;
    a[1][1] += w.x * y.x + w.y * y.y;
    a[1][2] += w.x * z.x + w.y * z.y;
  }
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) o[r][c] = warp_sum(a[r][c]);
}

// block_solve with the CTA's tables and rows in shared memory.
template <class BAR, class DONE>
__device__ __forceinline__ bool ps_solve(const BlockDev& b, BAR& bar, const PsShared& S, const double* rhs, double* y,
                                         double* planes, DONE done) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* sx = planes;
  double* sy = sx + b.vec;
  double* sz = sy + b.vec;
  double* part = sz + b.vec;
  const int phases = 2 * b.tiers - 1;
  for (int p = 0; p < phases; ++p) {
    const bool fwd = p < b.tiers;
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
              for (int q = C.v0 ? C.v0[i] : b.vptr[g]; q < e; ++q) v = v - ld3(b.contrib, q);
            }
          } else {
            v = ld3(y, g);
          }
        }
        sx[i] = v.x; sy[i] = v.y; sz[i] = v.z;
      }
      __syncthreads();
      for (int base = 0; base < C.rows; base += kBsRows) {
        const int nr = min(kBsRows, C.rows - base), pairs = (nr + 1) / 2;
        int seg = 1;  // column segments: power of two, up to one per warp and no shorter than 32 pairs of columns
        while (2 * seg * pairs <= kPsWarps && 64 * seg <= w2) seg *= 2;
        const int len = (w2 + seg - 1) / seg;
        if (base > 0) __syncthreads();
        for (int u = warp; u < pairs * seg; u += kPsWarps) {
          const int pr = u / seg, sg = u % seg;
          const int ra = base + 2 * pr, rb = min(ra + 1, C.rows - 1);
          double o[2][3];
          ps_row_pair(reinterpret_cast<const double2*>(C.mat + (size_t)ra * ld),
                      reinterpret_cast<const double2*>(C.mat + (size_t)rb * ld), reinterpret_cast<const double2*>(sx),
                      reinterpret_cast<const double2*>(sy), reinterpret_cast<const double2*>(sz), sg * len,
                      min(w2, (sg + 1) * len), o);
          if (lane == 0) {
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
              for (int c = 0; c < 3; ++c)
                if (2 * pr + r < nr) part[3 * ((2 * pr + r) * seg + sg) + c] = o[r][c];
          }
        }
        __syncthreads();
        for (int r = tid; r < nr; r += kPsThreads) {
          Vec3<double> v = ld3(part, r * seg);
          for (int sg = 1; sg < seg; ++sg) v = v + ld3(part, r * seg + sg);
          const int row = C.row0 + base + r;
          if (fwd && row >= C.n) {
            st3(b.contrib, b.cslot[C.rofs + row - C.n], v);
          } else {
            const int g = b.cols[C.cofs + row];
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
  for (int k = threadIdx.x & 31; k < n; k += 32) s += __ldcg(partial + k);
  return warp_sum(s);
}

// Sum of a vertex's slots by eight lanes (lane l adds slots l, l + 8, ..., then a fixed tree).
template <class T>
__device__ __forceinline__ Vec3<double> ps_sum_slots(const T* slot, int k0, int k1) {
  Vec3<double> a = mk3(0.0, 0.0, 0.0);
  for (int k = k0 + (int)(threadIdx.x & 7); k < k1; k += 8)
    a = a + mk3((double)slot[3 * (size_t)k], (double)slot[3 * (size_t)k + 1], (double)slot[3 * (size_t)k + 2]);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
    a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
    a.z += __shfl_xor_sync(0xffffffffu, a.z, o);
  }
  return a;
}

template <class BAR, bool MIXED>
__global__ void __launch_bounds__(kPsThreads, 1) k_pd_forward(SceneDev d, BlockDev b, PdSteps a) {
  extern __shared__ __align__(16) double pssh[];
  PsShared& S = *reinterpret_cast<PsShared*>(pssh);
  double* planes = pssh + (sizeof(PsShared) + 15) / 16 * 2;
  int* tab = reinterpret_cast<int*>(pssh + ps_fixed_doubles(b.vec));
  double* res = pssh + ps_fixed_doubles(b.vec) + a.tab_ints / 2;
  BAR bar(b.bar, b.status);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cta = BAR::cta(), nc = BAR::ctas();
  // items are dealt to the CTAs a warp's worth at a time
  const int first = 32 * (warp * nc + cta) + lane, stride = kPsThreads * nc;
  const bool lead = cta == 0 && tid == 0;
  const int s0 = a.step ? *a.step : a.s0;
  const int ncons = d.T + d.M + d.S + d.B;
  if (lead && a.zero)
    for (int q = 0; q < 4; ++q) a.status[q] = 0;
  ps_setup<BAR>(b, S, tab, a.tab_ints, res, a.res_doubles);
  if (a.x_in) {
    for (int i = first; i < d.N; i += stride) {
      const int u = a.to_user[i];
      st3(a.xt, i, ld3(a.x_in, u));
      st3(a.vt, i, ld3(a.v_in, u));
    }
    if (!bar.sync()) return;
  }
  int par = 0;
  double* xprev = a.xt;  // positions the step starts from, as every CTA reads them
  double* xk = a.xk;
  double* xo = a.xk2;
  for (int st = 0; st < a.n; ++st) {
    const int s = s0 + st;
    double* hist = a.hist + (size_t)s * a.hist_step;
    // begin (after the end of the step before): v_wc, q_n, x^0 = q_n, c0 = M/h^2 q_n - Hs x + J_att d_att
    double q2 = 0.0;
    for (int i = first; i < d.N; i += stride) {
      Vec3<double> x, v;
      if (st > 0) {
        x = ld3(xprev, i);
        v = (d.damping / d.h) * (x - ld3(a.xt, i));
        if (a.traj) st3(a.traj + (size_t)(s - 1) * 3 * d.N, a.to_user[i], x);
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
      if (!MIXED) {
        Vec3<double> acc = (d.mass[i] / (d.h * d.h)) * q;
        const int k1 = d.hs_ptr[i + 1];
        for (int k = d.hs_ptr[i]; k < k1; k += 8) {  // eight entries in flight, subtracted in order
          double w[8];
          Vec3<double> xj[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const bool in = k + u < k1;
            w[u] = in ? d.hs_val[k + u] : 0.0;
            xj[u] = in ? ld3(xprev, d.hs_col[k + u]) : mk3(0.0, 0.0, 0.0);
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) acc = acc - w[u] * xj[u];
        }
        st3(a.c0, i, acc + ld3(d.attach_jd, i));
      }
      if (st > 0) st3(a.xt, i, x);
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
      for (int t = first; t < ncons; t += stride) {
        if (MIXED) force_item(d, t, xk, act_row, reinterpret_cast<float*>(a.slot));
        else local_item(d, t, xk, act_row, a.slot);
      }
      if (!bar.sync()) return;
      for (int g = first >> 3; g < ((d.N + 3) & ~3); g += stride >> 3) {  // eight lanes per vertex
        const int i = min(g, d.N - 1);
        const int k0 = d.vslot_ptr[i], k1 = d.vslot_ptr[i + 1];
        if (MIXED) {
          const Vec3<double> f = ps_sum_slots(reinterpret_cast<const float*>(a.slot), k0, k1);
          if ((lane & 7) == 0 && g < d.N) {
            const Vec3<double> xi = ld3(xk, i);
            const double m = d.mass[i] / (d.h * d.h);
            st3(a.rhs, i, m * (ld3(a.qn, i) - xi) + ld3(d.attach_jd, i) - d.attach_k[i] * xi + f);
          }
        } else {
          const Vec3<double> f = ps_sum_slots(a.slot, k0, k1);
          if ((lane & 7) == 0 && g < d.N) st3(a.rhs, i, ld3(a.c0, i) + f);
        }
      }
      if (!bar.sync()) return;
      double e2 = 0.0;
      double* h1 = hist + (size_t)(k + 1) * 3 * d.N;
      const bool ok = ps_solve(b, bar, S, a.rhs, a.y, planes, [&](int g, Vec3<double> z) {
        // plain form: x^{k+1} = x_t + z (the reference's delta form); mixed form: x^{k+1} = x^k + z
        const Vec3<double> xc = ld3(xk, g);
        const Vec3<double> xn = (MIXED ? xc : ld3(a.xt, g)) + z;
        const Vec3<double> dl = xn - xc;
        e2 += dot3(dl, dl);
        st3(xk, g, xn);
        st3(h1, g, xn);
        if (b.tiers > 1) st3(a.y, g, z);  // read by the blocks below
      });
      if (!ok) return;
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
  BAR bar(b.bar, b.status);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cta = BAR::cta(), nc = BAR::ctas();
  const int first = 32 * (warp * nc + cta) + lane, stride = kPsThreads * nc;
  const int ncons = d.T + d.M + d.S + d.B, nmg = d.M + (d.sch ? d.S : 0);
  ps_setup<BAR>(b, S, tab, a.tab_ints, res, a.res_doubles);
  if (a.zero) {
    if (cta == 0 && tid < 4) a.status[tid] = 0;
    for (int t = first; t < d.T; t += stride) { a.gE[t] = 0.0; a.gnu[t] = 0.0; }
    for (int q = first; q < a.n * d.nseg; q += stride) a.gact[(size_t)a.s0 * d.nseg + q] = 0.0;
  }
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
      const bool ok = ps_solve(b, bar, S, a.xkb, a.y, planes, [&](int g, Vec3<double> y) {
        st3(a.y, g, y);
        st3(a.bb, g, ld3(a.bb, g) + y);
      });
      if (!ok || !bar.sync()) return;
      const double* x = hist + (size_t)k * 3 * d.N;
      const double* x1 = x + 3 * (size_t)d.N;
      if (warp < a.tape_warps) {
        for (int t = first; t < ncons; t += tstride * nc) {
          adj_local_item(d, t, x, a.y, act_row, a.slot, a.gE, a.gnu, a.mg, x1, nullptr, tape + tid, tstride);
          // activation terms: summed over the step's iterations by their constraint's thread
          const int m = t - d.T, q = m < d.M ? m : m - d.M;  // muscles, then springs
          if (m >= 0 && m < nmg && (m < d.M || d.sch[q] >= 0))
            a.mg[nmg + m] = k == nit - 1 ? a.mg[m] : a.mg[nmg + m] + a.mg[m];
        }
      }
      if (!bar.sync()) return;
      for (int g = first >> 3; g < ((d.N + 3) & ~3); g += stride >> 3) {
        const int i = min(g, d.N - 1);
        const Vec3<double> f = ps_sum_slots(a.slot, d.vslot_ptr[i], d.vslot_ptr[i + 1]);
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
