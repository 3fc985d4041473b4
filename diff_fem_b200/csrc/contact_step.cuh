// contact_step.cuh — the obstacle contact phase of a step (no soft contact),
// and its reverse sweep, each as one cooperative launch.
//
// Forward: the state machine of the kernels in contact_kernels.cuh (detection;
// Jacobi iterations until ori_x's max-norm change drops below EPS or K of them
// ran; detection again, until one finds no impact) on CTAs that are all
// resident, with grid barriers for kernel boundaries.  Every thread keeps the
// same copy of the state, updated from values read after a barrier; thread 0
// writes it to c.state for the step's record.  ori_x and x_n1 are two buffers
// that change places, so a Jacobi iteration has two phases: the local step,
// and the right-hand sides with the update and the next convergence test.
//
// Reverse: the recorded computed iterations j = top .. 1, two phases each.
// An iteration's local step and its impacts' frames need only its record, so
// they run beside the VJP of the iterations after it; the gather of one
// iteration and the right-hand-side VJP of the one before meet at the same
// vertex.
//
// What bounds both: dependent FP64 operations and L2 reads at less than a warp
// per scheduler (a scene of 10^4 elements).  So the work that a thread did in
// a row is spread: a tet on two threads (step_kernels.cuh), a vertex on eight
// lanes that read its slots and its row of Hs at once, an impact of it on
// each; a detection on a warp.  Only the sums stay in order, one lane per
// component, from shared memory: every result has the bits of the kernels'.
// 9,840-tet star on its ground: 33,500 cycles per Jacobi iteration with one
// thread per vertex (rows and slots read one by one) and 75,000 per reverse
// iteration; a detection of the 2,401-vertex cloth against the 1,280-face
// ball 160,000-210,000 with one thread per vertex, 18,000-20,000 now.  Six
// steps and their gradient: 8.5 -> 4.7 ms (star), 10.2 -> 5.3 ms (cloth).
#pragma once
#include "contact_kernels.cuh"
#include "step_kernels.cuh"

namespace dfem {

constexpr int kCtPlane = 33;                           // 32 values, odd: a vertex's components in different banks
constexpr int kCtSlots = 64;                           // slots of a vertex in one round
constexpr int kCtStage = 3 * kCtSlots + 4 * kCtPlane;  // doubles of a vertex: they, and 32 entries of its row (value, x_j)
constexpr int kCtWarpStage = 4 * kCtStage;             // four vertices per warp
constexpr int kCtAdjWarps = kPsWarps / 4;              // warps of a half that run the VJP (as many: the local step)
constexpr size_t kCtSmemFwd = sizeof(double) * (size_t)(kPsWarps * kCtWarpStage > kPsXch * kPsPair ? kPsWarps * kCtWarpStage : kPsXch * kPsPair);
constexpr int kCtTape = kPsXch * kPsPair;              // adjoint: the exchange, the tape, stages of the local step's warps
constexpr int kCtFrames = kCtTape + kVolTape * 32 * kCtAdjWarps;
constexpr size_t kCtSmemAdj = sizeof(double) * (size_t)(kCtFrames + 2 * kCtAdjWarps * kCtWarpStage);
static_assert(2 * kBroadMaxCandidates * sizeof(int) <= kCtWarpStage * sizeof(double), "a detection's lists");
static_assert(kMaxImpactsPerVertex <= 8, "one lane per impact");
static_assert(kCtSmemAdj >= kCtSmemFwd, "the adjoint's shared memory holds the stages");

// Sums of a vertex i (eight lanes each, four vertices per warp; every lane
// gets its vertex's): ss = init + its slots k0 .. k1 in order; sr = the sum
// over its row h0 .. h1 of Hs (the diagonal left out unless DIAG) of sign
// Hs_ij (p_j - q_j) in order (q: DIFF), from zero or (CHAIN) from ss; hii: the
// diagonal entry.  All reads of a round are in flight before the first sum
// (the slots go straight to the warp's stage w); the sums run on one lane per
// component.
template <bool DIFF, bool CHAIN, bool DIAG>
__device__ __forceinline__ void ct_sums(const SceneDev& d, int i, int k0, int k1, int h0, int h1, Vec3<double> init,
                                        const double* slot, const double* p, const double* q, double sign, double* w,
                                        Vec3<double>& ss, Vec3<double>& sr, double& hii) {
  const int l = threadIdx.x & 7;
  double* g = w + ((threadIdx.x & 31) >> 3) * kCtStage;
  double* gr = g + 3 * kCtSlots;
  const unsigned gs = (unsigned)__cvta_generic_to_shared(g);
  double as = l == 0 ? init.x : l == 1 ? init.y : init.z, ar = 0.0;
  hii = 0.0;
  for (bool start = false;;) {
    const bool last = !__any_sync(0xffffffffu, k1 - k0 > kCtSlots);  // the rest of the slots: rows too
    const int n = 3 * max(0, min(kCtSlots, k1 - k0)), m = last ? max(0, min(32, h1 - h0)) : 0;
    const double* ps = slot + 3 * (size_t)k0;
    double val[4];
    int col[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool on = l + 8 * u < m;
      col[u] = on ? d.hs_col[h0 + l + 8 * u] : i;
      val[u] = on ? sign * d.hs_val[h0 + l + 8 * u] : 0.0;
    }
#pragma unroll 4
    for (int e = l; e < n; e += 8)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(gs + 8 * e), "l"(ps + e) : "memory");
    Vec3<double> x[4], y[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool on = l + 8 * u < m;
      x[u] = on ? ld3(p, col[u]) : mk3(0.0, 0.0, 0.0);
      if (DIFF) y[u] = on ? ld3(q, col[u]) : mk3(0.0, 0.0, 0.0);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = l + 8 * u;
      Vec3<double> v = DIFF ? x[u] - y[u] : x[u];
      if (!DIAG && e < m && col[u] == i) {  // adds an exact zero
        hii = sign * val[u];
        val[u] = 0.0;
        v = mk3(0.0, 0.0, 0.0);
      }
      gr[e] = val[u];
      gr[kCtPlane + e] = v.x;
      gr[2 * kCtPlane + e] = v.y;
      gr[3 * kCtPlane + e] = v.z;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    if (l < 3) {
#pragma unroll 8
      for (int k = l; k < n; k += 3) as += g[k];
      if (CHAIN && last && !start) ar = as;
#pragma unroll 8
      for (int k = 0; k < m; ++k) ar = __fma_rn(gr[k], gr[kCtPlane * (1 + l) + k], ar);
    }
    __syncwarp();
    start = start || last;
    k0 += kCtSlots;
    h0 += last ? 32 : 0;
    if (last && !__any_sync(0xffffffffu, h0 < h1)) break;
  }
  if (!DIAG) {  // one lane of the vertex met it
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      const double t = __shfl_xor_sync(0xffffffffu, hii, o);
      hii = hii != 0.0 ? hii : t;
    }
  }
  ss = mk3(__shfl_sync(0xffffffffu, as, 0, 8), __shfl_sync(0xffffffffu, as, 1, 8), __shfl_sync(0xffffffffu, as, 2, 8));
  sr = mk3(__shfl_sync(0xffffffffu, ar, 0, 8), __shfl_sync(0xffffffffu, ar, 1, 8), __shfl_sync(0xffffffffu, ar, 2, 8));
}

// Detection of contact vertex a by a warp (contact_detect_item's result): the
// lanes read the candidate cells' faces and keep those whose boxes meet the
// swept vertex, each once; these are tested 32 at a time in ascending order,
// and lane 0 applies the hits.  list: 2 kBroadMaxCandidates ints.
__device__ __forceinline__ bool ct_detect(const ContactDev& c, int a, const double* xt, const double* xk, int* list,
                                          int* status) {
  const int lane = threadIdx.x & 31;
  const int gv = c.cverts[a];
  const Vec3<double> p0 = ld3(xt, gv), p1 = ld3(xk, gv);
  const Vec3<double> lo = mk3(fmin(p0.x, p1.x), fmin(p0.y, p1.y), fmin(p0.z, p1.z));
  const Vec3<double> hi = mk3(fmax(p0.x, p1.x), fmax(p0.y, p1.y), fmax(p0.z, p1.z));
  int* sorted = list + kBroadMaxCandidates;
  bool culled = c.bp_max_cells > 0 && c.bp_dim[0] > 0;
  int n = 0;
  if (culled) {
    const int x0 = bp_cell(c, lo.x - kBroadPad, 0), x1 = bp_cell(c, hi.x + kBroadPad, 0);
    const int y0 = bp_cell(c, lo.y - kBroadPad, 1), y1 = bp_cell(c, hi.y + kBroadPad, 1);
    const int z0 = bp_cell(c, lo.z - kBroadPad, 2), z1 = bp_cell(c, hi.z + kBroadPad, 2);
    culled = (long long)(x1 - x0 + 1) * (y1 - y0 + 1) * (z1 - z0 + 1) <= c.bp_max_cells;
    for (int z = z0; culled && z <= z1; ++z)
      for (int y = y0; culled && y <= y1; ++y) {  // a row of cells: their faces are consecutive
        const int row = (z * c.bp_dim[1] + y) * c.bp_dim[0];
        const int k1 = c.bp_ptr[row + x1 + 1];
        for (int k0 = c.bp_ptr[row + x0]; culled && k0 < k1; k0 += 32) {
          const int f = k0 + lane < k1 ? c.bp_face[k0 + lane] : -1 - lane;
          bool in = f >= 0;
          if (in) {
            const int* fv = c.obs_f + 3 * f;
            const Vec3<double> q0 = ld3(c.obs_x, fv[0]), q1 = ld3(c.obs_x, fv[1]), q2 = ld3(c.obs_x, fv[2]);
            const double th = kContactThickness;  // vf_impact's box test
            in = !(hi.x < fmin(q0.x, fmin(q1.x, q2.x)) - th || lo.x > fmax(q0.x, fmax(q1.x, q2.x)) + th ||
                   hi.y < fmin(q0.y, fmin(q1.y, q2.y)) - th || lo.y > fmax(q0.y, fmax(q1.y, q2.y)) + th ||
                   hi.z < fmin(q0.z, fmin(q1.z, q2.z)) - th || lo.z > fmax(q0.z, fmax(q1.z, q2.z)) + th);
          }
          const unsigned same = __match_any_sync(0xffffffffu, in ? f : -1 - lane);
          in = in && (same & ((1u << lane) - 1)) == 0;  // the face's first lane
          for (int k = 0; in && k < n; ++k) in = list[k] != f;
          const unsigned m = __ballot_sync(0xffffffffu, in);
          if (n + __popc(m) > kBroadMaxCandidates) {
            culled = false;  // as many as that: every face instead
          } else {
            if (in) list[n + __popc(m & ((1u << lane) - 1))] = f;
            n += __popc(m);
          }
          __syncwarp();
        }
      }
    if (culled) {
      for (int k = lane; k < n; k += 32) {
        int r = 0;
        for (int q = 0; q < n; ++q) r += list[q] < list[k];
        sorted[r] = list[k];
      }
      __syncwarp();
    }
  }
  const int total = culled ? n : c.nof;
  bool any = false;
  for (int b = 0; b < total; b += 32) {
    const int f = b + lane < total ? (culled ? sorted[b + lane] : b + lane) : -1;
    Vec3<double> nrm = mk3(0.0, 0.0, 0.0);
    bool hit = false;
    if (f >= 0) {
      const int* fv = c.obs_f + 3 * f;
      hit = vf_impact(p0, p1, ld3(c.obs_x, fv[0]), ld3(c.obs_x, fv[1]), ld3(c.obs_x, fv[2]), 1.0, &nrm);
    }
    unsigned m = __ballot_sync(0xffffffffu, hit);
    any = any || m != 0;
    while (m) {
      const int src = __ffs(m) - 1;
      m &= m - 1;
      const int fs = __shfl_sync(0xffffffffu, f, src);
      const Vec3<double> ns = mk3(__shfl_sync(0xffffffffu, nrm.x, src), __shfl_sync(0xffffffffu, nrm.y, src),
                                  __shfl_sync(0xffffffffu, nrm.z, src));
      if (lane == 0) impact_add(c, a, fs, ns, status);
    }
  }
  __syncwarp();
  return any;
}

// Max over the CTA into *partial; ct_max gives every thread the grid's after a barrier.
__device__ __forceinline__ void ct_put_max(double e, double* ws, double* partial) {
  for (int o = 16; o > 0; o >>= 1) e = fmax(e, __shfl_xor_sync(0xffffffffu, e, o));
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = e;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = ws[0];
#pragma unroll
    for (int w = 1; w < kPsWarps; ++w) m = fmax(m, ws[w]);
    *partial = m;
  }
}
// (One warp reads: with all of them the reads of the same few lines queue.)
__device__ __forceinline__ double ct_max(const double* partial, int n, double* ws) {
  if (threadIdx.x < 32) {
    double m = 0.0;
#pragma unroll 5
    for (int b = threadIdx.x; b < n; b += 32) m = fmax(m, __ldcg(partial + b));
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) ws[0] = m;
  }
  __syncthreads();
  return ws[0];
}
__device__ __forceinline__ double ct_norm(Vec3<double> a) { return fmax(fabs(a.x), fmax(fabs(a.y), fabs(a.z))); }

// A half of a tet's local step and its corners' slots after the exchange
// (local_item's bits: wr md + wv md_volume as one fused multiply-add).
struct CtTet {
  double G[4][3], wr;
  Vec3<double> P[3];
  int4 sl;
};
__device__ __forceinline__ void ct_tet_give(const SceneDev& d, int t, int4 v, const double* x, bool rot, double* xch, int me,
                                            CtTet& T) {
  const Vec3<double> xv[4] = {ld3(x, v.x), ld3(x, v.y), ld3(x, v.z), ld3(x, v.w)};
  load_g(d.tinv, d.T, t, T.G);
  const double wv = d.twv[t];
  T.wr = d.twr[t];
  T.sl = d.tslot[t];
  const Mat3<double> F = deformation_rn(T.G, xv);
  Mat3<double> m;
  if (rot) corot_rotation(F, m);
  else corot_volume(F, m);
#pragma unroll
  for (int j = 0; j < 3; ++j) T.P[j] = rot ? m.c[j] : rn_scale(wv, m.c[j]);
  ps_give(xch, rot, me, T.P);
}
__device__ __forceinline__ void ct_tet_take(bool rot, const double* xch, int me, CtTet& T, double* slot) {
  const double* o = xch + (rot ? 9 : 0) * kPsPair + me;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const Vec3<double> q = mk3(o[(3 * j) * kPsPair], o[(3 * j + 1) * kPsPair], o[(3 * j + 2) * kPsPair]);
    T.P[j] = rot ? rn_axpy(T.wr, T.P[j], q) : rn_axpy(T.wr, q, T.P[j]);
  }
  ps_corners(T.G, T.P, T.sl, rot, slot);
}

__global__ void __launch_bounds__(kPsThreads, 1) k_contact_phase(const __grid_constant__ SceneDev d,
                                                                 const __grid_constant__ ContactDev c, const double* xt,
                                                                 double* xk, const double* act_all, const int* step,
                                                                 double* slot, double* partial, unsigned* counter, int tries,
                                                                 int* status) {
  extern __shared__ __align__(16) double dyn[];
  __shared__ double ws[kPsWarps];
  if (GridBarrier::gave_up(status)) return;
  GridBarrier bar(counter, status, tries);
  const int nc = gridDim.x, cta = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wid = warp * nc + cta, nw = kPsWarps * nc;  // a warp's share: CTAs first
  const int tid = wid * 32 + lane, nthr = nw * 32;
  const bool lead = tid == 0;
  const int me = threadIdx.x & (kPsPair - 1);
  const bool rot = warp < kPsWarps / 2;
  double* stage = dyn + warp * kCtWarpStage;
  const double* act_row = act_all + (size_t)(*step) * d.nseg;
  const int t0 = 32 * ((warp & (kPsWarps / 2 - 1)) * nc + cta) + lane;  // this thread's first tet
  const int4 tv0 = t0 < d.T ? d.tv[t0] : make_int4(0, 0, 0, 0);
  const int rec_on = c.rec_on ? *c.rec_on : 0, rec_base = rec_on ? *c.rec_base : 0;
  // k_contact_begin: L x_t, empty lists; ori_x = x_n1 = the PD result, xold = 0
  double e = 0.0;
  for (int b = 4 * wid; b < d.N; b += 4 * nw) {
    const int i = b + (lane >> 3), ii = min(i, d.N - 1);
    Vec3<double> s, none;
    double hii;
    ct_sums<false, false, true>(d, ii, 0, 0, d.hs_ptr[ii], i < d.N ? d.hs_ptr[ii + 1] : 0, mk3(0.0, 0.0, 0.0), slot, xt, xt, 1.0,
                                stage, none, s, hii);
    if (i < d.N && (lane & 7) == 0) {
      st3(c.lxt, i, rn_axpy(-(d.mass[i] / (d.h * d.h)), ld3(xt, i), s));
      e = fmax(e, ct_norm(ld3(xk, i)));
    }
  }
  for (int a = tid; a < c.nc; a += nthr) {
    c.imp_cnt[a] = 0;
    if (c.ncf > 0) c.simp_cnt[a] = 0;
  }
  if (lead)
    for (int k = 0; k < CS_SIZE; ++k) c.state[k] = 0;
  if (!(c.nc > 0 && c.nof > 0)) return;  // uniform, before any barrier
  ct_put_max(e, ws, partial + cta);
  if (!bar.sync()) return;
  int ori = 0, nxt = 0;  // the buffers of ori_x and x_n1 (xk, c.xn1)
  int mode = 0, pass = 0, it = 0, bodies = 0, comp = 0, src = 0, ndet = 0;
  const int cap = c.max_passes * (c.K + 2) + 2;
  for (;;) {
    bodies += 1;
    if (mode == 0) {  // detection pass (k_contact_detect, k_contact_ctl_detect)
      int* flag = c.state + CS_HIT + hit_word(ndet);
      for (int a = wid; a < c.nc; a += nw)
        if (ct_detect(c, a, xt, ori ? c.xn1 : xk, (int*)stage, status) && lane == 0) atomicOr(flag, 1);
      if (!bar.sync()) return;
      const bool any = *(volatile int*)flag != 0;
      if (lead) c.state[CS_HIT + cleared_word(ndet)] = 0;  // (contact_flags.h)
      ++ndet;
      if (!any) break;
      if (pass >= c.max_passes) {
        if (lead) cap_reached(status, kCapContactPasses);
        break;
      }
      mode = 1;
      it = 0;
      pass += 1;
    }
    // one Jacobi iteration (k_contact_prep, k_local, k_contact_rhs, k_contact_ctl_iter)
    const int rk = rec_on && rec_base + comp < c.rec_cap ? rec_base + comp : -1;
    ori = nxt;
    src = comp;
    if (ct_max(partial, nc, ws) < kConvergenceEps) {
      mode = 0;  // back to detection
    } else {
      const double* x = ori ? c.xn1 : xk;
      double* xn = ori ? xk : c.xn1;
      for (int base = 0; base < d.T; base += kPsPair * nc) {
        const int t = base + t0;
        CtTet T;
        if (t < d.T) ct_tet_give(d, t, base == 0 ? tv0 : d.tv[t], x, rot, dyn, me, T);
        __syncthreads();
        if (t < d.T) ct_tet_take(rot, dyn, me, T, slot);
        if (base + kPsPair * nc < d.T) __syncthreads();
      }
      for (int t = nthr - 32 * (wid + 1) + lane; t < d.M + d.S + d.B; t += nthr) local_rest(d, t, x, act_row, slot);
      if (!bar.sync()) return;
      const bool first = it == 0;
      e = 0.0;
      for (int b = 4 * wid; b < d.N; b += 4 * nw) {
        const int i = b + (lane >> 3), ii = min(i, d.N - 1), l = lane & 7;
        const bool on = i < d.N;
        const int a = on ? c.cidx[ii] : -1, cnt = a >= 0 ? c.imp_cnt[a] : 0;
        const int k0 = d.vslot_ptr[ii], k1 = on ? d.vslot_ptr[ii + 1] : 0, h0 = d.hs_ptr[ii], h1 = on ? d.hs_ptr[ii + 1] : 0;
        const Vec3<double> xi = ld3(x, ii), xti = ld3(xt, ii), vwc = ld3(c.vwc, ii), lxt = ld3(c.lxt, ii);
        const Vec3<double> before = ld3(c.prev, ii);
        const double mass = d.mass[ii], hdiag = c.hdiag[ii];
        Vec3<double> nrm = mk3(0.0, 0.0, 0.0), jd, cdx;
        if (l < cnt) nrm = ld3(c.imp_n, a * kMaxImpactsPerVertex + l);
        double hii;
        ct_sums<true, false, false>(d, ii, k0, k1, h0, h1, ld3(d.attach_jd, ii), slot, x, xt, 1.0, stage, jd, cdx, hii);
        const Vec3<double> rhs = contact_rhs_value(mass, vwc, d.h, jd, lxt, cdx);
        Vec3<double> post = rhs, r = rhs;
        const bool hit = l < cnt && contact_reaction(nrm, rhs, c.mu, &r);
        const unsigned m = (__ballot_sync(0xffffffffu, hit) >> (lane & 24)) & 0xffu;
        const int win = m ? 31 - __clz(m) : 0;  // the last impact's reaction
        const Vec3<double> rw = mk3(__shfl_sync(0xffffffffu, r.x, win, 8), __shfl_sync(0xffffffffu, r.y, win, 8),
                                    __shfl_sync(0xffffffffu, r.z, win, 8));
        if (m) post = rw;
        if (on && l == 0) {
          const Vec3<double> prev = contact_relax(c.alpha, post, first ? rhs : before);
          const Vec3<double> xnew = contact_xn1(d.h, hdiag, prev, xti);
          st3(c.prev, i, prev);
          st3(xn, i, xnew);
          e = fmax(e, ct_norm(xnew - xi));
          if (rk >= 0) {
            st3(c.rec_x + (size_t)rk * 3 * d.N, i, xi);
            st3(c.rec_prev + (size_t)rk * 3 * d.N, i, prev);
            if (i == 0) c.rec_first[rk] = first ? 1 : 0;
          }
        }
        if (rk >= 0 && a >= 0) {  // the impacts this iteration used
          if (l == 0) c.rec_cnt[(size_t)rk * c.nc + a] = cnt;
          if (l < cnt) st3(c.rec_n + ((size_t)rk * c.nc + a) * kMaxImpactsPerVertex * 3, l, nrm);
        }
      }
      nxt = 1 - ori;
      ct_put_max(e, ws, partial + cta);
      if (!bar.sync()) return;
      it += 1;
      if (lead && rec_on == 1 && rec_base + comp >= c.rec_cap) atomicExch(status, 6);
      comp += 1;
      if (it >= c.K) mode = 0;
    }
    if (bodies > cap) {  // unreachable: passes and iterations are bounded above
      if (lead) cap_reached(status, kCapContactPasses);
      break;
    }
  }
  if (ori == 1)  // the phase's result; x_n1 there is not needed any more
    for (int k = tid; k < 3 * d.N; k += nthr) xk[k] = c.xn1[k];
  if (lead) {
    c.state[CS_MODE] = mode; c.state[CS_PASS] = pass; c.state[CS_IT] = it; c.state[CS_BODIES] = bodies;
    c.state[CS_COMP] = comp; c.state[CS_SRC] = src;
  }
  bar.leave();
}

// Reverse sweep: k_cadj_start, the iterations j = top .. 1 (records base + j -
// 1; contact_adjoint_step's kernels), the diag(Hs) terms of dL/dE and the PD
// part's cotangent.  Round j: the constraints' VJP at iteration j's input, and
// on other warps the frames of iteration j - 1's impacts and the local step at
// j - 2's input (both need records only); then the vertices, which gather
// iteration j and reverse the update of j - 1.  yb and a.orib alternate as the
// iterations' y-bar, slot2 holds the local step's slots of two iterations
// (slot: the VJP's).
struct CtFrames {
  double* slot2;  // 2 x 3 nslots
  size_t slots3;
  double* fr;     // nc x 12: W, r of the winning impact (contact_frame)
  int* hit;       // nc
};

__global__ void __launch_bounds__(kPsThreads, 1) k_cadj_phase(const __grid_constant__ SceneDev d,
                                                              const __grid_constant__ ContactDev c,
                                                              const __grid_constant__ ContactAdj a, const CtFrames fr,
                                                              const double* xt, const double* act_all, const int* step,
                                                              double* slot, double* gE, double* gnu, double* mg, double* gact,
                                                              int base, int top, double cv, double* io_a, double* io_b,
                                                              unsigned* counter, int tries, int* status) {
  extern __shared__ __align__(16) double dyn[];
  if (GridBarrier::gave_up(status)) return;
  GridBarrier bar(counter, status, tries);
  const int nc = gridDim.x, cta = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wid = warp * nc + cta, nw = kPsWarps * nc;
  const int tid = wid * 32 + lane, nthr = nw * 32;
  const int me = threadIdx.x & (kPsPair - 1);
  const bool rot = warp < kPsWarps / 2;
  const int hw = warp & (kPsWarps / 2 - 1), hq = hw & (kCtAdjWarps - 1);
  const bool vjp = hw < kCtAdjWarps;  // this warp's tets: the VJP, or the local step
  double* stage = dyn + warp * kCtWarpStage;
  double* tape = dyn + kCtTape + 32 * hq + lane;
  const int fw = (rot ? 0 : kCtAdjWarps) + hq;  // a local-step warp's place among them
  double* fstage = dyn + kCtFrames + fw * kCtWarpStage;
  const size_t n3 = 3 * (size_t)d.N;
  const int st = *step, rest = d.M + d.S + d.B;
  const double* act_row = act_all + (size_t)st * d.nseg;
  const int t0 = 32 * (hq * nc + cta) + lane;
  const int4 tv0 = t0 < d.T ? d.tv[t0] : make_int4(0, 0, 0, 0);
  for (int j = top + 2; j >= 1; --j) {
    const double* yb = (j & 1) ? a.yb : a.orib;   // of iteration j
    double* ybn = (j & 1) ? a.orib : a.yb;        // of j - 1
    {  // constraints
      const bool do_vjp = j <= top, do_loc = j >= 3;
      const double* x = c.rec_x + ((size_t)base + (do_vjp ? j - 1 : 0)) * n3;
      const double* xl = c.rec_x + ((size_t)base + (do_loc ? j - 3 : 0)) * n3;
      double* lslot = fr.slot2 + (j & 1) * fr.slots3;
      const bool run = vjp ? do_vjp : do_loc;
      if (!vjp && j >= 2 && j <= top + 1) {  // the frames of iteration j - 1
        const size_t r = (size_t)base + j - 2;
        const double* ori = c.rec_x + r * n3;
        const int* rcnt = c.rec_cnt + r * c.nc;
        const double* rn = c.rec_n + r * c.nc * kMaxImpactsPerVertex * 3;
        const double* fslot = fr.slot2 + ((j + 1) & 1) * fr.slots3;
        for (int b = 4 * (fw * nc + cta); b < c.nc; b += 8 * kCtAdjWarps * nc) {
          const int ac = b + (lane >> 3), l = lane & 7, cnt = ac < c.nc ? rcnt[ac] : 0;
          if (!__any_sync(0xffffffffu, cnt > 0)) {
            if (l == 0 && ac < c.nc) fr.hit[ac] = 0;
            continue;
          }
          const int i = c.cverts[min(ac, c.nc - 1)];
          const bool on = cnt > 0;
          const int k0 = d.vslot_ptr[i], k1 = on ? d.vslot_ptr[i + 1] : 0, h0 = d.hs_ptr[i], h1 = on ? d.hs_ptr[i + 1] : 0;
          const Vec3<double> vwc = ld3(c.vwc, i), lxt = ld3(c.lxt, i);
          const double mass = d.mass[i];
          Vec3<double> nrm = mk3(0.0, 0.0, 0.0), jd, cdx, W[3];
          if (l < cnt) nrm = ld3(rn, ac * kMaxImpactsPerVertex + l);
          double hii, rc[3];
          ct_sums<true, false, false>(d, i, k0, k1, h0, h1, ld3(d.attach_jd, i), fslot, ori, xt, 1.0, fstage, jd, cdx, hii);
          const Vec3<double> f = contact_rhs_value(mass, vwc, d.h, jd, lxt, cdx);
          const bool hit = l < cnt && contact_frame(nrm, f, W, rc);
          const unsigned m = (__ballot_sync(0xffffffffu, hit) >> (lane & 24)) & 0xffu;
          if (ac < c.nc) {
            if (l == 0) fr.hit[ac] = m != 0;
            if (m && l == 31 - __clz(m)) {
              double* o = fr.fr + 12 * (size_t)ac;
#pragma unroll
              for (int q = 0; q < 3; ++q) {
                st3(o, q, W[q]);
                o[9 + q] = rc[q];
              }
            }
          }
        }
      }
      for (int b = 0; b < d.T; b += 32 * kCtAdjWarps * nc) {
        const int t = run ? b + t0 : d.T;
        CtTet T;
        double yv = 0.0;
        if (t < d.T) {
          const int4 v = b == 0 ? tv0 : d.tv[t];
          if (vjp) {
            const int vi[4] = {v.x, v.y, v.z, v.w};
            Vec3<double> xv[4], yw[4];
            Mat3<double> gF;
#pragma unroll
            for (int q = 0; q < 4; ++q) { xv[q] = ld3(x, vi[q]); yw[q] = ld3(yb, vi[q]); }
            load_g(d.tinv, d.T, t, T.G);
            T.sl = d.tslot[t];
            const Mat3<double> F = deformation_rn(T.G, xv), Y = deformation_rn(T.G, yw);
            if (rot) {
              double yr;
              corot_adjoint_rotation(F, Y, d.twr[t], yr, gF);
              dyn[18 * kPsPair + me] = yr;
#pragma unroll
              for (int q = 0; q < 4; ++q) { xv[q] = ld3(x, vi[q]); yw[q] = ld3(yb, vi[q]); }  // again: fewer live registers
              dyn[19 * kPsPair + me] = contact_yh(T.G, F, Y, yw, xv, xt, vi);
            } else {
              corot_adjoint_volume(F, Y, d.twv[t], yv, gF, tape, 32 * kCtAdjWarps);
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) T.P[q] = gF.c[q];
            ps_give(dyn, rot, me, T.P);
          } else {
            ct_tet_give(d, t, v, xl, rot, dyn, me, T);
          }
        }
        __syncthreads();
        if (t < d.T) {
          if (vjp) {
            ps_take(dyn, rot, me, T.P);
            ps_corners(T.G, T.P, T.sl, rot, slot);
            if (!rot) {
              tet_moduli_grad(gE, gnu, t, d.tE[t], d.tnu[t], d.tvol[t], dyn[18 * kPsPair + me], yv, dyn[19 * kPsPair + me]);
            }
          } else {
            ct_tet_take(rot, dyn, me, T, lslot);
          }
        }
        if (b + 32 * kCtAdjWarps * nc < d.T) __syncthreads();
      }
      for (int q = nthr - 32 * (wid + 1) + lane; q < 2 * rest; q += nthr) {  // the last warps first
        if (q < rest) {
          if (do_vjp) adj_local_rest(d, q, x, yb, act_row, slot, mg);
        } else if (do_loc) {
          local_rest(d, q - rest, xl, act_row, lslot);
        }
      }
      if (!bar.sync()) return;
    }
    if (j > top + 1) continue;
    // vertices: the gather of iteration j (x_n1 bar of j - 1; at top + 1 the phase's own), the reverse of j - 1's update
    const bool gather = j <= top, rhs = j >= 2;
    const size_t r = (size_t)base + (rhs ? j - 2 : 0);
    const double* prev = c.rec_prev + r * n3;
    const int first = rhs ? c.rec_first[r] : 0;
    for (int b = 4 * wid; b < d.N; b += 4 * nw) {
      const int i = b + (lane >> 3), ii = min(i, d.N - 1), l = lane & 7;
      const bool on = i < d.N;
      Vec3<double> xb;
      const int ac = rhs ? c.cidx[ii] : -1;
      const int hit = ac >= 0 ? fr.hit[ac] : 0;
      Vec3<double> W[3], pv = mk3(0.0, 0.0, 0.0);
      double rc[3] = {0.0, 0.0, 0.0};
      if (rhs) pv = ld3(prev, ii);
      if (hit) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          W[q] = ld3(fr.fr + 12 * (size_t)ac, q);
          rc[q] = fr.fr[12 * (size_t)ac + 9 + q];
        }
      }
      if (!gather) {
        const Vec3<double> gv = ld3(io_b, ii);
        xb = ld3(io_a, ii) + cv * gv;
        if (on && l == 0) {
          st3(a.cxtb, i, (-cv) * gv);
          st3(a.vwcb, i, mk3(0.0, 0.0, 0.0));
          st3(a.pb, i, mk3(0.0, 0.0, 0.0));
          a.hdb[i] = 0.0;
        }
      } else {
        const int k0 = d.vslot_ptr[ii], k1 = on ? d.vslot_ptr[ii + 1] : 0, h0 = d.hs_ptr[ii], h1 = on ? d.hs_ptr[ii + 1] : 0;
        const Vec3<double> yi = ld3(yb, ii), xtb = ld3(a.cxtb, ii);
        const double mass = d.mass[ii];
        double hii;
        Vec3<double> none;
        ct_sums<false, true, false>(d, ii, k0, k1, h0, h1, mk3(0.0, 0.0, 0.0), slot, yb, yb, -1.0, stage, none, xb, hii);
        if (on && l == 0) st3(a.cxtb, i, rn_axpy(mass / (d.h * d.h) - hii, yi, xtb));
      }
      if (on && l == 0) {
        if (rhs) {
          cadj_rhs_finish(d, c, a, i, xb, pv, first, hit != 0, W, rc, ybn);
        } else {  // k_cadj_to_pd
          st3(io_a, i, xb);
          st3(io_b, i, mk3(0.0, 0.0, 0.0));
        }
      }
      __syncwarp();
    }
    if (gather)
      for (int q = nthr - 1 - tid; q < d.nseg; q += nthr) {  // k_seg_reduce
        double sum = 0;
#pragma unroll 4
        for (int k = d.seg_ptr[q]; k < d.seg_ptr[q + 1]; ++k) sum += mg[member_slot(d.M, d.seg_mus[k])];
        gact[(size_t)st * d.nseg + q] += sum;
      }
    if (j > 1 && !bar.sync()) return;
  }
  if (top > 0)  // hdb: complete since the barriers after iteration 1 (zero without one)
    for (int t = tid; t < d.T; t += nthr) cadj_hd_item(d, a, t, gE);
  bar.leave();
}

}  // namespace dfem
