// pd_math.cuh — per-element math of the PD local step and its adjoint, for
// one thread per element (templated on the arithmetic type: double for the
// plain form, float for the mixed form).
//
// Corotated projection (diff_fem sim/fem/Constraint/CorotateFEMConstraint.h:354-377):
//   F = Ds * invDm;  SVD F = U S V^T (S >= 0, like Eigen::JacobiSVD);
//   md = R = U V^T, with column 2 negated when det F < 0;
//   md_volume = U diag(S + D) V^T, D from 5 Newton steps projecting S onto prod = 1.
// R and U diag(g(S)) V^T do not depend on the SVD's sign/ordering choices, so
// the result equals the reference's for any exact SVD.  The SVD here is the
// one-sided (Hestenes) Jacobi method: rotate column pairs of F until they are
// orthogonal; singular values are the column norms.
#pragma once
#include <cuda_runtime.h>

namespace dfem {

template <typename T> struct Vec3 { T x, y, z; };
template <typename T> __device__ __forceinline__ Vec3<T> mk3(T a, T b, T c) { return {a, b, c}; }
template <typename T> __device__ __forceinline__ Vec3<T> operator+(Vec3<T> a, Vec3<T> b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
template <typename T> __device__ __forceinline__ Vec3<T> operator-(Vec3<T> a, Vec3<T> b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
template <typename T> __device__ __forceinline__ Vec3<T> operator*(T s, Vec3<T> a) { return {s * a.x, s * a.y, s * a.z}; }
template <typename T> __device__ __forceinline__ T dot3(Vec3<T> a, Vec3<T> b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
template <typename T> __device__ __forceinline__ Vec3<T> cross3(Vec3<T> a, Vec3<T> b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

template <typename T> __device__ __forceinline__ T dsqrt(T v);
template <> __device__ __forceinline__ double dsqrt<double>(double v) { return sqrt(v); }
template <> __device__ __forceinline__ float dsqrt<float>(float v) { return sqrtf(v); }
template <typename T> __device__ __forceinline__ T drsqrt(T v);
template <> __device__ __forceinline__ double drsqrt<double>(double v) { return rsqrt(v); }
template <> __device__ __forceinline__ float drsqrt<float>(float v) { return rsqrtf(v); }
template <typename T> __device__ __forceinline__ T dabs(T v) { return v < T(0) ? -v : v; }

template <typename T> struct Eps;
template <> struct Eps<double> { static constexpr double rot = 1e-15; static constexpr double rel = 1e-14; static constexpr int sweeps = 10; };
template <> struct Eps<float> { static constexpr float rot = 1e-7f; static constexpr float rel = 1e-6f; static constexpr int sweeps = 6; };

// 3x3 matrices as three column vectors c[0..2]
template <typename T> struct Mat3 { Vec3<T> c[3]; };

template <typename T> __device__ __forceinline__ T det3(const Mat3<T>& a) { return dot3(a.c[0], cross3(a.c[1], a.c[2])); }

template <typename T> struct Svd3 {
  Vec3<T> u[3], v[3];  // columns of U and V
  T s[3];              // singular values (>= 0), unsorted
};

template <typename T>
__device__ __forceinline__ void jacobi_rotate(Vec3<T>& bp, Vec3<T>& bq, Vec3<T>& vp, Vec3<T>& vq, bool& rotated) {
  T a = dot3(bp, bp), b = dot3(bq, bq), g = dot3(bp, bq);
  if (!(dabs(g) > Eps<T>::rot * dsqrt(a * b))) return;
  rotated = true;
  T zeta = (b - a) / (T(2) * g);
  T t = (zeta >= T(0) ? T(1) : T(-1)) / (dabs(zeta) + dsqrt(T(1) + zeta * zeta));
  T c = drsqrt(T(1) + t * t);
  T s = c * t;
  Vec3<T> nbp = c * bp - s * bq, nbq = s * bp + c * bq;
  Vec3<T> nvp = c * vp - s * vq, nvq = s * vp + c * vq;
  bp = nbp; bq = nbq; vp = nvp; vq = nvq;
}

template <typename T>
__device__ __forceinline__ Svd3<T> svd3(const Mat3<T>& F) {
  Svd3<T> o;
  Vec3<T> b0 = F.c[0], b1 = F.c[1], b2 = F.c[2];
  Vec3<T> v0 = mk3<T>(1, 0, 0), v1 = mk3<T>(0, 1, 0), v2 = mk3<T>(0, 0, 1);
#pragma unroll 1
  for (int sweep = 0; sweep < Eps<T>::sweeps; ++sweep) {
    bool rotated = false;
    jacobi_rotate(b0, b1, v0, v1, rotated);
    jacobi_rotate(b0, b2, v0, v2, rotated);
    jacobi_rotate(b1, b2, v1, v2, rotated);
    if (!rotated) break;
  }
  T s0 = dsqrt(dot3(b0, b0)), s1 = dsqrt(dot3(b1, b1)), s2 = dsqrt(dot3(b2, b2));
  // sort descending (keeps the degenerate-completion rule simple)
  if (s0 < s1) { T t = s0; s0 = s1; s1 = t; Vec3<T> tb = b0; b0 = b1; b1 = tb; Vec3<T> tv = v0; v0 = v1; v1 = tv; }
  if (s0 < s2) { T t = s0; s0 = s2; s2 = t; Vec3<T> tb = b0; b0 = b2; b2 = tb; Vec3<T> tv = v0; v0 = v2; v2 = tv; }
  if (s1 < s2) { T t = s1; s1 = s2; s2 = t; Vec3<T> tb = b1; b1 = b2; b2 = tb; Vec3<T> tv = v1; v1 = v2; v2 = tv; }
  o.s[0] = s0; o.s[1] = s1; o.s[2] = s2;
  o.v[0] = v0; o.v[1] = v1; o.v[2] = v2;
  const T tiny = Eps<T>::rel * s0;
  if (s0 > T(0)) o.u[0] = (T(1) / s0) * b0; else o.u[0] = mk3<T>(1, 0, 0);
  if (s1 > tiny) {
    o.u[1] = (T(1) / s1) * b1;
  } else {  // complete the basis: a direction orthogonal to u0
    Vec3<T> e = dabs(o.u[0].x) < T(0.9) ? mk3<T>(1, 0, 0) : mk3<T>(0, 1, 0);
    Vec3<T> w = cross3(o.u[0], e);
    o.u[1] = drsqrt(dot3(w, w)) * w;
  }
  if (s2 > tiny) o.u[2] = (T(1) / s2) * b2;
  else o.u[2] = cross3(o.u[0], o.u[1]);
  return o;
}

// Newton projection of S onto prod(S + D) = 1 (5 iterations, CorotateFEMConstraint.h:366-374).
template <typename T>
__device__ __forceinline__ void volume_projection(const T s[3], T g[3]) {
  T D0 = 0, D1 = 0, D2 = 0;
#pragma unroll
  for (int it = 0; it < 5; ++it) {
    T p0 = s[0] + D0, p1 = s[1] + D1, p2 = s[2] + D2;
    T C = p0 * p1 * p2 - T(1);
    T g0 = p1 * p2, g1 = p0 * p2, g2 = p0 * p1;
    T c = (g0 * D0 + g1 * D1 + g2 * D2 - C) / (g0 * g0 + g1 * g1 + g2 * g2);
    D0 = c * g0; D1 = c * g1; D2 = c * g2;
  }
  g[0] = s[0] + D0; g[1] = s[1] + D1; g[2] = s[2] + D2;
}

// Same projection with its derivatives for the adjoint:
//   J[i][k] = d g_i / d s_k (forward mode through the 5 iterations),
//   dd[q]   = (g_i - g_j) / (s_i - s_j) for the pairs (0,1), (0,2), (1,2), computed
//             by the exact recurrence r <- 1 - c * p_k * r (no cancellation, valid
//             for equal singular values too).
template <typename T>
__device__ __forceinline__ void volume_projection_d(const T s[3], T g[3], T J[3][3], T dd[3]) {
  T D[3] = {0, 0, 0};
  T dD[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
  T r0 = 1, r1 = 1, r2 = 1;
#pragma unroll 1
  for (int it = 0; it < 5; ++it) {
    T p[3] = {s[0] + D[0], s[1] + D[1], s[2] + D[2]};
    T C = p[0] * p[1] * p[2] - T(1);
    T gr[3] = {p[1] * p[2], p[0] * p[2], p[0] * p[1]};
    T gg = gr[0] * gr[0] + gr[1] * gr[1] + gr[2] * gr[2];
    T num = gr[0] * D[0] + gr[1] * D[1] + gr[2] * D[2] - C;
    T c = num / gg;
    r0 = T(1) - c * p[2] * r0;
    r1 = T(1) - c * p[1] * r1;
    r2 = T(1) - c * p[0] * r2;
    T nD[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      T dp[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) dp[i] = (i == k ? T(1) : T(0)) + dD[i][k];
      T dC = gr[0] * dp[0] + gr[1] * dp[1] + gr[2] * dp[2];
      T dg0 = dp[1] * p[2] + p[1] * dp[2], dg1 = dp[0] * p[2] + p[0] * dp[2], dg2 = dp[0] * p[1] + p[0] * dp[1];
      T dnum = dg0 * D[0] + dg1 * D[1] + dg2 * D[2] + gr[0] * dD[0][k] + gr[1] * dD[1][k] + gr[2] * dD[2][k] - dC;
      T dgg = T(2) * (gr[0] * dg0 + gr[1] * dg1 + gr[2] * dg2);
      T dc = (dnum * gg - num * dgg) / (gg * gg);
      nD[0][k] = dc * gr[0] + c * dg0;
      nD[1][k] = dc * gr[1] + c * dg1;
      nD[2][k] = dc * gr[2] + c * dg2;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      D[i] = c * gr[i];
#pragma unroll
      for (int k = 0; k < 3; ++k) dD[i][k] = nD[i][k];
    }
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    g[i] = s[i] + D[i];
#pragma unroll
    for (int k = 0; k < 3; ++k) J[i][k] = (i == k ? T(1) : T(0)) + dD[i][k];
  }
  dd[0] = r0; dd[1] = r1; dd[2] = r2;
}

// md (reflected rotation) and md_volume of the corotated constraint, from the
// SVD of F (corot_project computes it; the adjoint shares one SVD between the
// projection and its VJP)
template <typename T>
__device__ __forceinline__ void corot_project_sv(const Svd3<T>& sv, const Mat3<T>& F, Mat3<T>& md, Mat3<T>& mdv,
                                                 T* s_ratio = nullptr) {
  if (s_ratio) {  // smallest / largest singular value (conditioning of the element)
    T smax = sv.s[0] > sv.s[1] ? (sv.s[0] > sv.s[2] ? sv.s[0] : sv.s[2]) : (sv.s[1] > sv.s[2] ? sv.s[1] : sv.s[2]);
    T smin = sv.s[0] < sv.s[1] ? (sv.s[0] < sv.s[2] ? sv.s[0] : sv.s[2]) : (sv.s[1] < sv.s[2] ? sv.s[1] : sv.s[2]);
    *s_ratio = smax > T(0) ? smin / smax : T(0);
  }
  T g[3];
  volume_projection(sv.s, g);
  // R = sum_i u_i v_i^T ; G = sum_i g_i u_i v_i^T   (column j of u v^T is v[j] * u)
  const T vj[3][3] = {{sv.v[0].x, sv.v[1].x, sv.v[2].x}, {sv.v[0].y, sv.v[1].y, sv.v[2].y}, {sv.v[0].z, sv.v[1].z, sv.v[2].z}};
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    md.c[j] = vj[j][0] * sv.u[0] + vj[j][1] * sv.u[1] + vj[j][2] * sv.u[2];
    mdv.c[j] = (g[0] * vj[j][0]) * sv.u[0] + (g[1] * vj[j][1]) * sv.u[1] + (g[2] * vj[j][2]) * sv.u[2];
  }
  if (det3(F) < T(0)) md.c[2] = T(-1) * md.c[2];
}

template <typename T>
__device__ __forceinline__ void corot_project(const Mat3<T>& F, Mat3<T>& md, Mat3<T>& mdv, T* s_ratio = nullptr) {
  const Svd3<T> sv = svd3(F);
  corot_project_sv(sv, F, md, mdv, s_ratio);
}

// ------------------------------------ corotated projection without an SVD ---
//
// The FP64 projection and its VJP need only the polar factor Q = U V^T and
// md_volume = U diag(S + D) V^T, and both have iterations on the 3x3 matrix
// itself (no singular vectors):
//   Q: Newton's iteration X <- (zeta X + X^-T / zeta) / 2 (Higham), X^-T =
//      cof(X) / det(X), from X = F; the scaling zeta = (|X^-T| / |X|)^(1/2)
//      (an FP32 estimate: any positive value keeps U and V) runs while it is
//      far from 1, then the plain iteration converges quadratically.
//   md_volume: with P = F + D = U diag(s + D) V^T the reference's step
//      D_i <- c g_i, g_i = prod_{j != i} (s_j + D_j), is D <- c C with
//      C = sigma cof(P), sigma = sign(det F) (U, V orthogonal with
//      det(U) det(V) = sigma), c = (C : D - (sigma det(P) - 1)) / (C : C): the
//      same five iterates, written in matrix form.
// One division per iteration and short FMA chains: the one-sided Jacobi SVD
// takes two square roots, two divisions and a reciprocal square root per
// rotation, three rotations per sweep, about five sweeps for an element at
// ordinary strain, all dependent.  Elements near a lower rank (|det F| <
// 0.01 (|F|^2/3)^(3/2): X^-T loses digits there) and non-finite ones keep the
// SVD.  Products and sums that feed both the step and its VJP are written
// with explicitly rounded operations, so every kernel that inlines them
// computes the same bits.
__device__ __forceinline__ Vec3<double> rn_cross(Vec3<double> a, Vec3<double> b) {
  return {__fma_rn(a.y, b.z, -__dmul_rn(a.z, b.y)), __fma_rn(a.z, b.x, -__dmul_rn(a.x, b.z)),
          __fma_rn(a.x, b.y, -__dmul_rn(a.y, b.x))};
}
__device__ __forceinline__ double rn_dot(Vec3<double> a, Vec3<double> b) {
  return __fma_rn(a.x, b.x, __fma_rn(a.y, b.y, __dmul_rn(a.z, b.z)));
}
__device__ __forceinline__ double rn_dot(const Mat3<double>& a, const Mat3<double>& b) {
  return __dadd_rn(rn_dot(a.c[0], b.c[0]), __dadd_rn(rn_dot(a.c[1], b.c[1]), rn_dot(a.c[2], b.c[2])));
}
__device__ __forceinline__ Vec3<double> rn_scale(double s, Vec3<double> a) {
  return {__dmul_rn(s, a.x), __dmul_rn(s, a.y), __dmul_rn(s, a.z)};
}
__device__ __forceinline__ Vec3<double> rn_axpy(double s, Vec3<double> a, Vec3<double> b) {  // s a + b
  return {__fma_rn(s, a.x, b.x), __fma_rn(s, a.y, b.y), __fma_rn(s, a.z, b.z)};
}
__device__ __forceinline__ Vec3<double> rn_comb(double a, Vec3<double> u, double b, Vec3<double> v, double c, Vec3<double> w) {
  return rn_axpy(c, w, rn_axpy(b, v, rn_scale(a, u)));  // a u + b v + c w
}
__device__ __forceinline__ Vec3<double> rn_add(Vec3<double> a, Vec3<double> b) {
  return {__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y), __dadd_rn(a.z, b.z)};
}
__device__ __forceinline__ void rn_cof(const Mat3<double>& a, Mat3<double>& c) {  // a^-T det(a)
  c.c[0] = rn_cross(a.c[1], a.c[2]);
  c.c[1] = rn_cross(a.c[2], a.c[0]);
  c.c[2] = rn_cross(a.c[0], a.c[1]);
}

// Polar factor of F (C = cof(F) and det = det(F) given); false when the
// element is near a lower rank (or not finite).
constexpr int kPolarIterations = 16;
__device__ __forceinline__ bool full_rank(const Mat3<double>& F, double det) {
  const double q = __dmul_rn(rn_dot(F, F), 1.0 / 3.0);
  return __dmul_rn(det, det) > __dmul_rn(1e-4, __dmul_rn(q, __dmul_rn(q, q))) && isfinite(det);
}
__device__ __forceinline__ bool polar_newton(const Mat3<double>& F, Mat3<double> C, double det, Mat3<double>& Q) {
  if (!full_rank(F, det)) return false;
  Q = F;
  double d2 = 1.0;
#pragma unroll 1
  for (int it = 0; it < kPolarIterations; ++it) {
    if (it > 0) {
      rn_cof(Q, C);
      det = rn_dot(Q.c[0], C.c[0]);
    }
    const double inv = 1.0 / det;
    double a = 0.5, b = __dmul_rn(0.5, inv);
    bool scaled = false;
    if (d2 > 0.1) {  // the first iteration, and the next ones of a strongly deformed element
      const float fi = (float)inv, r = (float)rn_dot(C, C) * fi * fi / (float)rn_dot(Q, Q);  // (|X^-T| / |X|)^2
      scaled = !(r > 0.8f && r < 1.25f);
      if (scaled) {
        const float z = sqrtf(sqrtf(r));
        a = __dmul_rn(a, (double)z);
        b = __dmul_rn(b, (double)(1.0f / z));
      }
    }
    d2 = 0.0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const Vec3<double> x = rn_axpy(a, Q.c[j], rn_scale(b, C.c[j]));
      const Vec3<double> d = rn_axpy(-1.0, Q.c[j], x);
      d2 = __dadd_rn(d2, rn_dot(d, d));
      Q.c[j] = x;
    }
    if (!scaled && d2 < 1e-17) return true;  // quadratic: the error left is about d2 / 2
  }
  return false;
}

// The five steps of the volume projection.  Its VJP's tape: D before steps
// 1 .. 4 (it is 0 before step 0), c and 1 / (C : C) of every step, in kVolTape
// doubles of shared memory per thread (value q at sh[q * stride]; in registers
// they would spill).
constexpr int kVolTape = 46;
struct VolTape {
  double* sh;
  int stride;
};
__device__ __forceinline__ void tape_store(const VolTape& t, int k, const Mat3<double>& D) {
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    double* o = t.sh + (9 * k + 3 * j) * t.stride;
    o[0] = D.c[j].x; o[t.stride] = D.c[j].y; o[2 * t.stride] = D.c[j].z;
  }
}
__device__ __forceinline__ void tape_load(const VolTape& t, int k, Mat3<double>& D) {
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const double* o = t.sh + (9 * k + 3 * j) * t.stride;
    D.c[j] = mk3(o[0], o[t.stride], o[2 * t.stride]);
  }
}
template <bool TAPE>
__device__ __forceinline__ void volume_newton(const Mat3<double>& F, Mat3<double> C, double det, Mat3<double>& D,
                                              VolTape* tape) {
  const double sg = det < 0.0 ? -1.0 : 1.0;
#pragma unroll
  for (int j = 0; j < 3; ++j) D.c[j] = mk3(0.0, 0.0, 0.0);
#pragma unroll 1
  for (int it = 0; it < 5; ++it) {
    double num = __fma_rn(-sg, det, 1.0);
    if (it > 0) {
      Mat3<double> P;
#pragma unroll
      for (int j = 0; j < 3; ++j) P.c[j] = rn_add(F.c[j], D.c[j]);
      rn_cof(P, C);
      num = __dadd_rn(__fma_rn(-sg, rn_dot(P.c[0], C.c[0]), 1.0), __dmul_rn(sg, rn_dot(C, D)));
    }
    const double iden = 1.0 / rn_dot(C, C), c = __dmul_rn(num, iden), cs = __dmul_rn(sg, c);
    if (TAPE) {
      if (it > 0) tape_store(*tape, it - 1, D);
      tape->sh[(36 + it) * tape->stride] = c;
      tape->sh[(41 + it) * tape->stride] = iden;
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) D.c[j] = rn_scale(cs, C.c[j]);
  }
}

static __device__ __noinline__ void corot_project_svd(const Mat3<double>& F, Mat3<double>& md, Mat3<double>& mdv) {
  corot_project(F, md, mdv);
}

// The two halves of the projection, for kernels that give them to two threads:
// md (reflected rotation) and md_volume of an element.
__device__ __forceinline__ void corot_rotation(const Mat3<double>& F, Mat3<double>& md) {
  Mat3<double> C;
  rn_cof(F, C);
  const double det = rn_dot(F.c[0], C.c[0]);
  if (!polar_newton(F, C, det, md)) {
    Mat3<double> f = F, a, b;
    corot_project_svd(f, a, b);
    md = a;
    return;
  }
  if (det < 0.0) md.c[2] = rn_scale(-1.0, md.c[2]);
}
__device__ __forceinline__ void corot_volume(const Mat3<double>& F, Mat3<double>& mdv) {
  Mat3<double> C, D;
  rn_cof(F, C);
  const double det = rn_dot(F.c[0], C.c[0]);
  if (!full_rank(F, det)) {
    Mat3<double> f = F, a, b;
    corot_project_svd(f, a, b);
    mdv = b;
    return;
  }
  volume_newton<false>(F, C, det, D, nullptr);
#pragma unroll
  for (int j = 0; j < 3; ++j) mdv.c[j] = rn_add(F.c[j], D.c[j]);
}

// md (reflected rotation) and md_volume of an element.
__device__ __forceinline__ void corot_project_polar(const Mat3<double>& F, Mat3<double>& md, Mat3<double>& mdv) {
  Mat3<double> C;
  rn_cof(F, C);
  const double det = rn_dot(F.c[0], C.c[0]);
  if (!polar_newton(F, C, det, md)) {
    Mat3<double> f = F, a, b;  // the call takes addresses: keep the common path's values in registers
    corot_project_svd(f, a, b);
    md = a;
    mdv = b;
    return;
  }
  if (det < 0.0) md.c[2] = rn_scale(-1.0, md.c[2]);
  Mat3<double> D;
  volume_newton<false>(F, C, det, D, nullptr);
#pragma unroll
  for (int j = 0; j < 3; ++j) mdv.c[j] = rn_add(F.c[j], D.c[j]);
}

// Near-degenerate test for the mixed form: an element whose smallest singular
// value is below kDegenerateRatio of its largest (nearly flat or inverted)
// has a badly conditioned U/V in FP32 and is recomputed in FP64.
constexpr float kDegenerateRatio = 0.05f;

// Unit quaternion (w, x, y, z) of a nearly orthogonal matrix with det > 0
// (Shepperd's method: the branch on the largest of trace and diagonal keeps
// the square root away from cancellation).
__device__ __forceinline__ void quat_from_rot(const Mat3<float>& R, float q[4]) {
  const float m00 = R.c[0].x, m11 = R.c[1].y, m22 = R.c[2].z;
  const float m01 = R.c[1].x, m10 = R.c[0].y, m02 = R.c[2].x, m20 = R.c[0].z, m12 = R.c[2].y, m21 = R.c[1].z;
  const float tr = m00 + m11 + m22;
  if (tr > 0.0f) {
    const float S = 2.0f * sqrtf(tr + 1.0f);
    q[0] = 0.25f * S; q[1] = (m21 - m12) / S; q[2] = (m02 - m20) / S; q[3] = (m10 - m01) / S;
  } else if (m00 > m11 && m00 > m22) {
    const float S = 2.0f * sqrtf(fmaxf(1.0f + m00 - m11 - m22, 1e-30f));
    q[0] = (m21 - m12) / S; q[1] = 0.25f * S; q[2] = (m01 + m10) / S; q[3] = (m02 + m20) / S;
  } else if (m11 > m22) {
    const float S = 2.0f * sqrtf(fmaxf(1.0f + m11 - m00 - m22, 1e-30f));
    q[0] = (m02 - m20) / S; q[1] = (m01 + m10) / S; q[2] = 0.25f * S; q[3] = (m12 + m21) / S;
  } else {
    const float S = 2.0f * sqrtf(fmaxf(1.0f + m22 - m00 - m11, 1e-30f));
    q[0] = (m10 - m01) / S; q[1] = (m02 + m20) / S; q[2] = (m12 + m21) / S; q[3] = 0.25f * S;
  }
}

// The rotation of quaternion q, normalised and evaluated in FP64: orthogonal
// to FP64 round-off whatever the FP32 rounding of q.
__device__ __forceinline__ Mat3<double> rot_from_quat(const float qf[4]) {
  double w = qf[0], x = qf[1], y = qf[2], z = qf[3];
  const double n = rsqrt(w * w + x * x + y * y + z * z);
  w *= n; x *= n; y *= n; z *= n;
  Mat3<double> R;
  R.c[0] = mk3(1.0 - 2.0 * (y * y + z * z), 2.0 * (x * y + w * z), 2.0 * (x * z - w * y));
  R.c[1] = mk3(2.0 * (x * y - w * z), 1.0 - 2.0 * (x * x + z * z), 2.0 * (y * z + w * x));
  R.c[2] = mk3(2.0 * (x * z + w * y), 2.0 * (y * z - w * x), 1.0 - 2.0 * (x * x + y * y));
  return R;
}

// The mixed form's FP32 SVD: svd3's method in explicitly rounded operations,
// so that its singular vectors, whose FP32 roundings reach the results, are
// the same bits in every kernel that inlines it (left to itself, the compiler
// fuses products and sums differently from one kernel to the next).
__device__ __forceinline__ float rn_dot(Vec3<float> a, Vec3<float> b) {
  return __fmaf_rn(a.z, b.z, __fmaf_rn(a.x, b.x, __fmul_rn(a.y, b.y)));
}
__device__ __forceinline__ Vec3<float> rn_scale(float s, Vec3<float> a) {
  return {__fmul_rn(s, a.x), __fmul_rn(s, a.y), __fmul_rn(s, a.z)};
}
__device__ __forceinline__ Vec3<float> rn_axpy(float s, Vec3<float> a, Vec3<float> b) {  // s a + b
  return {__fmaf_rn(s, a.x, b.x), __fmaf_rn(s, a.y, b.y), __fmaf_rn(s, a.z, b.z)};
}
__device__ __forceinline__ void jacobi_rotate_f(Vec3<float>& bp, Vec3<float>& bq, Vec3<float>& vp, Vec3<float>& vq,
                                                bool& rotated) {
  const float a = rn_dot(bp, bp), b = rn_dot(bq, bq), g = rn_dot(bp, bq);
  if (!(fabsf(g) > __fmul_rn(Eps<float>::rot, __fsqrt_rn(__fmul_rn(a, b))))) return;
  rotated = true;
  const float zeta = __fdiv_rn(__fsub_rn(b, a), __fmul_rn(2.0f, g));
  const float t = __fdiv_rn(zeta >= 0.0f ? 1.0f : -1.0f, __fadd_rn(fabsf(zeta), __fsqrt_rn(__fmaf_rn(zeta, zeta, 1.0f))));
  const float c = rsqrtf(__fmaf_rn(t, t, 1.0f)), s = __fmul_rn(c, t);
  const Vec3<float> nbp = rn_axpy(c, bp, rn_scale(-s, bq)), nbq = rn_axpy(c, bq, rn_scale(s, bp));
  const Vec3<float> nvp = rn_axpy(c, vp, rn_scale(-s, vq)), nvq = rn_axpy(c, vq, rn_scale(s, vp));
  bp = nbp; bq = nbq; vp = nvp; vq = nvq;
}
__device__ __forceinline__ Svd3<float> svd3_f(const Mat3<float>& F) {
  Svd3<float> o;
  Vec3<float> b0 = F.c[0], b1 = F.c[1], b2 = F.c[2];
  Vec3<float> v0 = mk3(1.0f, 0.0f, 0.0f), v1 = mk3(0.0f, 1.0f, 0.0f), v2 = mk3(0.0f, 0.0f, 1.0f);
#pragma unroll 1
  for (int sweep = 0; sweep < Eps<float>::sweeps; ++sweep) {
    bool rotated = false;
    jacobi_rotate_f(b0, b1, v0, v1, rotated);
    jacobi_rotate_f(b0, b2, v0, v2, rotated);
    jacobi_rotate_f(b1, b2, v1, v2, rotated);
    if (!rotated) break;
  }
  float s0 = __fsqrt_rn(rn_dot(b0, b0)), s1 = __fsqrt_rn(rn_dot(b1, b1)), s2 = __fsqrt_rn(rn_dot(b2, b2));
  auto swap3 = [](float& s, float& t, Vec3<float>& b, Vec3<float>& e, Vec3<float>& v, Vec3<float>& w) {
    if (s < t) { const float q = s; s = t; t = q; Vec3<float> x = b; b = e; e = x; x = v; v = w; w = x; }
  };
  swap3(s0, s1, b0, b1, v0, v1);
  swap3(s0, s2, b0, b2, v0, v2);
  swap3(s1, s2, b1, b2, v1, v2);
  o.s[0] = s0; o.s[1] = s1; o.s[2] = s2;
  o.v[0] = v0; o.v[1] = v1; o.v[2] = v2;
  const float tiny = __fmul_rn(Eps<float>::rel, s0);
  o.u[0] = s0 > 0.0f ? rn_scale(__fdiv_rn(1.0f, s0), b0) : mk3(1.0f, 0.0f, 0.0f);
  if (s1 > tiny) {
    o.u[1] = rn_scale(__fdiv_rn(1.0f, s1), b1);
  } else {  // complete the basis (such an element takes the FP64 branch)
    const Vec3<float> w = cross3(o.u[0], fabsf(o.u[0].x) < 0.9f ? mk3(1.0f, 0.0f, 0.0f) : mk3(0.0f, 1.0f, 0.0f));
    o.u[1] = rsqrtf(rn_dot(w, w)) * w;
  }
  o.u[2] = s2 > tiny ? rn_scale(__fdiv_rn(1.0f, s2), b2) : cross3(o.u[0], o.u[1]);
  return o;
}

// Mixed-form corotated deviations DR = md - F and DV = md_volume - F (columns;
// the tet's J d - L x is G (wr DR + wv DV)).  Only the SVD runs in FP32; its
// error enters the deviations at second order:
//   1. FP32 SVD of F -> R0 = U V^T, its quaternion, and R = R(q) exactly
//      orthogonal in FP64;
//   2. A = R^T F, H = A - I in FP64 (strain-sized; its skew part is only
//      R0's rounding);
//   3. polar of A = (I + Omega) S_A to first order in the tiny skew part, in
//      the V basis: Omega_kl = 2 (V^T skew(H) V)_kl / (s_k + s_l);
//   4. md - F = R (Omega - H);  the volume projection's 5 Newton steps run on
//      e_k = v_k^T sym(H) v_k (= s_k - 1 to second order) with
//      prod(1 + a) - 1 expanded, and md_volume - F = R V diag(D) V^T.
// Steps 2-4 are FP64 arithmetic on the FP32 singular vectors (the one FP32
// rounding of the force is then the caller's store into its slots).
// Returns false (caller takes the full FP64 branch) for inverted or
// near-degenerate elements.
__device__ __forceinline__ bool corot_delta_mixed(const Mat3<double>& F, Vec3<double> DR[3], Vec3<double> DV[3]) {
  Mat3<float> Ff;
#pragma unroll
  for (int j = 0; j < 3; ++j) Ff.c[j] = mk3((float)F.c[j].x, (float)F.c[j].y, (float)F.c[j].z);
  const Svd3<float> sv = svd3_f(Ff);
  const float smax = fmaxf(sv.s[0], fmaxf(sv.s[1], sv.s[2]));
  const float smin = fminf(sv.s[0], fminf(sv.s[1], sv.s[2]));
  if (!(smax > 0.0f) || !(smin >= kDegenerateRatio * smax) || !(det3(F) > 0.0)) return false;
  const float vjf[3][3] = {{sv.v[0].x, sv.v[1].x, sv.v[2].x}, {sv.v[0].y, sv.v[1].y, sv.v[2].y},
                           {sv.v[0].z, sv.v[1].z, sv.v[2].z}};
  Mat3<float> R0;
#pragma unroll
  for (int j = 0; j < 3; ++j) R0.c[j] = rn_axpy(vjf[j][2], sv.u[2], rn_axpy(vjf[j][0], sv.u[0], rn_scale(vjf[j][1], sv.u[1])));
  float q[4];
  quat_from_rot(R0, q);
  const Mat3<double> R = rot_from_quat(q);
  Vec3<double> v[3];  // the FP32 right singular vectors, widened
#pragma unroll
  for (int k = 0; k < 3; ++k) v[k] = mk3((double)sv.v[k].x, (double)sv.v[k].y, (double)sv.v[k].z);
  double H[3][3];  // H[i][j] = (R^T F - I)_ij
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) H[i][j] = dot3(R.c[i], F.c[j]) - (i == j ? 1.0 : 0.0);
  Vec3<double> Hvl[3], HTvl[3];  // H v_l and H^T v_l
#pragma unroll
  for (int l = 0; l < 3; ++l) {
    const Vec3<double> w = v[l];
    Hvl[l] = mk3(H[0][0] * w.x + H[0][1] * w.y + H[0][2] * w.z, H[1][0] * w.x + H[1][1] * w.y + H[1][2] * w.z,
                 H[2][0] * w.x + H[2][1] * w.y + H[2][2] * w.z);
    HTvl[l] = mk3(H[0][0] * w.x + H[1][0] * w.y + H[2][0] * w.z, H[0][1] * w.x + H[1][1] * w.y + H[2][1] * w.z,
                  H[0][2] * w.x + H[1][2] * w.y + H[2][2] * w.z);
  }
  double e[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) e[k] = dot3(v[k], Hvl[k]);  // v^T H v = v^T sym(H) v
  // Omega in the V basis (pairs 01, 02, 12); Omega = sum_{k<l} om_kl (v_k v_l^T - v_l v_k^T)
  const int pk[3] = {0, 0, 1}, pl[3] = {1, 2, 2};
  double om[3];
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    const int k = pk[p], l = pl[p];
    const double kskew = 0.5 * (dot3(v[k], Hvl[l]) - dot3(v[k], HTvl[l]));  // v_k^T skew(H) v_l
    om[p] = 2.0 * kskew / ((double)sv.s[k] + (double)sv.s[l]);
  }
  // volume projection on the small quantities (same iterates as on s + D)
  double D[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int it = 0; it < 5; ++it) {
    const double a0 = e[0] + D[0], a1 = e[1] + D[1], a2 = e[2] + D[2];
    const double C = (a0 + a1 + a2) + (a0 * a1 + a0 * a2 + a1 * a2) + a0 * a1 * a2;
    const double g0 = 1.0 + a1 + a2 + a1 * a2, g1 = 1.0 + a0 + a2 + a0 * a2, g2 = 1.0 + a0 + a1 + a0 * a1;
    const double c = (g0 * D[0] + g1 * D[1] + g2 * D[2] - C) / (g0 * g0 + g1 * g1 + g2 * g2);
    D[0] = c * g0; D[1] = c * g1; D[2] = c * g2;
  }
  // md - F = R (Omega - H), md_volume - F = R V diag(D) V^T
  const double vj[3][3] = {{v[0].x, v[1].x, v[2].x}, {v[0].y, v[1].y, v[2].y}, {v[0].z, v[1].z, v[2].z}};
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    Vec3<double> col = mk3(-H[0][j], -H[1][j], -H[2][j]);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const int k = pk[p], l = pl[p];
      col = col + (om[p] * vj[j][l]) * v[k] - (om[p] * vj[j][k]) * v[l];
    }
    const Vec3<double> vol = (D[0] * vj[j][0]) * v[0] + (D[1] * vj[j][1]) * v[1] + (D[2] * vj[j][2]) * v[2];
    DR[j] = col.x * R.c[0] + col.y * R.c[1] + col.z * R.c[2];
    DV[j] = vol.x * R.c[0] + vol.y * R.c[1] + vol.z * R.c[2];
  }
  return true;
}

// Mixed-form corotated force P = wr (md - F) + wv (md_volume - F) (columns).
__device__ __forceinline__ bool corot_force_mixed(const Mat3<double>& F, double wr, double wv, Vec3<double> P[3]) {
  Vec3<double> DR[3], DV[3];
  if (!corot_delta_mixed(F, DR, DV)) return false;
#pragma unroll
  for (int j = 0; j < 3; ++j) P[j] = wr * DR[j] + wv * DV[j];
  return true;
}

// VJP of (md, md_volume) with respect to F.  gmd, gmdv: cotangents (3x3).
//   P_bar_ij (i != j) = a_ij sym(M_G)_ij + b_ij asym(M_G)_ij + (M_R_ij - M_R_ji)/(s_i + s_j)
//   P_bar_ii = sum_k (M_G)_kk dg_k/ds_i
//   with M_X = U^T X V, a_ij = (g_i - g_j)/(s_i - s_j), b_ij = (g_i + g_j)/(s_i + s_j);
//   F_bar = U P_bar V^T.
template <typename T>
__device__ __forceinline__ Mat3<T> corot_vjp_sv(const Svd3<T>& sv, const Mat3<T>& F, Mat3<T> gmd,
                                                const Mat3<T>& gmdv) {
  T g[3], J[3][3], dd[3];
  volume_projection_d(sv.s, g, J, dd);
  if (det3(F) < T(0)) gmd.c[2] = T(-1) * gmd.c[2];
  // M = U^T X V : M_ij = u_i . (X v_j) ; X v_j = sum_k X.c[k] * v_j[k]
  T MR[3][3], MG[3][3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    Vec3<T> xr = sv.v[j].x * gmd.c[0] + sv.v[j].y * gmd.c[1] + sv.v[j].z * gmd.c[2];
    Vec3<T> xg = sv.v[j].x * gmdv.c[0] + sv.v[j].y * gmdv.c[1] + sv.v[j].z * gmdv.c[2];
#pragma unroll
    for (int i = 0; i < 3; ++i) { MR[i][j] = dot3(sv.u[i], xr); MG[i][j] = dot3(sv.u[i], xg); }
  }
  T P[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
    P[i][i] = MG[0][0] * J[0][i] + MG[1][1] * J[1][i] + MG[2][2] * J[2][i];
  const int pi[3] = {0, 0, 1}, pj[3] = {1, 2, 2};
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    int i = pi[q], j = pj[q];
    T ssum = sv.s[i] + sv.s[j];
    T b = (g[i] + g[j]) / ssum;
    T a = dd[q];
    T symG = T(0.5) * (MG[i][j] + MG[j][i]);
    T asymG = T(0.5) * (MG[i][j] - MG[j][i]);
    T asymR = (MR[i][j] - MR[j][i]) / ssum;
    P[i][j] = a * symG + b * asymG + asymR;
    P[j][i] = a * symG - b * asymG - asymR;
  }
  // F_bar = U P V^T : column c = sum_{i,j} P_ij u_i v_j[c]
  Mat3<T> out;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const T vc[3] = {c == 0 ? sv.v[0].x : (c == 1 ? sv.v[0].y : sv.v[0].z),
                     c == 0 ? sv.v[1].x : (c == 1 ? sv.v[1].y : sv.v[1].z),
                     c == 0 ? sv.v[2].x : (c == 1 ? sv.v[2].y : sv.v[2].z)};
    Vec3<T> acc = mk3<T>(0, 0, 0);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      T w = P[i][0] * vc[0] + P[i][1] * vc[1] + P[i][2] * vc[2];
      acc = acc + w * sv.u[i];
    }
    out.c[c] = acc;
  }
  return out;
}

template <typename T>
__device__ __forceinline__ Mat3<T> corot_vjp(const Mat3<T>& F, Mat3<T> gmd, const Mat3<T>& gmdv) {
  const Svd3<T> sv = svd3(F);
  return corot_vjp_sv(sv, F, gmd, gmdv);
}

static __device__ __noinline__ void corot_adjoint_svd(const Mat3<double>& F, const Mat3<double>& Y, double wr, double wv,
                                               double& yr, double& yv, Mat3<double>& gF) {
  Mat3<double> md, mdv, gmd, gmdv;
  const Svd3<double> sv = svd3(F);  // one SVD for the projection and its VJP
  corot_project_sv(sv, F, md, mdv);
  yr = yv = 0.0;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    yr += dot3(Y.c[j], md.c[j]);
    yv += dot3(Y.c[j], mdv.c[j]);
    gmd.c[j] = wr * Y.c[j];
    gmdv.c[j] = wv * Y.c[j];
  }
  gF = corot_vjp_sv(sv, F, gmd, gmdv);
}

// Adjoint of an element: yr = Y : md, yv = Y : md_volume and the VJP
// gF = (d md / dF)^T (wr Y) + (d md_volume / dF)^T (wv Y).
//   polar factor F = Q S: dQ = Q [w]x, (tr(S) I - S) w = ax(Q^T dF), so with
//   b = ax(Q^T gQ) and z = (tr(S) I - S)^-1 b its VJP is Q [z]x;
//   volume steps in reverse, D' = c C, c = num / (C : C):
//     gc = gD' : C,  gC = c gD' + gc / (C : C) (D - 2 c C),
//     gP = sigma cofT(P, gC) - gc / (C : C) C,  gD = gc / (C : C) C + gP, gF += gP.
__device__ __forceinline__ void rotation_vjp(const Mat3<double>& F, const Mat3<double>& Q, double sg, const Mat3<double>& Y,
                                             double wr, double& yr, Mat3<double>& gF) {
  const Vec3<double> g2 = rn_scale(sg, Y.c[2]);  // md's column 2 is sigma times Q's
  yr = __dadd_rn(rn_dot(Y.c[0], Q.c[0]), __dadd_rn(rn_dot(Y.c[1], Q.c[1]), rn_dot(g2, Q.c[2])));
  const double b0 = __dadd_rn(rn_dot(Q.c[2], Y.c[1]), -rn_dot(Q.c[1], g2));
  const double b1 = __dadd_rn(rn_dot(Q.c[0], g2), -rn_dot(Q.c[2], Y.c[0]));
  const double b2 = __dadd_rn(rn_dot(Q.c[1], Y.c[0]), -rn_dot(Q.c[0], Y.c[1]));
  const double s00 = rn_dot(Q.c[0], F.c[0]), s11 = rn_dot(Q.c[1], F.c[1]), s22 = rn_dot(Q.c[2], F.c[2]);
  const double k01 = __dmul_rn(-0.5, __dadd_rn(rn_dot(Q.c[0], F.c[1]), rn_dot(Q.c[1], F.c[0])));
  const double k02 = __dmul_rn(-0.5, __dadd_rn(rn_dot(Q.c[0], F.c[2]), rn_dot(Q.c[2], F.c[0])));
  const double k12 = __dmul_rn(-0.5, __dadd_rn(rn_dot(Q.c[1], F.c[2]), rn_dot(Q.c[2], F.c[1])));
  const double k00 = __dadd_rn(s11, s22), k11 = __dadd_rn(s00, s22), k22 = __dadd_rn(s00, s11);
  // the symmetric 3x3 system by its cofactors
  const double a00 = __fma_rn(k11, k22, -__dmul_rn(k12, k12)), a01 = __fma_rn(k02, k12, -__dmul_rn(k01, k22));
  const double a02 = __fma_rn(k01, k12, -__dmul_rn(k02, k11)), a11 = __fma_rn(k00, k22, -__dmul_rn(k02, k02));
  const double a12 = __fma_rn(k01, k02, -__dmul_rn(k00, k12)), a22 = __fma_rn(k00, k11, -__dmul_rn(k01, k01));
  const double w = wr / rn_dot(mk3(k00, k01, k02), mk3(a00, a01, a02));
  const Vec3<double> b = mk3(b0, b1, b2);
  const double z0 = __dmul_rn(w, rn_dot(mk3(a00, a01, a02), b)), z1 = __dmul_rn(w, rn_dot(mk3(a01, a11, a12), b)),
               z2 = __dmul_rn(w, rn_dot(mk3(a02, a12, a22), b));
  gF.c[0] = rn_axpy(z2, Q.c[1], rn_scale(-z1, Q.c[2]));
  gF.c[1] = rn_axpy(z0, Q.c[2], rn_scale(-z2, Q.c[0]));
  gF.c[2] = rn_axpy(z1, Q.c[0], rn_scale(-z0, Q.c[1]));
}

// gF: the volume part of the VJP alone.
__device__ __forceinline__ void volume_vjp(const Mat3<double>& F, const Mat3<double>& C0, double det, const Mat3<double>& Y,
                                           double wv, double& yv, Mat3<double>& gF, double* tape_sh, int stride) {
  const double sg = det < 0.0 ? -1.0 : 1.0;
  Mat3<double> C, gD;
  VolTape tape;
  tape.sh = tape_sh;
  tape.stride = stride;
  {
    Mat3<double> D;
    volume_newton<true>(F, C0, det, D, &tape);
    yv = 0.0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      yv = __dadd_rn(yv, rn_dot(Y.c[j], rn_add(F.c[j], D.c[j])));
      gD.c[j] = rn_scale(wv, Y.c[j]);
      gF.c[j] = gD.c[j];
    }
  }
#pragma unroll 1
  for (int it = 4; it >= 0; --it) {
    Mat3<double> P, D, gC;
    if (it > 0) {
      tape_load(tape, it - 1, D);
    } else {
#pragma unroll
      for (int j = 0; j < 3; ++j) D.c[j] = mk3(0.0, 0.0, 0.0);
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) P.c[j] = rn_add(F.c[j], D.c[j]);
    rn_cof(P, C);  // sigma times the step's C
    const double c = tape.sh[(36 + it) * stride], gn = __dmul_rn(__dmul_rn(sg, rn_dot(gD, C)), tape.sh[(41 + it) * stride]);
    const double sn = __dmul_rn(sg, gn);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      gC.c[j] = rn_axpy(c, gD.c[j], rn_scale(__dmul_rn(-2.0, __dmul_rn(sn, c)), C.c[j]));
      gC.c[j] = rn_scale(sg, rn_axpy(gn, D.c[j], gC.c[j]));
    }
    Mat3<double> gP;
    gP.c[0] = rn_add(rn_cross(P.c[1], gC.c[2]), rn_cross(gC.c[1], P.c[2]));
    gP.c[1] = rn_add(rn_cross(P.c[2], gC.c[0]), rn_cross(gC.c[2], P.c[0]));
    gP.c[2] = rn_add(rn_cross(P.c[0], gC.c[1]), rn_cross(gC.c[0], P.c[1]));
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const Vec3<double> nc = rn_scale(sn, C.c[j]);  // gc / (C : C) times the step's C
      const Vec3<double> g = rn_axpy(-1.0, nc, gP.c[j]);
      gF.c[j] = rn_add(gF.c[j], g);
      gD.c[j] = rn_add(nc, g);
    }
  }
}

// The two halves for two threads: gF of each (the element's is their sum).
__device__ __forceinline__ void corot_adjoint_rotation(const Mat3<double>& F, const Mat3<double>& Y, double wr, double& yr,
                                                       Mat3<double>& gF) {
  Mat3<double> C, Q;
  rn_cof(F, C);
  const double det = rn_dot(F.c[0], C.c[0]);
  if (!polar_newton(F, C, det, Q)) {
    Mat3<double> f = F, y = Y, g;
    double a, b;
    corot_adjoint_svd(f, y, wr, 0.0, a, b, g);
    yr = a;
    gF = g;
    return;
  }
  rotation_vjp(F, Q, det < 0.0 ? -1.0 : 1.0, Y, wr, yr, gF);
}
__device__ __forceinline__ void corot_adjoint_volume(const Mat3<double>& F, const Mat3<double>& Y, double wv, double& yv,
                                                     Mat3<double>& gF, double* tape_sh, int stride) {
  Mat3<double> C;
  rn_cof(F, C);
  const double det = rn_dot(F.c[0], C.c[0]);
  if (!full_rank(F, det)) {
    Mat3<double> f = F, y = Y, g;
    double a, b;
    corot_adjoint_svd(f, y, 0.0, wv, a, b, g);
    yv = b;
    gF = g;
    return;
  }
  volume_vjp(F, C, det, Y, wv, yv, gF, tape_sh, stride);
}

// Both (an element near a lower rank takes the SVD's VJP once for each half,
// as two threads do).
__device__ __forceinline__ void corot_adjoint_polar(const Mat3<double>& F, const Mat3<double>& Y, double wr, double wv,
                                                    double& yr, double& yv, Mat3<double>& gF, double* tape_sh,
                                                    int stride) {
  Mat3<double> gV;
  corot_adjoint_rotation(F, Y, wr, yr, gF);
  corot_adjoint_volume(F, Y, wv, yv, gV, tape_sh, stride);
#pragma unroll
  for (int j = 0; j < 3; ++j) gF.c[j] = rn_add(gF.c[j], gV.c[j]);
}

}  // namespace dfem
