// elem.cu -- element residual + tangent (calc_r_K's element loop) and the
// element kernels of the batched rounds.
//
// Reference: src/analysis/FiniteElement.jl:75-200 (calc_r_K), :208-242
// (calc_elem_residual), :253-330 (calc_elem_dof_residuals), :338-400
// (calc_bdry_element_residual), :431-452 (calc_τ_ν); GP kinematics and
// stresses from src/analysis/GeoDynStress.jl:91-178.
//
// The reference differentiates the element residual by complex steps, one
// residual evaluation per active element dof (FiniteElement.jl:109-126).  Here
// the same derivative is formed at the Gauss points.  A residual row of node b
// is linear in node b's basis values, r_(b,i) = sum_s phi_s[b] c_(i,s) with
// phi = (N_,1, N_,2, nn_11, nn_22, nn_12, N), nn the covariant second
// derivatives, and the coefficients c depend on
// the unknowns only through the fields' interpolants sum_a phi_t[a] u_a.  So
// the element tangent is
//   K_(b,i),(a,f) = sum_points sum_s sum_t phi_s[b] D_(i,s),(f,t) phi_t[a],
// with D = dc / d(interpolant t of field f): at most 29 directions (field,
// interpolant) per point instead of the element's 72 dofs.  Mesh-motion fields
// carry the node positions with them, dx = dt du, which is the reference's two
// complex steps of one column merged by linearity (FiniteElement.jl:113-122).
// The derivative of |τ| is dropped in the boundary term, exactly as the
// reference's conjugating `dot` drops it (FiniteElement.jl:448).
//
// One to four elements per CTA (elem_body), in phases:
//   0  nodes, Gauss-point tables; the interpolants of every point;
//   1  the primal values of every point, one thread per point, kept in shared
//      memory (each is needed by every direction; formed once);
//   2  D, one lane per direction and one warp per point (two points per warp
//      in the Lagrangian motion's 16 directions): forward-mode derivatives on
//      the stored primal values;
//   3  the two contractions: a thread owns one (row field i, column (a, f))
//      pair, forms W_s = sum_t D_(i,s),(f,t) phi_t[a] and adds sum_s phi_s[b]
//      W_s to its nine rows b, kept in registers over the points;
//   4  the block through shared memory to K_el[e][col][row], coalesced.
// What bounds it: FP64 issue in the plain form (one warp-wide FP64 instruction
// per 64 cycles and sub-partition), FP32 issue and shared-memory reads in the
// FP32 form.  Work per ALEVB element: 9 x ~400 warp instructions in phase 2
// and 9 x ~700 in phase 3, against 72 x 9 dual residual evaluations of ~2400
// (FP64) when every element dof is a direction of its own.
// Measured on a GB300, against one dual residual evaluation per dof: assembly
// with its gathers (mafem_calc_r_K) in FP64 3.16 -> 0.78 ms on 32 x 32 ALEVB,
// 0.58 -> 0.09 ms on 8 x 8 LAG; the FP32 tangent of 32 x 32 ALEVB alone
// 171 -> 72 us.
//
// Two precisions.  The plain FP64 form evaluates everything in FP64 and takes
// the residual from the primal values.  The FP32 form splits the work by pipe:
// the tangent in FP32 (inputs converted once per element), and the residual
// alone in FP64 by elem_resid_kernel, one thread per (element, Gauss point).
// The residual's summation order (Gauss points 0..8, the Dohrmann-Bochev term,
// then the Neumann points) is the same in both.
//
// A second kernel (assemble.cu) gathers, for every band entry, the <= 9 element
// contributions that land on it.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "batch_common.cuh"
#include "mafem_internal.h"

namespace mafem {

// ---- dual numbers ------------------------------------------------------------
// primal P, tangent T (Nil: primal only)
struct Nil {
  __device__ __forceinline__ Nil() {}
  __device__ __forceinline__ explicit Nil(double) {}
  __device__ __forceinline__ explicit Nil(float) {}
  __device__ __forceinline__ explicit Nil(int) {}
};
__device__ __forceinline__ Nil operator+(Nil, Nil) { return Nil(); }
__device__ __forceinline__ Nil operator-(Nil, Nil) { return Nil(); }
__device__ __forceinline__ Nil operator-(Nil) { return Nil(); }
__device__ __forceinline__ Nil operator*(Nil, Nil) { return Nil(); }

template <class P, class T>
struct Dual {
  P v;
  T d;
};
template <class P, class T>
__device__ __forceinline__ Dual<P, T> mk(P v, T d) { return Dual<P, T>{v, d}; }
template <class P, class T>
__device__ __forceinline__ Dual<P, T> cst(P v) { return Dual<P, T>{v, T(0.0)}; }
template <class P, class T>
__device__ __forceinline__ Dual<P, T> operator+(Dual<P, T> a, Dual<P, T> b) { return {a.v + b.v, a.d + b.d}; }
template <class P, class T>
__device__ __forceinline__ Dual<P, T> operator-(Dual<P, T> a, Dual<P, T> b) { return {a.v - b.v, a.d - b.d}; }
template <class P, class T>
__device__ __forceinline__ Dual<P, T> operator-(Dual<P, T> a) { return {-a.v, -a.d}; }
template <class P, class T>
__device__ __forceinline__ Dual<P, T> operator*(Dual<P, T> a, Dual<P, T> b) {
  return {a.v * b.v, a.d * T(b.v) + T(a.v) * b.d};
}
// scalars are converted to the primal type (constants fold at compile time;
// runtime parameters are converted once, in Coef)
template <class P, class T>
__device__ __forceinline__ Dual<P, T> operator*(Dual<P, T> a, P c) { return {a.v * c, a.d * T(c)}; }
template <class P, class T>
__device__ __forceinline__ Dual<P, T> operator*(P c, Dual<P, T> a) { return {a.v * c, a.d * T(c)}; }
template <class P, class T>
__device__ __forceinline__ Dual<P, T> operator+(Dual<P, T> a, P c) { return {a.v + c, a.d}; }
template <class P, class T>
__device__ __forceinline__ Dual<P, T> operator-(Dual<P, T> a, P c) { return {a.v - c, a.d}; }
template <class P, class T>
__device__ __forceinline__ Dual<P, T> inv(Dual<P, T> a) {
  P r = P(1) / a.v;
  return {r, -a.d * T(r * r)};
}
template <class P, class T>
__device__ __forceinline__ Dual<P, T> dsqrt(Dual<P, T> a) {
  P s = sqrt(a.v);
  return {s, a.d * T(P(0.5) / s)};
}

// material coefficients in the primal type (PhysParams holds doubles)
template <class P>
struct Coef {
  P kb, kg, zv, pn, adb_zv, am;
  __device__ __forceinline__ explicit Coef(const PhysParams& pp)
      : kb(P(pp.kb)), kg(P(pp.kg)), zv(P(pp.zv)), pn(P(pp.pn)), adb_zv(P(pp.adb / pp.zv)), am(P(pp.am)) {}
};

// Primal values of one (element, area Gauss point) formed from the nodes: a_α
// and x_,αβ (sums over the 9 nodes of the mesh positions) and the interpolants
// of the 8 unknowns -- u N for u = 0..7, u N_,1 and u N_,2 for u = 0..5 (zero
// for an unknown the motion lacks).
constexpr int kPreA = 0, kPreX = 6, kPreN = 15, kPreD0 = 23, kPreD1 = 29, kPre = 35;
template <class P>
__device__ __forceinline__ P gp_pre_value(int j, const PhysParams& pp, const P* X, const P* C, const P* f) {
  const P* wts;
  const P* src;
  int stride;
  if (j < kPreX) {  // a[i][α] = sum_b N_,α[b] x[b][i]
    wts = f + 10 + 9 * (j & 1);
    src = X + (j >> 1);
    stride = 3;
  } else if (j < kPreN) {  // xab[i][k] = sum_b N_,k[b] x[b][i]
    const int i = (j - kPreX) / 3, k = j - kPreX - 3 * i;
    wts = f + 28 + 9 * k;
    src = X + i;
    stride = 3;
  } else {
    const int u = j < kPreD0 ? j - kPreN : j < kPreD1 ? j - kPreD0 : j - kPreD1;
    const int d = pp.dof_of[u];
    if (d < 0) return P(0);  // get_dof_cps zero-fills absent unknowns (GeoDynStress.jl:190-205)
    wts = f + (j < kPreD0 ? 1 : j < kPreD1 ? 10 : 19);
    src = C + d;
    stride = 8;
  }
  P s = 0;
#pragma unroll
  for (int b = 0; b < 9; ++b) s += wts[b] * src[b * stride];
  return s;
}

// ---- one Gauss point ---------------------------------------------------------------
// motion is a template parameter; the dof maps are runtime (PhysParams).
enum { STATIC_ = 1, EUL_ = 2, LAG_ = 3, ALEV_ = 4, ALEVB_ = 5 };
// basis kinds t (and s): N_,1, N_,2, nn_11, nn_22, nn_12, N
constexpr int kN = 5;

// A direction of differentiation at a point: interpolant t of one field.
// comp: its vector component; v, m, l, p: which field; geo: the field moves the
// mesh (component comp), so the positions follow with dt.
template <class T>
struct Seed {
  int comp, t;
  bool v, m, l, p, geo;
  T dt;
  __device__ __forceinline__ T x(int i, int k) const { return (geo && comp == i && t == k) ? dt : T(0); }
  __device__ __forceinline__ T vel(int i, int k) const { return (v && comp == i && t == k) ? T(1) : T(0); }
  __device__ __forceinline__ T mesh(int i, int k) const { return (m && comp == i && t == k) ? T(1) : T(0); }
  __device__ __forceinline__ T lam() const { return l ? T(1) : T(0); }
  __device__ __forceinline__ T pres() const { return p ? T(1) : T(0); }
};
template <>
struct Seed<Nil> {
  __device__ __forceinline__ Nil x(int, int) const { return Nil(); }
  __device__ __forceinline__ Nil vel(int, int) const { return Nil(); }
  __device__ __forceinline__ Nil mesh(int, int) const { return Nil(); }
  __device__ __forceinline__ Nil lam() const { return Nil(); }
  __device__ __forceinline__ Nil pres() const { return Nil(); }
};

// What happens to the primal value of a named intermediate: kept as computed,
// stored for the tangent pass, or (tangent pass) read back -- the compiler then
// drops its computation.  The index follows the order of evaluation.
struct Keep {
  template <class D>
  __device__ __forceinline__ void operator()(D&) {}
};
template <class P>
struct Store {
  P* p;
  int id;
  __device__ __forceinline__ void operator()(Dual<P, Nil>& x) { p[id++] = x.v; }
};
template <class P>
struct Load {
  const P* p;
  int id;
  template <class T>
  __device__ __forceinline__ void operator()(Dual<P, T>& x) { x.v = p[id++]; }
};
constexpr int kNamed = 74;              // named intermediates of gp_eval at most (ALE, ALEVB)
constexpr int kPreGam = kPre + 14;     // where Γ^1_k, Γ^2_k, b_k (k = 11, 22, 12) stand in the table
constexpr int kPrim = kPre + kNamed;   // table stride per point (odd: conflict-free over points)

// One area Gauss point: calc_elem_dof_residuals' GP body (FiniteElement.jl:284-321)
// with geo_dyn_stress (GeoDynStress.jl:91-178) inlined, on dual numbers.  The
// residual rows (node-major packing of calc_elem_residual, FiniteElement.jl:
// 225-239) are linear in the node's basis values -- with the covariant second
// derivatives nn_k = N_,k - Γ^α_k N_,α,
//   r_v,i = (a_i,1 S1 + a_i,2 S3) N_,1 + (a_i,1 S3 + a_i,2 S2) N_,2
//           + n_i M_k J w nn_k - n_i pn J w N,     S = (σ11, σ22, σ12) J w,
// and likewise for the mesh, pressure and λ rows -- and `out` receives each
// row's coefficients of (N_,1, N_,2, nn_11, nn_22, nn_12, N): v(i, c[6], Gam),
// m6(i, c[6], Gam) / m3(i, c of N_,1, N_,2, N) / m1(i, c of N), p(c of N), l(c of N).
//
// The directions use the same covariant basis: a position direction t = γ < 2
// moves a_γ by e_j and x_,k by Γ^γ_k e_j, one with t = 2 + k moves x_,k alone,
// with weights N_,γ and nn_k of the node.  The derivatives of the geometry are
// then closed forms without cancellation,
//   ∂a^αβ = -(a^α_j a^γβ + a^αγ a^β_j), ∂n = -n_j a^γ, ∂J = J a^γ_j,
//   ∂a^α = a^αγ n_j n - a^α_j a^γ, ∂b_k = 0, ∂Γ^α_k = a^αγ n_j b_k    (t = γ),
//   ∂b_k = n_j, ∂Γ^α_k = a^α_j, nothing else                       (t = 2 + k)
// where N_,k-based directions would leave differences of terms of the size of
// the parametrisation's Γ N_,α to the rounding.  The row coefficients of N_,α
// carry the change of nn_k: -n_i M_k J w ∂Γ^α_k.
template <class P, class T, int MOTION, class Named, class Out>
__device__ __forceinline__ void gp_eval(const Coef<P>& cf, const P* pre, const P w, const Seed<T>& sd, Named nm,
                                        Out& out) {
  using D = Dual<P, T>;
  constexpr bool kTan = !std::is_same<T, Nil>::value;
  auto val = [](P v) { return cst<P, T>(v); };
  // geometry: a_α, x_,αβ (x itself is not used by the residual)
  D a[3][2];
  P xab[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    a[i][0] = mk<P, T>(pre[kPreA + 2 * i], sd.x(i, 0));
    a[i][1] = mk<P, T>(pre[kPreA + 2 * i + 1], sd.x(i, 1));
#pragma unroll
    for (int k = 0; k < 3; ++k) xab[i][k] = pre[kPreX + 3 * i + k];
  }
  D J, i11, i12, i22, aup[3][2], n[3], bf[3];
  P Gam[3][2];
  {
    auto dot = [&](int k, int l) { return a[0][k].v * a[0][l].v + a[1][k].v * a[1][l].v + a[2][k].v * a[2][l].v; };
    const P a11 = dot(0, 0), a12 = dot(0, 1), a22 = dot(1, 1);
    const P det = a11 * a22 - a12 * a12;
    D idet = val(P(1) / det);
    nm(idet);
    J = val(sqrt(det));
    nm(J);
    const P iJ = P(1) / J.v;
    i11 = val(a22 * idet.v), i12 = val(-(a12 * idet.v)), i22 = val(a11 * idet.v);  // a^αβ
    nm(i11), nm(i12), nm(i22);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      aup[i][0] = val(a[i][0].v * i11.v + a[i][1].v * i12.v);
      aup[i][1] = val(a[i][0].v * i12.v + a[i][1].v * i22.v);
      nm(aup[i][0]), nm(aup[i][1]);
    }
    n[0] = val((a[1][0].v * a[2][1].v - a[2][0].v * a[1][1].v) * iJ);
    n[1] = val((a[2][0].v * a[0][1].v - a[0][0].v * a[2][1].v) * iJ);
    n[2] = val((a[0][0].v * a[1][1].v - a[1][0].v * a[0][1].v) * iJ);
    nm(n[0]), nm(n[1]), nm(n[2]);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      D g0 = val(xab[0][k] * aup[0][0].v + xab[1][k] * aup[1][0].v + xab[2][k] * aup[2][0].v);
      D g1 = val(xab[0][k] * aup[0][1].v + xab[1][k] * aup[1][1].v + xab[2][k] * aup[2][1].v);
      bf[k] = val(xab[0][k] * n[0].v + xab[1][k] * n[1].v + xab[2][k] * n[2].v);
      nm(g0), nm(g1), nm(bf[k]);
      Gam[k][0] = g0.v;
      Gam[k][1] = g1.v;
    }
  }
  // the direction's scalars: a^α_j and n_j (0 unless it moves the mesh), a^αγ
  [[maybe_unused]] T u0{}, u1{}, nj{}, ig0{}, ig1{};
  if constexpr (kTan) {
    const bool g1 = sd.t == 1;
    const T gj = sd.geo ? sd.dt : T(0);
    u0 = gj * T(sd.comp == 0 ? aup[0][0].v : sd.comp == 1 ? aup[1][0].v : aup[2][0].v);
    u1 = gj * T(sd.comp == 0 ? aup[0][1].v : sd.comp == 1 ? aup[1][1].v : aup[2][1].v);
    nj = gj * T(sd.comp == 0 ? n[0].v : sd.comp == 1 ? n[1].v : n[2].v);
    const T fa = sd.t < 2 ? T(1) : T(0);  // moves a_γ
    const T v0 = fa * u0, v1 = fa * u1, vn = fa * nj;
    ig0 = T(g1 ? i12.v : i11.v);  // a^0γ
    ig1 = T(g1 ? i22.v : i12.v);  // a^1γ
    i11.d = T(-2) * v0 * ig0;
    i12.d = -(v0 * ig1 + ig0 * v1);
    i22.d = T(-2) * v1 * ig1;
    J.d = T(J.v) * (g1 ? v1 : v0);
    const T p0 = ig0 * vn, p1 = ig1 * vn;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const T ag = T(g1 ? aup[i][1].v : aup[i][0].v);  // a^γ_i
      aup[i][0].d = p0 * T(n[i].v) - v0 * ag;
      aup[i][1].d = p1 * T(n[i].v) - v1 * ag;
      n[i].d = -(vn * ag);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) bf[k].d = sd.t == 2 + k ? nj : T(0);
  }
  // b^αβ = a⁻¹ b a⁻¹ (symmetric)
  D t11 = i11 * bf[0] + i12 * bf[2], t12 = i11 * bf[2] + i12 * bf[1];
  D t21 = i12 * bf[0] + i22 * bf[2], t22 = i12 * bf[2] + i22 * bf[1];
  nm(t11), nm(t12), nm(t21), nm(t22);
  D bu11 = t11 * i11 + t12 * i12, bu12 = t11 * i12 + t12 * i22, bu22 = t21 * i12 + t22 * i22;
  nm(bu11), nm(bu12), nm(bu22);
  D H = (t11 + t22) * P(0.5);  // tr(a⁻¹ b) / 2
  nm(H);
  // K = det b / det a, as a determinant of the mixed components
  D K = t11 * t22 - t12 * t21;

  // dynamics
  D dv[3][2];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    dv[i][0] = mk<P, T>(pre[kPreD0 + i], sd.vel(i, 0));
    dv[i][1] = mk<P, T>(pre[kPreD1 + i], sd.vel(i, 1));
  }
  D lam = mk<P, T>(pre[kPreN + 6], sd.lam());

  // π^αβ = ζv sym(a^αᵀ v_,α a⁻¹)  (GeoDynStress.jl:148-149)
  auto visc = [&](const D (&g)[3][2], D& p11, D& p12, D& p22) {
    D u[3][2];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      u[i][0] = g[i][0] * i11 + g[i][1] * i12;
      u[i][1] = g[i][0] * i12 + g[i][1] * i22;
      nm(u[i][0]), nm(u[i][1]);
    }
    D P11 = aup[0][0] * u[0][0] + aup[1][0] * u[1][0] + aup[2][0] * u[2][0];
    D P12 = aup[0][0] * u[0][1] + aup[1][0] * u[1][1] + aup[2][0] * u[2][1];
    D P21 = aup[0][1] * u[0][0] + aup[1][1] * u[1][0] + aup[2][1] * u[2][0];
    D P22 = aup[0][1] * u[0][1] + aup[1][1] * u[1][1] + aup[2][1] * u[2][1];
    p11 = (P11 + P11) * cf.zv;
    p12 = (P12 + P21) * cf.zv;
    p22 = (P22 + P22) * cf.zv;
  };
  D p11, p12, p22;
  visc(dv, p11, p12, p22);
  // tr(a^αᵀ v_,α) for rλ (FiniteElement.jl:298)
  D tr = aup[0][0] * dv[0][0] + aup[1][0] * dv[1][0] + aup[2][0] * dv[2][0] + aup[0][1] * dv[0][1] +
         aup[1][1] * dv[1][1] + aup[2][1] * dv[2][1];
  nm(tr);
  // σ, M in Voigt form (GeoDynStress.jl:150-154)
  D cb = cf.kb * (H * H) - cf.kg * K;
  D cs = cb + lam;
  D hb = H * (P(2) * cf.kb);
  nm(cb), nm(cs), nm(hb);
  D sg0 = i11 * cs - bu11 * hb + p11;
  D sg1 = i22 * cs - bu22 * hb + p22;
  D sg2 = i12 * cs - bu12 * hb + p12;
  D hm = H * (cf.kb + P(2) * cf.kg);
  nm(hm);
  D M0 = i11 * hm - bu11 * cf.kg;
  D M1 = i22 * hm - bu22 * cf.kg;
  D M2 = (i12 * hm - bu12 * cf.kg) * P(2);
  nm(sg0), nm(sg1), nm(sg2), nm(M0), nm(M1), nm(M2);
  D JW = J * w;
  nm(JW);
  D MJ[3] = {M0 * JW, M1 * JW, M2 * JW};  // bending: nn·M J w = sum_k N_,k MJ_k - N_,α GM_α
  nm(MJ[0]), nm(MJ[1]), nm(MJ[2]);
  D qm = val(bf[0].v * MJ[0].v + bf[1].v * MJ[1].v + bf[2].v * MJ[2].v);  // M_k J w b_k
  nm(qm);
  [[maybe_unused]] T dg0{}, dg1{};  // M_k J w ∂Γ^α_k
  if constexpr (kTan) {
    const T mk_ = sd.t == 2 ? T(MJ[0].v) : sd.t == 3 ? T(MJ[1].v) : sd.t == 4 ? T(MJ[2].v) : T(0);
    const T qn = sd.t < 2 ? nj * T(qm.v) : T(0);
    dg0 = ig0 * qn + u0 * mk_;
    dg1 = ig1 * qn + u1 * mk_;
  }
  auto bend = [&](int i, D c, [[maybe_unused]] T dg) {  // the change of nn_k in the row's coefficient of N_,α
    if constexpr (kTan) c.d -= T(n[i].v) * dg;
    return c;
  };
  {
    D S0 = sg0 * JW, S1 = sg1 * JW, S2 = sg2 * JW;
    nm(S0), nm(S1), nm(S2);
    const D PN = JW * cf.pn;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const D c[6] = {bend(i, a[i][0] * S0 + a[i][1] * S2, dg0), bend(i, a[i][0] * S2 + a[i][1] * S1, dg1),
                      n[i] * MJ[0], n[i] * MJ[1], n[i] * MJ[2], -(n[i] * PN)};
      out.v(i, c, Gam);
    }
  }
  if constexpr (MOTION == ALEV_ || MOTION == ALEVB_) {
    D dvm[3][2];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      dvm[i][0] = mk<P, T>(pre[kPreD0 + 3 + i], sd.mesh(i, 0));
      dvm[i][1] = mk<P, T>(pre[kPreD1 + 3 + i], sd.mesh(i, 1));
    }
    D m11, m12, m22;
    visc(dvm, m11, m12, m22);
    D sm0 = i11 * cb - bu11 * hb + m11;  // GeoDynStress.jl:156-159
    D sm1 = i22 * cb - bu22 * hb + m22;
    D sm2 = i12 * cb - bu12 * hb + m12;
    nm(sm0), nm(sm1), nm(sm2);
    D pm = mk<P, T>(pre[kPreN + 7], sd.pres());
    D nd = cst<P, T>(P(0));
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      D dvn = mk<P, T>(pre[kPreN + 3 + i], sd.mesh(i, kN)) - mk<P, T>(pre[kPreN + i], sd.vel(i, kN));
      nd = nd + n[i] * dvn;
    }
    nm(nd);
    D E0 = sm0 * JW, E1 = sm1 * JW, E2 = sm2 * JW, PJ = pm * JW;
    nm(E0), nm(E1), nm(E2), nm(PJ);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      if constexpr (MOTION == ALEVB_) {  // the mesh rows carry the bending term too
        const D c[6] = {bend(i, a[i][0] * E0 + a[i][1] * E2, dg0), bend(i, a[i][0] * E2 + a[i][1] * E1, dg1),
                        n[i] * MJ[0], n[i] * MJ[1], n[i] * MJ[2], -(n[i] * PJ)};
        out.m6(i, c, Gam);
      } else {
        const D c[3] = {a[i][0] * E0 + a[i][1] * E2, a[i][0] * E2 + a[i][1] * E1, -(n[i] * PJ)};
        out.m3(i, c);
      }
    }
    out.p(-(JW * nd) - pm * (w * cf.adb_zv));
  }
  if constexpr (MOTION == EUL_) {
    D v[3], vmv[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      v[i] = mk<P, T>(pre[kPreN + i], sd.vel(i, kN));
      vmv[i] = mk<P, T>(pre[kPreN + 3 + i], sd.mesh(i, kN));
    }
    D nv = n[0] * v[0] + n[1] * v[1] + n[2] * v[2];
    nm(nv);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      D s = vmv[i] - n[i] * nv;
      nm(s);
      out.m1(i, s * JW * cf.am);
    }
  }
  out.l((J * tr - cf.adb_zv * lam) * w);
}

// ---- one boundary Gauss point ------------------------------------------------------
// calc_bdry_element_residual (FiniteElement.jl:363-384): the coefficients of
// N_,1, N_,2 and N of the three velocity rows at one point of boundary `bdry`,
// out(i, c[3]).  f: the point's table (w, N, N_,1, N_,2); X: the nodes.
template <class P, class T, class Tab, class Out>
__device__ __forceinline__ void bdry_eval(const P* X, const Tab* f, int bdry, int ntype, P nval, P mscale,
                                          const Seed<T>& sd, Out& out) {
  using D = Dual<P, T>;
  const P w = P(f[0]);
  D a[3][2];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    P s0 = 0, s1 = 0;
#pragma unroll
    for (int b = 0; b < 9; ++b) {
      s0 += P(f[10 + b]) * X[b * 3 + i];
      s1 += P(f[19 + b]) * X[b * 3 + i];
    }
    a[i][0] = mk<P, T>(s0, sd.x(i, 0));
    a[i][1] = mk<P, T>(s1, sd.x(i, 1));
  }
  D a11 = a[0][0] * a[0][0] + a[1][0] * a[1][0] + a[2][0] * a[2][0];
  D a12 = a[0][0] * a[0][1] + a[1][0] * a[1][1] + a[2][0] * a[2][1];
  D a22 = a[0][1] * a[0][1] + a[1][1] * a[1][1] + a[2][1] * a[2][1];
  D det = a11 * a22 - a12 * a12;
  D idet = inv(det);
  D i11 = a22 * idet, i12 = -(a12 * idet), i22 = a11 * idet;
  D aup[3][2];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    aup[i][0] = a[i][0] * i11 + a[i][1] * i12;
    aup[i][1] = a[i][0] * i12 + a[i][1] * i22;
  }
  D iJ = inv(dsqrt(det));
  D n[3];
  n[0] = (a[1][0] * a[2][1] - a[2][0] * a[1][1]) * iJ;
  n[1] = (a[2][0] * a[0][1] - a[0][0] * a[2][1]) * iJ;
  n[2] = (a[0][0] * a[1][1] - a[1][0] * a[0][1]) * iJ;
  // τ = ±a_α / |a_α|; the norm is a primal constant (conjugating dot, FiniteElement.jl:448)
  const bool c0 = bdry == 0 || bdry == 2;
  const P sgn = (bdry == 0 || bdry == 1) ? P(1) : P(-1);
  D ac[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) ac[i] = c0 ? a[i][0] : a[i][1];
  const P sc = sgn / sqrt(ac[0].v * ac[0].v + ac[1].v * ac[1].v + ac[2].v * ac[2].v);
  D tau[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) tau[i] = ac[i] * sc;
  D nu[3];
  nu[0] = tau[1] * n[2] - tau[2] * n[1];
  nu[1] = tau[2] * n[0] - tau[0] * n[2];
  nu[2] = tau[0] * n[1] - tau[1] * n[0];
  D t0 = aup[0][0] * tau[0] + aup[1][0] * tau[1] + aup[2][0] * tau[2];
  D t1 = aup[0][1] * tau[0] + aup[1][1] * tau[1] + aup[2][1] * tau[2];
  D JG = inv(dsqrt(t0 * t0 + t1 * t1));
  const D zero = cst<P, T>(P(0));
  if (ntype == MAFEM_STRETCH || ntype == MAFEM_SHEAR) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const D fi = (ntype == MAFEM_STRETCH ? nu[i] : tau[i]) * (nval * w) * JG;
      const D c[3] = {zero, zero, -fi};
      out(i, c);
    }
  } else {  // MOMENT (F_BEND only; other types are rejected on the host)
    D s = JG * (nval * mscale * w);
    D nu0 = (aup[0][0] * nu[0] + aup[1][0] * nu[1] + aup[2][0] * nu[2]) * s;
    D nu1 = (aup[0][1] * nu[0] + aup[1][1] * nu[1] + aup[2][1] * nu[2]) * s;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const D c[3] = {-(n[i] * nu0), -(n[i] * nu1), zero};
      out(i, c);
    }
  }
}

// ---- layout of D -------------------------------------------------------------------
// Per area point: "heavy" blocks of 6 x 5 (s over all six kinds, t over the five
// derivative kinds) for the pairs of a row field that carries the bending term
// and a field that moves the mesh, [pair 3 i + j][s][t], padded to kHS values
// per pair (16-byte reads; the three pairs of a warp in different banks); then
// "light" pairs of at most 2 x 3, kLS values each.
template <class P>
constexpr int kHS = sizeof(P) == 8 ? 30 : 36;
constexpr int kLS = 6;
template <int MOTION>
struct Lay {
  static constexpr bool ale = MOTION == ALEV_ || MOTION == ALEVB_;
  static constexpr bool lag = MOTION == LAG_, eul = MOTION == EUL_;
  static constexpr int nheavy = ale ? 2 : (lag || eul) ? 1 : 0;  // blocks of 9 pairs: v rows, then mesh rows
  static constexpr int dirs = lag ? 16 : 32;                     // lanes per point in phase 2
  static constexpr int warps = lag ? 5 : 9;
  static constexpr int threads = 32 * warps;
  template <class P>
  __host__ __device__ static constexpr int ctas() {  // resident CTAs per SM to compile for
    return lag ? (sizeof(P) == 8 ? 3 : 4) : 2;
  }
  // light groups of three pairs, in units of pairs
  static constexpr int vv = 0;                          // (v_i, v_j), i major: 9 pairs (not LAG)
  static constexpr int vl = lag ? 0 : 9;                // (v_i, λ)
  static constexpr int lv = vl + 3, ll = lv + 3;        // (λ, v_j), (λ, λ)
  static constexpr int lm = ll + 1;                     // (λ, m_j) (ALE, EUL)
  static constexpr int mp = lm + 3, pv = mp + 3, pm = pv + 3, pp = pm + 3;  // ALE: (m_i, p), (p, v_j), (p, m_j), (p, p)
  static constexpr int mv = lm + 3, mm = mv + 9;        // EUL: (m_i, v_j), (m_i, m_j)
  static constexpr int nlight = ale ? pp + 1 : eul ? mm + 9 : ll + 1;
  template <class P>
  __host__ __device__ static constexpr int light0() { return nheavy * 9 * kHS<P>; }
  template <class P>
  __host__ __device__ static constexpr int dsize() { return (light0<P>() + nlight * kLS + 3) & ~3; }
};

// Phase 2's output: the lane's direction selects where its derivatives go.
template <class P, int MOTION>
struct OutD {
  using LY = Lay<MOTION>;
  P* D;                 // the point's block
  int ov, sv, qv, nv;   // v rows: offset, stride per i and per s, number of s (0: none)
  int om, sm, qm;       // mesh rows (om < 0: none); qm = 0: only the last kind (N) is kept
  int op, ol;           // pressure, λ rows (< 0: none)
  template <class T>
  __device__ __forceinline__ void v(int i, const Dual<P, T> (&c)[6], const P (&)[3][2]) {
#pragma unroll
    for (int s = 0; s < 6; ++s)
      if (s < nv) D[ov + i * sv + s * qv] = c[s].d;
  }
  template <class T>
  __device__ __forceinline__ void m6(int i, const Dual<P, T> (&c)[6], const P (&)[3][2]) {
    if (om < 0) return;
#pragma unroll
    for (int s = 0; s < 6; ++s)
      if (qm || s == 5) D[om + i * sm + s * qm] = c[s].d;
  }
  template <class T>
  __device__ __forceinline__ void m3(int i, const Dual<P, T> (&c)[3]) {
    if (om < 0) return;
    if (qm) {
      D[om + i * sm] = c[0].d;
      D[om + i * sm + qm] = c[1].d;
#pragma unroll
      for (int s = 2; s < 5; ++s) D[om + i * sm + s * qm] = T(0);
    }
    D[om + i * sm + 5 * qm] = c[2].d;
  }
  template <class T>
  __device__ __forceinline__ void m1(int i, const Dual<P, T>& c) {
    if (om >= 0) D[om + i * sm] = c.d;
  }
  template <class T>
  __device__ __forceinline__ void p(const Dual<P, T>& c) {
    if (op >= 0) D[op] = c.d;
  }
  template <class T>
  __device__ __forceinline__ void l(const Dual<P, T>& c) {
    if (ol >= 0) D[ol] = c.d;
  }
};

// The direction of lane `dl` (0 .. dirs - 1) and where its derivatives go.
// LAG: v_j's five derivative kinds (3 x 5), λ; the other motions: v_j with
// N_,1, N_,2, N (3 x 3), m_j with all six kinds (3 x 6), λ, p.
template <class P, class T, int MOTION>
__host__ __device__ __forceinline__ bool direction(int dl, T dt, Seed<T>& sd, OutD<P, MOTION>& o) {
  using LY = Lay<MOTION>;
  constexpr int L0 = LY::template light0<P>();
  sd.dt = dt;
  sd.comp = 0;
  sd.t = kN;
  sd.v = sd.m = sd.l = sd.p = sd.geo = false;
  o.ov = o.sv = o.qv = o.nv = 0;
  o.om = -1;
  o.sm = o.qm = 0;
  o.op = o.ol = -1;
  if constexpr (LY::lag) {
    if (dl < 15) {
      sd.comp = dl / 5;
      sd.t = dl - 5 * sd.comp;
      sd.v = sd.geo = true;
    } else {
      sd.l = true;
    }
  } else {
    if (dl < 9) {
      sd.comp = dl / 3;
      const int r = dl - 3 * sd.comp;
      sd.t = r == 2 ? kN : r;
      sd.v = true;
    } else if (dl < 27) {
      sd.comp = (dl - 9) / 6;
      sd.t = dl - 9 - 6 * sd.comp;
      sd.m = sd.geo = MOTION != STATIC_;
      if (MOTION == STATIC_) return false;
    } else if (dl == 27) {
      sd.l = true;
    } else if (dl == 28 && LY::ale) {
      sd.p = true;
    } else {
      return false;
    }
  }
  const int j = sd.comp, t = sd.t;
  if (sd.geo && t < 5) {
    o.ov = j * kHS<P> + t;
    o.sv = 3 * kHS<P>;
    o.qv = 5;
    o.nv = 6;
    if constexpr (LY::ale) {
      o.om = 9 * kHS<P> + j * kHS<P> + t;
      o.sm = 3 * kHS<P>;
      o.qm = 5;
    }
  } else if (sd.v && t < 2) {
    o.ov = L0 + (LY::vv + j) * kLS + t;
    o.sv = 3 * kLS;
    o.qv = 3;
    o.nv = 2;
  } else if (sd.l) {
    o.ov = L0 + LY::vl * kLS;
    o.sv = kLS;
    o.qv = 3;
    o.nv = 2;
  }
  if constexpr (LY::ale) {
    if (sd.p) {
      o.om = L0 + LY::mp * kLS;
      o.sm = kLS;
      o.qm = 0;
      o.op = L0 + LY::pp * kLS;
    } else if (sd.v && t == kN) {
      o.op = L0 + (LY::pv + j) * kLS;
    } else if (sd.m && (t < 2 || t == kN)) {
      o.op = L0 + (LY::pm + j) * kLS + (t == kN ? 2 : t);
    }
  }
  if constexpr (LY::eul) {
    if (sd.v && t == kN) {
      o.om = L0 + (LY::mv + j) * kLS;
      o.sm = 3 * kLS;
    } else if (sd.m && (t < 2 || t == kN)) {
      o.om = L0 + (LY::mm + j) * kLS + (t == kN ? 2 : t);
      o.sm = 3 * kLS;
    }
  }
  if (sd.l) o.ol = L0 + LY::ll * kLS;
  else if (sd.v && t < 2) o.ol = L0 + (LY::lv + j) * kLS + t;
  else if (sd.m && t < 2) o.ol = L0 + (LY::lm + j) * kLS + t;
  return true;
}

// Phase 3's light units: a warp takes up to three pairs (27 lanes: pair x node
// a) of one group.  Row unknown r0 + q dr, column unknown c0 + q dc for pair q;
// s0: kN, or 0 for the two kinds N_,1, N_,2; t0..t2: the column's kinds (absent
// ones meet stored zeros).
struct LightUnit {
  short pair, npair, r0, dr, c0, dc, s0, t0, t1, t2;
};
template <int MOTION>
__host__ __device__ __forceinline__ LightUnit light_unit(int k) {
  using LY = Lay<MOTION>;
  // groups in order; LAG has no (v, v) group of its own
  if constexpr (!LY::lag) {
    if (k < 3) return LightUnit{(short)(LY::vv + 3 * k), 3, (short)k, 0, 0, 1, 0, 0, 1, 0};
    k -= 3;
  }
  if (k == 0) return LightUnit{LY::vl, 3, 0, 1, 6, 0, 0, kN, 0, 0};
  if (k == 1) return LightUnit{LY::lv, 3, 6, 0, 0, 1, kN, 0, 1, 0};
  if (k == 2) return LightUnit{LY::ll, 1, 6, 0, 6, 0, kN, kN, 0, 0};
  if constexpr (LY::ale || LY::eul) {
    if (k == 3) return LightUnit{LY::lm, 3, 6, 0, 3, 1, kN, 0, 1, 0};
  }
  if constexpr (LY::eul) {
    if (k < 7) return LightUnit{(short)(LY::mv + 3 * (k - 4)), 3, (short)(3 + k - 4), 0, 0, 1, kN, kN, 0, 0};
    return LightUnit{(short)(LY::mm + 3 * (k - 7)), 3, (short)(3 + k - 7), 0, 3, 1, kN, 0, 1, kN};
  }
  if (k == 4) return LightUnit{LY::mp, 3, 3, 1, 7, 0, kN, kN, 0, 0};
  if (k == 5) return LightUnit{LY::pv, 3, 7, 0, 0, 1, kN, kN, 0, 0};
  if (k == 6) return LightUnit{LY::pm, 3, 7, 0, 3, 1, kN, 0, 1, kN};
  return LightUnit{LY::pp, 1, 7, 0, 7, 0, kN, kN, 0, 0};
}
template <int MOTION>
__host__ __device__ constexpr int light_units() {
  return Lay<MOTION>::lag ? 3 : Lay<MOTION>::ale ? 11 : Lay<MOTION>::eul ? 13 : 6;
}

// Residual rows from the primal coefficients (plain form): c[row field][s] of
// every point; kCf per point: v 3 x 6, mesh 3 x 6, p, λ.
constexpr int kCf = 38;
template <class P>
struct OutCoef {
  P* c;
  __device__ __forceinline__ void v(int i, const Dual<P, Nil> (&x)[6], const P (&)[3][2]) {
#pragma unroll
    for (int s = 0; s < 6; ++s) c[i * 6 + s] = x[s].v;
  }
  __device__ __forceinline__ void m6(int i, const Dual<P, Nil> (&x)[6], const P (&)[3][2]) {
#pragma unroll
    for (int s = 0; s < 6; ++s) c[18 + i * 6 + s] = x[s].v;
  }
  __device__ __forceinline__ void m3(int i, const Dual<P, Nil> (&x)[3]) {
    c[18 + i * 6] = x[0].v;
    c[18 + i * 6 + 1] = x[1].v;
#pragma unroll
    for (int s = 2; s < 5; ++s) c[18 + i * 6 + s] = P(0);
    c[18 + i * 6 + 5] = x[2].v;
  }
  __device__ __forceinline__ void m1(int i, const Dual<P, Nil>& x) {
#pragma unroll
    for (int s = 0; s < 5; ++s) c[18 + i * 6 + s] = P(0);
    c[18 + i * 6 + 5] = x.v;
  }
  __device__ __forceinline__ void p(const Dual<P, Nil>& x) { c[36] = x.v; }
  __device__ __forceinline__ void l(const Dual<P, Nil>& x) { c[37] = x.v; }
};
struct OutNone {
  template <class X, class G>
  __device__ __forceinline__ void v(int, const X&, const G&) {}
  template <class X, class G>
  __device__ __forceinline__ void m6(int, const X&, const G&) {}
  template <class X>
  __device__ __forceinline__ void m3(int, const X&) {}
  template <class X>
  __device__ __forceinline__ void m1(int, const X&) {}
  template <class X>
  __device__ __forceinline__ void p(const X&) {}
  template <class X>
  __device__ __forceinline__ void l(const X&) {}
};

// Shared memory of elem_body, in values of P.  kBd: per boundary point, the
// 3 x 3 pairs' 3 x 2 derivatives, the nodes' (N_,1, N_,2, N) and the three rows'
// coefficients.  Per element of the CTA: phi, unknowns, positions, primal table,
// coefficients (plain form) and boundary points; D and the block once.
constexpr int kBd = 54 + 27 + 9;
constexpr int kPhi = 54;  // phi[b][s] of a point, then w (stride kTab)
template <class P>
__host__ __device__ constexpr int elem_slot(int max_bt) {
  return (9 * kTab + 72 + 28 + 9 * kPrim + 1 + (sizeof(P) == 8 ? 9 * kCf : 0) + max_bt * kBd + 3) & ~3;
}
template <class P, int MOTION, int EPB>
constexpr size_t elem_smem_values(int nq, int max_bt) {
  const size_t ks = (size_t)nq * (nq + 1), tab = (size_t)EPB * 9 * kTab;  // the raw tables share the block's place
  return 9 * Lay<MOTION>::template dsize<P>() + (size_t)EPB * elem_slot<P>(max_bt) + (ks > tab ? ks : tab);
}

// 16-byte (N values from a 16-byte boundary) and 2-value shared-memory reads
template <class P, int N, int M>
__device__ __forceinline__ void ld_quads(P (&r)[M], const P* p) {
  constexpr int E = 16 / (int)sizeof(P);
  using V = typename std::conditional<sizeof(P) == 8, double2, float4>::type;
#pragma unroll
  for (int k = 0; k < N / E; ++k) {
    const V v = reinterpret_cast<const V*>(p)[k];
    const P* e = reinterpret_cast<const P*>(&v);
#pragma unroll
    for (int i = 0; i < E; ++i) r[k * E + i] = e[i];
  }
}
template <class P, int N, int M>
__device__ __forceinline__ void ld_pairs(P (&r)[M], const P* p) {
  using V = typename std::conditional<sizeof(P) == 8, double2, float2>::type;
#pragma unroll
  for (int k = 0; k < N / 2; ++k) {
    const V v = reinterpret_cast<const V*>(p)[k];
    r[2 * k] = v.x;
    r[2 * k + 1] = v.y;
  }
}

// EPB elements per CTA, list positions kk0 .. kk0 + EPB - 1 below nel: elements
// elist[kk] (or kk).  Phases 0 and 1 run for all of them at once (phase 1 is a
// chain of ~250 instructions in nine lanes: a warp per element), phases 2 to 4
// one element after another.  Plain form (P = double, WANT_R): residual and
// tangent.  FP32 form (!WANT_R): the tangent alone.  area_only: the area Gauss
// points alone (calc_elem_dof_residuals without the Dohrmann-Bochev projection
// or boundary terms, as PullForce.jl uses it); K_el may be null (no tangent
// formed).  Shared by the single-patch kernel and the batched kernel, which
// reads Pt / pp from a job table into shared memory.
template <class P, bool WANT_R, int MOTION, int EPB>
__device__ __forceinline__ void elem_body(const DevPatch& Pt, const PhysParams& pp, double time, double dt,
                                          double* __restrict__ r_el, P* __restrict__ K_el,
                                          const int* __restrict__ elist, int kk0, int nel, int area_only,
                                          unsigned char* smem_raw) {
  using LY = Lay<MOTION>;
  static_assert(EPB <= LY::warps, "a warp per element in phase 1");
  constexpr int NT = LY::threads, DS = LY::template dsize<P>(), L0 = LY::template light0<P>();
  const int nq = pp.nq, ndf = pp.ndf, ldk = nq + 1;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ne = min(EPB, nel - kk0), slot = elem_slot<P>(pp.max_btask);
  auto elem_of = [&](int l) { return elist ? elist[kk0 + l] : kk0 + l; };
  P* D = reinterpret_cast<P*>(smem_raw);  // [9][DS]
  P* S0 = D + 9 * DS;                     // [EPB][slot]
  P* Ks = S0 + EPB * slot;                // [nq][ldk]: column, row
  P* tab = Ks;                            // [EPB][9][kTab]: the raw tables, until the interpolants are formed
  // places in a slot
  constexpr int oC = 9 * kTab, oX = oC + 72, oP = oX + 28, oF = oP + 9 * kPrim + 1,
                oB = oF + (sizeof(P) == 8 ? 9 * kCf : 0);

  // phase 0
  for (int k0 = tid; k0 < ne * 9 * kTab; k0 += NT) {
    const int l = k0 / (9 * kTab), k = k0 - l * 9 * kTab;
    P* phi = S0 + l * slot;  // [9][kTab]: phi[b][s], w at kPhi
    const P v = P(Pt.tab[(size_t)Pt.uel[elem_of(l)] * 9 * kTab + k]);
    tab[k0] = v;
    const int g = k / kTab, r = k - g * kTab;
    if (r == 0) phi[g * kTab + kPhi] = v;
    else if (r < 10) phi[g * kTab + (r - 1) * 6 + kN] = v;
    else if (r < 55) phi[g * kTab + ((r - 10) % 9) * 6 + (r - 10) / 9] = v;
  }
  for (int k0 = tid; k0 < ne * 27; k0 += NT) {
    const int l = k0 / 27, k = k0 - 27 * l, b = k / 3, i = k - 3 * b;
    S0[l * slot + oX + k] = P(Pt.xms[(size_t)i * Pt.numnp + Pt.ix[elem_of(l) * 9 + b]]);
  }
  for (int k0 = tid; k0 < ne * 72; k0 += NT) {
    const int l = k0 / 72, k = k0 - 72 * l, b = k / 8, d = k - 8 * b;
    S0[l * slot + oC + k] = d < ndf ? P(Pt.cps[(size_t)d * Pt.numnp + Pt.ix[elem_of(l) * 9 + b]]) : P(0);
  }
  if (K_el)  // the light pairs' unused places stay zero
    for (int k = tid; k < 9 * LY::nlight * kLS; k += NT) {
      const int g = k / (LY::nlight * kLS);
      D[g * DS + L0 + k - g * LY::nlight * kLS] = P(0);
    }
  __shared__ int s_nbt[EPB], s_u[EPB];  // an element's boundary points (Neumann entry, point); its tables
  if (tid < ne) {
    const int e = elem_of(tid);
    int n = 0;
    if (!area_only)
      for (int k = 0; k < pp.n_neu; ++k) n += Pt.bref[e * 4 + pp.neu_bdry[k]] >= 0 ? 3 : 0;
    s_nbt[tid] = n;
    s_u[tid] = Pt.uel[e];
  }
  __syncthreads();
  for (int k0 = tid; k0 < ne * 9 * kPre; k0 += NT) {
    const int l = k0 / (9 * kPre), k = k0 - l * 9 * kPre, gp = k / kPre;
    P* S = S0 + l * slot;
    S[oP + gp * kPrim + k - gp * kPre] =
        gp_pre_value<P>(k - gp * kPre, pp, S + oX, S + oC, tab + (l * 9 + gp) * kTab);
  }
  __syncthreads();
  // phase 1
  const Coef<P> cf(pp);
  if (warp < ne && lane < 9) {
    P* S = S0 + warp * slot;
    P* pr = S + oP + lane * kPrim;
    if constexpr (WANT_R) {
      OutCoef<P> oc{S + oF + lane * kCf};
      gp_eval<P, Nil, MOTION>(cf, pr, S[lane * kTab + kPhi], Seed<Nil>(), Store<P>{pr, kPre}, oc);
    } else {
      OutNone oc;
      gp_eval<P, Nil, MOTION>(cf, pr, S[lane * kTab + kPhi], Seed<Nil>(), Store<P>{pr, kPre}, oc);
    }
  }
  if (K_el)  // the raw tables in Ks are no longer read; blocks of uncoupled fields stay zero
    for (int k = tid; k < nq * ldk; k += NT) Ks[k] = P(0);
  // boundary points: six directions each (component j, N_,1 / N_,2), five points a warp, taken by the last warps
  for (int l = 0; l < ne; ++l) {
    const int e = elem_of(l), nbt = s_nbt[l];
    P* S = S0 + l * slot;
    const int bl = lane / 6, q = lane - 6 * bl;  // point slot, direction
    for (int b0 = (LY::warps - 1 - warp) * 5; b0 < nbt; b0 += LY::warps * 5) {
      const int bt = b0 + bl;
      if (bl < 5 && bt < nbt) {
        int k = 0, left = bt;  // the bt-th (entry, point)
        for (; k < pp.n_neu; ++k) {
          if (Pt.bref[e * 4 + pp.neu_bdry[k]] < 0) continue;
          if (left < 3) break;
          left -= 3;
        }
        const int bb = pp.neu_bdry[k], ntype = pp.neu_type[k];
        const double* src = Pt.btab + ((size_t)Pt.bref[e * 4 + bb] * 3 + left) * kTab;
        const P mscale = P(ntype == MAFEM_MOMENT ? fmin(time / pp.bend_tm, 1.0) : 1.0);
        Seed<P> sd;
        sd.comp = q >> 1;
        sd.t = q & 1;
        sd.v = sd.m = sd.l = sd.p = false;
        sd.geo = MOTION != STATIC_;
        sd.dt = P(dt);
        P* B = S + oB + bt * kBd;
        auto put = [&](int i, const Dual<P, P> (&c)[3]) {
#pragma unroll
          for (int s = 0; s < 3; ++s) {
            B[(i * 3 + (q >> 1)) * 6 + s * 2 + (q & 1)] = c[s].d;
            if (q == 0) B[81 + i * 3 + s] = c[s].v;
          }
        };
        bdry_eval<P, P>(S + oX, src, bb, ntype, P(pp.neu_val[k]), mscale, sd, put);
        for (int k2 = q; k2 < 27; k2 += 6) {
          const int b = k2 / 3, s = k2 - 3 * b;
          B[54 + k2] = P(src[s == 2 ? 1 + b : 10 + 9 * s + b]);
        }
      }
    }
  }
  __syncthreads();
  // nn_k[b] = N_,k - Γ^α_k N_,α in place of N_,k (Γ: named intermediates of gp_eval)
  for (int k0 = tid; k0 < ne * 243; k0 += NT) {
    const int l = k0 / 243, k = k0 - 243 * l, g = k / 27, r = k - 27 * g, b = r / 3, kk2 = r - 3 * b;
    P* S = S0 + l * slot;
    const P* G = S + oP + g * kPrim + kPreGam + 3 * kk2;
    P* ph = S + g * kTab + b * 6;
    ph[2 + kk2] -= G[0] * ph[0] + G[1] * ph[1];
  }
  __syncthreads();
#pragma unroll 1
  for (int l = 0; l < ne; ++l) {
    const int e = elem_of(l), nbt = s_nbt[l], u = s_u[l];
    const P* S = S0 + l * slot;
    const P* phi = S;
    const P* bd = S + oB;
    if (K_el) {
      // phase 2
      constexpr int PPW = 32 / LY::dirs;  // points per warp
      const int gp = warp * PPW + lane / LY::dirs, dl = lane % LY::dirs;
      if (gp < 9) {
        Seed<P> sd;
        OutD<P, MOTION> o;
        o.D = D + gp * DS;
        if (direction<P, P, MOTION>(dl, P(dt), sd, o)) {
          const P* pr = S + oP + gp * kPrim;
          gp_eval<P, P, MOTION>(cf, pr, phi[gp * kTab + kPhi], sd, Load<P>{pr, kPre}, o);
        }
      }
      __syncthreads();
      // phase 3
      const int q = lane / 9, na = lane - 9 * q;  // pair and column node of this lane
      const bool on = q < 3;
      const double dbs = pp.adb / pp.zv;
      for (int un = warp; un < 3 * LY::nheavy; un += LY::warps) {  // heavy: row field `un`, column field m_q (LAG: v_q)
        if (on) {
          P acc[9];
#pragma unroll
          for (int b = 0; b < 9; ++b) acc[b] = P(0);
          const P* Dp = D + (un * 3 + q) * kHS<P>;
#pragma unroll 1
          for (int g = 0; g < 9; ++g) {
            const P* ph = phi + g * kTab;
            P pt[6], W[6], Dg[32];
            ld_pairs<P, 6>(pt, ph + na * 6);
            ld_quads<P, sizeof(P) == 8 ? 30 : 32>(Dg, Dp + g * DS);
#pragma unroll
            for (int s = 0; s < 6; ++s) {
              W[s] = Dg[s * 5] * pt[0];
#pragma unroll
              for (int t = 1; t < 5; ++t) W[s] += Dg[s * 5 + t] * pt[t];
            }
#pragma unroll
            for (int b2 = 0; b2 < 10; b2 += 2) {  // two rows' basis values: 12 values, 16-byte aligned
              P f[12];
              ld_quads<P, 12>(f, ph + b2 * 6);  // (b = 9: the point's weight and the next point's first values, unused)
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int b = b2 + h;
                if (b > 8) continue;
                // FP32: the point's sum first, one rounding at the size of acc per point
                P v = sizeof(P) == 8 ? acc[b] + f[h * 6] * W[0] : f[h * 6] * W[0];
#pragma unroll
                for (int s = 1; s < 6; ++s) v += f[h * 6 + s] * W[s];
                acc[b] = sizeof(P) == 8 ? v : acc[b] + v;
              }
            }
          }
          if (un < 3)  // the velocity rows' boundary points
            for (int bt = 0; bt < nbt; ++bt) {
              const P* B = bd + bt * kBd;
              const P p0 = B[54 + na * 3], p1 = B[54 + na * 3 + 1];
              P W[3];
#pragma unroll
              for (int s = 0; s < 3; ++s) W[s] = B[(un * 3 + q) * 6 + 2 * s] * p0 + B[(un * 3 + q) * 6 + 2 * s + 1] * p1;
#pragma unroll
              for (int b = 0; b < 9; ++b)
#pragma unroll
                for (int s = 0; s < 3; ++s) acc[b] += B[54 + b * 3 + s] * W[s];
            }
          const int rd = pp.dof_of[un], cd = pp.dof_of[(LY::lag ? 0 : 3) + q];
          if (rd >= 0 && cd >= 0) {
            P* dst = Ks + (na * ndf + cd) * ldk + rd;
#pragma unroll
            for (int b = 0; b < 9; ++b) dst[b * ndf] = acc[b];
          }
        }
      }
      // light units: the warps without a heavy one (every warp when there are none)
      constexpr int w0 = 3 * LY::nheavy;
      for (int k = warp - w0; k >= 0 && k < light_units<MOTION>(); k += LY::warps - w0) {
        const LightUnit U = light_unit<MOTION>(k);
        if (on && q < U.npair) {
          const int ru = U.r0 + q * U.dr, cu = U.c0 + q * U.dc;
          const int rd = pp.dof_of[ru], cd = pp.dof_of[cu];
          P acc[9];
#pragma unroll
          for (int b = 0; b < 9; ++b) acc[b] = P(0);
          if (ru == cu && ru >= 6 && !area_only) {
            // Dohrmann-Bochev projection (FiniteElement.jl:323-327): rλ += Gᵀ H⁻¹ G λ αdb/ζv,
            // and for ALEV/ALEVB rp += Gᵀ H⁻¹ G p αdb/ζv.  Linear in λ / p.
            const double* T81 = Pt.db + (size_t)u * 81;
#pragma unroll
            for (int b = 0; b < 9; ++b) acc[b] = P(T81[b * 9 + na] * dbs);
          }
          const P* Dp = D + L0 + (U.pair + q) * kLS;
#pragma unroll 1
          for (int g = 0; g < 9; ++g) {
            const P* ph = phi + g * kTab;
            const P p0 = ph[na * 6 + U.t0], p1 = ph[na * 6 + U.t1], p2 = ph[na * 6 + U.t2];
            P Dg[6];
            ld_pairs<P, 6>(Dg, Dp + g * DS);
            const P W0 = Dg[0] * p0 + Dg[1] * p1 + Dg[2] * p2;
            if (U.s0 == kN) {  // rows with the basis values alone
#pragma unroll
              for (int b = 0; b < 9; ++b) acc[b] += ph[b * 6 + kN] * W0;
            } else {  // N_,1 and N_,2
              const P W1 = Dg[3] * p0 + Dg[4] * p1 + Dg[5] * p2;
#pragma unroll
              for (int b = 0; b < 9; ++b) {
                P f[2];
                ld_pairs<P, 2>(f, ph + b * 6);
                acc[b] += f[0] * W0 + f[1] * W1;
              }
            }
          }
          if (rd >= 0 && cd >= 0) {
            P* dst = Ks + (na * ndf + cd) * ldk + rd;
#pragma unroll
            for (int b = 0; b < 9; ++b) dst[b * ndf] = acc[b];
          }
        }
      }
    }
    if constexpr (WANT_R) {
      for (int row = NT - 1 - tid; row < nq; row += NT) {  // the last warps: they hold the light units
        const int b = row / ndf, d = row - b * ndf, un = pp.unk_of[d];
        P r = P(0);
        for (int g = 0; g < 9; ++g) {
          const P* ph = phi + g * kTab + b * 6;
          const P* c = S + oF + g * kCf;
          if (un < 6) {
            P s = ph[0] * c[un * 6];
#pragma unroll
            for (int k = 1; k < 6; ++k) s += ph[k] * c[un * 6 + k];
            r += s;
          } else {
            r += ph[kN] * c[un == 6 ? 37 : 36];
          }
        }
        if (!area_only) {
          if (un == 6 || (un == 7 && LY::ale)) {
            const double* T81 = Pt.db + (size_t)u * 81;
            double s = 0;
            for (int c = 0; c < 9; ++c) s += T81[b * 9 + c] * S[oC + c * 8 + d];
            r += s * (pp.adb / pp.zv);
          }
          if (un < 3)
            for (int bt = 0; bt < nbt; ++bt) {
              const P* B = bd + bt * kBd;
              r += B[54 + b * 3] * B[81 + un * 3] + B[54 + b * 3 + 1] * B[81 + un * 3 + 1] +
                   B[54 + b * 3 + 2] * B[81 + un * 3 + 2];
            }
        }
        r_el[(size_t)(kk0 + l) * nq + row] = r;
      }
    }
    if (K_el) {
      // phase 4: column-major element block K_el[e][col][row]
      __syncthreads();
      P* dst = K_el + (size_t)e * nq * nq;
      for (int c = warp; c < nq; c += LY::warps)
        for (int r = lane; r < nq; r += 32) dst[c * nq + r] = Ks[c * ldk + r];
    }
  }
}

// Two CTAs per SM: one's serial phases (0, 1, 4) run beside the other's FP64
// work.  In FP64 that holds it to 96 registers, which spills 0.7 KB per thread,
// yet 32 x 32 ALEVB is assembled in 1.00 ms against 1.11 ms with one CTA and 168
// registers (both before the closed-form geometry derivatives).
template <class P, bool WANT_R, int MOTION, int EPB>
__global__ void __launch_bounds__(Lay<MOTION>::threads, (Lay<MOTION>::template ctas<P>()))
    elem_kernel(DevPatch Pt, PhysParams pp, double time, double dt, double* __restrict__ r_el, P* __restrict__ K_el,
                const int* __restrict__ elist, int nel, int area_only) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  elem_body<P, WANT_R, MOTION, EPB>(Pt, pp, time, dt, r_el, K_el, elist, blockIdx.x * EPB, nel, area_only, smem_raw);
}

// FP64 residual of the FP32 form: primal only, one thread per (element, area
// Gauss point).  Phase 1: each task adds its point's contribution to every
// element row into its own shared array; phase 2: one thread per (element,
// row) sums them in Gauss-point order and adds the Dohrmann-Bochev term;
// phase 3: the Neumann points (task = element, bc, point; velocity rows only)
// likewise, summed in (bc, point) order -- the plain form's order.
struct OutRows {  // adds a point's rows into R[row]
  double* R;      // [row]
  const double* f;
  const PhysParams& pp;
  __device__ __forceinline__ void add(int d, const double (&c)[6]) {
    if (d < 0) return;
#pragma unroll 1
    for (int b = 0; b < 9; ++b)
      R[b * pp.ndf + d] += f[10 + b] * c[0] + f[19 + b] * c[1] + f[28 + b] * c[2] + f[37 + b] * c[3] +
                           f[46 + b] * c[4] + f[1 + b] * c[5];
  }
  __device__ __forceinline__ void addn(int d, double c) {
    if (d < 0) return;
#pragma unroll 1
    for (int b = 0; b < 9; ++b) R[b * pp.ndf + d] += f[1 + b] * c;
  }
  // sum_k c_k nn_k = sum_k c_k N_,k - (sum_k c_k Γ^α_k) N_,α
  __device__ __forceinline__ void addc(int d, const Dual<double, Nil> (&x)[6], const double (&G)[3][2]) {
    const double c[6] = {x[0].v - (G[0][0] * x[2].v + G[1][0] * x[3].v + G[2][0] * x[4].v),
                         x[1].v - (G[0][1] * x[2].v + G[1][1] * x[3].v + G[2][1] * x[4].v),
                         x[2].v, x[3].v, x[4].v, x[5].v};
    add(d, c);
  }
  __device__ __forceinline__ void v(int i, const Dual<double, Nil> (&x)[6], const double (&G)[3][2]) {
    addc(pp.dof_of[i], x, G);
  }
  __device__ __forceinline__ void m6(int i, const Dual<double, Nil> (&x)[6], const double (&G)[3][2]) {
    addc(pp.dof_of[3 + i], x, G);
  }
  __device__ __forceinline__ void m3(int i, const Dual<double, Nil> (&x)[3]) {
    const double c[6] = {x[0].v, x[1].v, 0.0, 0.0, 0.0, x[2].v};
    add(pp.dof_of[3 + i], c);
  }
  __device__ __forceinline__ void m1(int i, const Dual<double, Nil>& x) { addn(pp.dof_of[3 + i], x.v); }
  __device__ __forceinline__ void p(const Dual<double, Nil>& x) { addn(pp.dof_of[7], x.v); }
  __device__ __forceinline__ void l(const Dual<double, Nil>& x) { addn(pp.dof_of[6], x.v); }
};
// Elements per CTA: 63 threads, so that a patch of 32 x 32 elements spreads over
// 147 SMs: an FP64 instruction holds its sub-partition for 64 cycles, so the
// kernel's time is its longest warp chain (98 us with 16 per CTA on 64 SMs).
constexpr int kResEPB = 7;
template <int MOTION>
__device__ __forceinline__ void resid_body(const DevPatch& Pt, const PhysParams& pp, double time, double dt,
                                           double* __restrict__ r_el, int blk, unsigned char* smem_raw) {
  const int nq = pp.nq, ndf = pp.ndf;
  double* X = reinterpret_cast<double*>(smem_raw);  // [kResEPB][27]
  double* C = X + kResEPB * 27;                       // [kResEPB][72]
  double* R = C + kResEPB * 72;                       // [kResEPB*9][nq], reused as [kResEPB*24][27]
  const int tid = threadIdx.x;
  const int e0 = blk * kResEPB;
  const int ne = min(kResEPB, Pt.numel - e0);
  for (int k = tid; k < ne * 27; k += blockDim.x) {
    const int el = k / 27, r = k - 27 * el, b = r / 3, i = r - 3 * b;
    X[k] = Pt.xms[(size_t)i * Pt.numnp + Pt.ix[(e0 + el) * 9 + b]];
  }
  for (int k = tid; k < ne * 72; k += blockDim.x) {
    const int el = k / 72, r = k - 72 * el, b = r / 8, d = r - 8 * b;
    C[k] = d < ndf ? Pt.cps[(size_t)d * Pt.numnp + Pt.ix[(e0 + el) * 9 + b]] : 0.0;
  }
  for (int k = tid; k < kResEPB * 9 * nq; k += blockDim.x) R[k] = 0.0;
  __syncthreads();
  const Coef<double> cf(pp);
  {
    const int el = tid / 9, gp = tid - 9 * el;
    if (el < ne) {
      const double* f = Pt.tab + ((size_t)Pt.uel[e0 + el] * 9 + gp) * kTab;
      double pre[kPre];
#pragma unroll
      for (int j = 0; j < kPre; ++j) pre[j] = gp_pre_value<double>(j, pp, X + el * 27, C + el * 72, f);
      OutRows acc{R + (size_t)tid * nq, f, pp};
      gp_eval<double, Nil, MOTION>(cf, pre, f[0], Seed<Nil>(), Keep(), acc);
    }
  }
  __syncthreads();
  // phase 2: rows (each thread keeps its sums for phase 3)
  constexpr int kMaxOwn = (kResEPB * 72 + kResEPB * 9 - 1) / (kResEPB * 9);  // 8
  double own[kMaxOwn];
  const double s = pp.adb / pp.zv;
  const int lo = pp.dof_of[6], po = pp.dof_of[7];
  const bool alep = (MOTION == ALEV_ || MOTION == ALEVB_);
#pragma unroll
  for (int j = 0; j < kMaxOwn; ++j) {
    const int pr = tid + j * kResEPB * 9;
    const int el = pr / nq, row = pr - el * nq;
    own[j] = 0.0;
    if (el < ne) {
      double r = 0.0;
      for (int gp = 0; gp < 9; ++gp) r += R[(size_t)(el * 9 + gp) * nq + row];
      const int b = row / ndf, d = row - b * ndf;
      if (d == lo || (alep && d == po)) {
        const double* T81 = Pt.db + (size_t)Pt.uel[e0 + el] * 81;
        double sv = 0;
        for (int c = 0; c < 9; ++c) sv += T81[b * 9 + c] * C[el * 72 + c * 8 + d];
        r += sv * s;
      }
      own[j] = r;
    }
  }
  // phase 3: Neumann points
  const int nn = pp.n_neu;
  if (nn > 0) {
    __syncthreads();
    const int ntask = ne * nn * 3;
    for (int k = tid; k < kResEPB * 24 * 27; k += blockDim.x) R[k] = 0.0;
    __syncthreads();
    for (int t = tid; t < ntask; t += blockDim.x) {
      const int el = t / (nn * 3), r = t - el * nn * 3, k = r / 3, g = r - 3 * k;
      const int bd = pp.neu_bdry[k];
      const int row = Pt.bref[(e0 + el) * 4 + bd];
      if (row < 0) continue;
      const double mscale = pp.neu_type[k] == MAFEM_MOMENT ? fmin(time / pp.bend_tm, 1.0) : 1.0;
      const double* f = Pt.btab + ((size_t)row * 3 + g) * kTab;
      double* Rt = R + (size_t)t * 27;  // velocity rows only: [b][i]
      auto put = [&](int i, const Dual<double, Nil> (&c)[3]) {
#pragma unroll 1
        for (int b = 0; b < 9; ++b) Rt[b * 3 + i] += f[10 + b] * c[0].v + f[19 + b] * c[1].v + f[1 + b] * c[2].v;
      };
      bdry_eval<double, Nil>(X + el * 27, f, bd, pp.neu_type[k], pp.neu_val[k], mscale, Seed<Nil>(), put);
    }
    __syncthreads();
    const int vd0 = pp.dof_of[0], vd1 = pp.dof_of[1], vd2 = pp.dof_of[2];
#pragma unroll
    for (int j = 0; j < kMaxOwn; ++j) {
      const int pr = tid + j * kResEPB * 9;
      const int el = pr / nq, row = pr - el * nq;
      if (el >= ne) continue;
      const int b = row / ndf, d = row - b * ndf;
      const int i = d == vd0 ? 0 : d == vd1 ? 1 : d == vd2 ? 2 : -1;
      if (i < 0) continue;
      for (int k = 0; k < nn; ++k) {
        if (Pt.bref[(e0 + el) * 4 + pp.neu_bdry[k]] < 0) continue;
        for (int g = 0; g < 3; ++g) own[j] += R[(size_t)((el * nn + k) * 3 + g) * 27 + b * 3 + i];
      }
    }
  }
#pragma unroll
  for (int j = 0; j < kMaxOwn; ++j) {
    const int pr = tid + j * kResEPB * 9;
    const int el = pr / nq, row = pr - el * nq;
    if (el < ne) r_el[(size_t)(e0 + el) * nq + row] = own[j];
  }
}

template <int MOTION>
__global__ void __launch_bounds__(kResEPB * 9) elem_resid_kernel(DevPatch Pt, PhysParams pp, double time, double dt,
                                                                double* __restrict__ r_el) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  resid_body<MOTION>(Pt, pp, time, dt, r_el, blockIdx.x, smem_raw);
}

// ---- batched element kernels of the FP32 form: every patch of a round in one launch per motion ----
// The CTA reads its patch's tables and parameters into shared memory, then runs
// the single-patch kernel's body on its CTA number within the patch.
template <int MOTION>
__global__ void __launch_bounds__(kResEPB * 9) batch_resid_kernel(const AsmJob* __restrict__ jobs,
                                                                 const AsmItem* __restrict__ items,
                                                                 const int* __restrict__ off, int m) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_k;
  __shared__ __align__(16) DevPatch sP;
  __shared__ __align__(16) PhysParams spp;
  const int k = batch_item(off, m, &s_k);
  const AsmItem it = items[k];
  const AsmJob* J = jobs + it.job;
  batch_copy(&sP, &J->P, (int)sizeof(DevPatch));
  batch_copy(&spp, &J->pp, (int)sizeof(PhysParams));
  __syncthreads();
  resid_body<MOTION>(sP, spp, it.time, it.dt, J->r_el, off[0] + (int)blockIdx.x - off[k], smem_raw);
}
// Elements per CTA of the FP32 tangent kernel: 2 or 4, chosen per motion by the
// batch's autotuner (four share a CTA's set-up and phases 0 and 1, two spread
// small rounds over more SMs).
template <int MOTION, int EPB>
__global__ void __launch_bounds__(Lay<MOTION>::threads, (Lay<MOTION>::template ctas<float>()))
    batch_tan_kernel(const AsmJob* __restrict__ jobs, const AsmItem* __restrict__ items, const int* __restrict__ off,
                     int m) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_k;
  __shared__ __align__(16) DevPatch sP;
  __shared__ __align__(16) PhysParams spp;
  const int k = batch_item(off, m, &s_k);
  const AsmItem it = items[k];
  const AsmJob* J = jobs + it.job;
  batch_copy(&sP, &J->P, (int)sizeof(DevPatch));
  batch_copy(&spp, &J->pp, (int)sizeof(PhysParams));
  __syncthreads();
  elem_body<float, false, MOTION, EPB>(sP, spp, it.time, it.dt, nullptr, J->K_el, nullptr,
                                       (off[0] + (int)blockIdx.x - off[k]) * EPB, sP.numel, 0, smem_raw);
}

// ---- launchers -----------------------------------------------------------------------
// The dynamic shared memory a kernel may ask for: the largest element (nq = 72)
// with the most boundary points it can have (8 Neumann entries).
template <class P, int MOTION, int EPB>
static size_t elem_smem(const PhysParams& pp) {
  return elem_smem_values<P, MOTION, EPB>(pp.nq, pp.max_btask) * sizeof(P);
}
template <class P, int MOTION, int EPB>
static size_t elem_smem_cap() {
  return elem_smem_values<P, MOTION, EPB>(72, 3 * kMaxNeu) * sizeof(P);
}
static size_t resid_smem(int nq) {
  return (size_t)kResEPB * (27 + 72) * 8 + (size_t)std::max(kResEPB * 9 * nq, kResEPB * 24 * 27) * 8;
}

template <class P, bool WANT_R, int MOTION, int EPB>
static cudaError_t launch_elem_t(const DevPatch& Pt, const PhysParams& pp, double time, double dt, double* r_el,
                                 P* K_el, cudaStream_t st, const int* elist, int nlist, int area_only) {
  auto kern = elem_kernel<P, WANT_R, MOTION, EPB>;
  cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)elem_smem_cap<P, MOTION, EPB>());
  if (e != cudaSuccess) return e;
  const int nel = elist ? nlist : Pt.numel;
  kern<<<(nel + EPB - 1) / EPB, Lay<MOTION>::threads, elem_smem<P, MOTION, EPB>(pp), st>>>(
      Pt, pp, time, dt, r_el, K_el, elist, nel, area_only);
  return cudaGetLastError();
}

template <int MOTION>
static cudaError_t launch_resid_t(const DevPatch& Pt, const PhysParams& pp, double time, double dt, double* r_el,
                                  cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(elem_resid_kernel<MOTION>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)resid_smem(72));
  if (e != cudaSuccess) return e;
  elem_resid_kernel<MOTION><<<(Pt.numel + kResEPB - 1) / kResEPB, kResEPB * 9, resid_smem(pp.nq), st>>>(Pt, pp, time,
                                                                                                     dt, r_el);
  return cudaGetLastError();
}

template <>
cudaError_t launch_elem<double>(const DevPatch& Pt, const PhysParams& pp, double time, double dt, double* r_el,
                                double* K_el, cudaStream_t st, const int* elist, int nlist, int area_only) {
  switch (pp.motion) {
    case MAFEM_STATIC:
      return launch_elem_t<double, true, STATIC_, 1>(Pt, pp, time, dt, r_el, K_el, st, elist, nlist, area_only);
    case MAFEM_EUL:
      return launch_elem_t<double, true, EUL_, 1>(Pt, pp, time, dt, r_el, K_el, st, elist, nlist, area_only);
    case MAFEM_LAG:
      return launch_elem_t<double, true, LAG_, 1>(Pt, pp, time, dt, r_el, K_el, st, elist, nlist, area_only);
    case MAFEM_ALEV:
      return launch_elem_t<double, true, ALEV_, 1>(Pt, pp, time, dt, r_el, K_el, st, elist, nlist, area_only);
    default:
      return launch_elem_t<double, true, ALEVB_, 1>(Pt, pp, time, dt, r_el, K_el, st, elist, nlist, area_only);
  }
}

// FP32 form: the FP64 residual kernel, then the FP32 tangent (whole patch only)
template <int MOTION>
static cudaError_t launch_elem_f(const DevPatch& Pt, const PhysParams& pp, double time, double dt, double* r_el,
                                 float* K_el, cudaStream_t st) {
  const cudaError_t e = launch_resid_t<MOTION>(Pt, pp, time, dt, r_el, st);
  if (e) return e;
  // One element per CTA while all of them are resident at once, else two (one wave less
  // of serial phases).  On 152 SMs, assembly with its gathers, one element -> two: LAG
  // (four CTAs per SM) 289 elements 93 -> 99 us, 400 100 -> 107, 600 104 -> 111, 900
  // 117 -> 114; ALEVB (two) 289 125 -> 132, 400 149 -> 151, 484 155 -> 153.
  int dev = 0, sms = 0;
  cudaError_t e2 = cudaGetDevice(&dev);
  if (e2 == cudaSuccess) e2 = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e2 != cudaSuccess) return e2;
  return Pt.numel <= Lay<MOTION>::template ctas<float>() * sms
             ? launch_elem_t<float, false, MOTION, 1>(Pt, pp, time, dt, r_el, K_el, st, nullptr, 0, 0)
             : launch_elem_t<float, false, MOTION, 2>(Pt, pp, time, dt, r_el, K_el, st, nullptr, 0, 0);
}
template <>
cudaError_t launch_elem<float>(const DevPatch& Pt, const PhysParams& pp, double time, double dt, double* r_el,
                               float* K_el, cudaStream_t st, const int* elist, int nlist, int area_only) {
  if (elist || nlist || area_only) return cudaErrorInvalidValue;
  switch (pp.motion) {
    case MAFEM_STATIC: return launch_elem_f<STATIC_>(Pt, pp, time, dt, r_el, K_el, st);
    case MAFEM_EUL: return launch_elem_f<EUL_>(Pt, pp, time, dt, r_el, K_el, st);
    case MAFEM_LAG: return launch_elem_f<LAG_>(Pt, pp, time, dt, r_el, K_el, st);
    case MAFEM_ALEV: return launch_elem_f<ALEV_>(Pt, pp, time, dt, r_el, K_el, st);
    default: return launch_elem_f<ALEVB_>(Pt, pp, time, dt, r_el, K_el, st);
  }
}

int batch_resid_ctas(int numel) { return (numel + kResEPB - 1) / kResEPB; }
int batch_tan_ctas(int numel, int epb) { return (numel + epb - 1) / epb; }

template <int MOTION>
static cudaError_t batch_setup_t() {
  cudaError_t e = cudaFuncSetAttribute(batch_resid_kernel<MOTION>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)resid_smem(72));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(batch_tan_kernel<MOTION, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)elem_smem_cap<float, MOTION, 2>());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(batch_tan_kernel<MOTION, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)elem_smem_cap<float, MOTION, 4>());
  return e;
}
cudaError_t batch_asm_setup() {
  cudaError_t e = batch_setup_t<STATIC_>();
  if (e == cudaSuccess) e = batch_setup_t<EUL_>();
  if (e == cudaSuccess) e = batch_setup_t<LAG_>();
  if (e == cudaSuccess) e = batch_setup_t<ALEV_>();
  if (e == cudaSuccess) e = batch_setup_t<ALEVB_>();
  return e;
}

cudaError_t launch_batch_resid(int motion, const AsmJob* jobs, const AsmItem* items, const int* off, int m, int ctas,
                               int nq, cudaStream_t st) {
  if (ctas <= 0) return cudaSuccess;
  const size_t sm = resid_smem(nq);
  switch (motion) {
    case MAFEM_STATIC: batch_resid_kernel<STATIC_><<<ctas, kResEPB * 9, sm, st>>>(jobs, items, off, m); break;
    case MAFEM_EUL: batch_resid_kernel<EUL_><<<ctas, kResEPB * 9, sm, st>>>(jobs, items, off, m); break;
    case MAFEM_LAG: batch_resid_kernel<LAG_><<<ctas, kResEPB * 9, sm, st>>>(jobs, items, off, m); break;
    case MAFEM_ALEV: batch_resid_kernel<ALEV_><<<ctas, kResEPB * 9, sm, st>>>(jobs, items, off, m); break;
    default: batch_resid_kernel<ALEVB_><<<ctas, kResEPB * 9, sm, st>>>(jobs, items, off, m); break;
  }
  return cudaGetLastError();
}
template <int MOTION>
static void launch_batch_tan_m(int epb, const AsmJob* jobs, const AsmItem* items, const int* off, int m, int ctas,
                               const PhysParams& pp, cudaStream_t st) {
  if (epb == 2)
    batch_tan_kernel<MOTION, 2>
        <<<ctas, Lay<MOTION>::threads, elem_smem<float, MOTION, 2>(pp), st>>>(jobs, items, off, m);
  else
    batch_tan_kernel<MOTION, 4>
        <<<ctas, Lay<MOTION>::threads, elem_smem<float, MOTION, 4>(pp), st>>>(jobs, items, off, m);
}
cudaError_t launch_batch_tan(int epb, const AsmJob* jobs, const AsmItem* items, const int* off, int m, int ctas,
                             const PhysParams& pp, cudaStream_t st) {
  if (ctas <= 0) return cudaSuccess;
  if (epb != 2 && epb != 4) return cudaErrorInvalidValue;
  switch (pp.motion) {
    case MAFEM_STATIC: launch_batch_tan_m<STATIC_>(epb, jobs, items, off, m, ctas, pp, st); break;
    case MAFEM_EUL: launch_batch_tan_m<EUL_>(epb, jobs, items, off, m, ctas, pp, st); break;
    case MAFEM_LAG: launch_batch_tan_m<LAG_>(epb, jobs, items, off, m, ctas, pp, st); break;
    case MAFEM_ALEV: launch_batch_tan_m<ALEV_>(epb, jobs, items, off, m, ctas, pp, st); break;
    default: launch_batch_tan_m<ALEVB_>(epb, jobs, items, off, m, ctas, pp, st); break;
  }
  return cudaGetLastError();
}

}  // namespace mafem
