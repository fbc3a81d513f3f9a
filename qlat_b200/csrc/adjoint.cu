// adjoint.cu -- reverse-mode derivative (VJP) of the gradient flow.
//
// Conventions.  A tangent or cotangent at a gauge field is an su(3) field X
// (traceless anti-Hermitian per link) acting by left multiplication,
// U -> exp(s X) U.  In the basis T_a of matrix-hmc.h:76-106 (tr T_a T_b =
// -2 delta_ab) the pairing is <X, Y> = sum_a X^a Y^a = -tr(X Y)/2, and the
// gradient of a function L is the su(3) field sum_a (dL/domega_a) T_a.
// (Qlattice's force set_gm_force is -1/2 of the action's gradient in this
// convention, since its kinetic term is sum_a p_a^2.)
//
// One flow stage W' = exp(eps Z) W with Z = a F(W) + b Z_prev pulls a
// cotangent lambda' at W' back to
//   lambda = Ad_{exp(-eps Z)} lambda' + a DF(W)^T mu,   mu = eps dexp_{-eps Z}(lambda') [+ carry],
// with dexp_A(B) = sum_k ad_A^k B / (k+1)! and a carry b mu to the previous
// stage's Z.  The transpose of the force Jacobian on the group is
// DF^T[Y] = DF[Y] + [F, Y]: the Hessian of the action is symmetric up to the
// commutator term of non-commuting left derivatives.  DF[Y] is evaluated in
// forward mode: every link U of the staple paths carries its tangent Y U.
// The forward exponential is the order-20 polynomial; its derivative is taken
// as that of the exact exponential (the difference is below rounding for the
// flow's step sizes).
#include <cuda_runtime.h>

#include "gauge_common.cuh"
#include "kernels.h"
#include "su3.cuh"

namespace qgb
{

template <typename R>
struct Dual {
  M3<R> v, d;  // value and tangent
};

template <typename R>
__device__ __forceinline__ Dual<R> dmul(const Dual<R>& a, const Dual<R>& b)
{
  Dual<R> r;
  r.v = mul(a.v, b.v);
  r.d = add_mul(mul(a.d, b.v), a.v, b.d);
  return r;
}

// link (site, dir) with tangent Y(site, dir) U(site, dir), optionally its adjoint
// (the tangent of U^+ is (Y U)^+ = -U^+ Y).
template <typename R>
__device__ __forceinline__ Dual<R> dlink(const CField<R>& U, const CField<R>& Y, long site, int dir, bool dagger)
{
  const M3<R> u = U.ld(site, dir);
  const M3<R> y = Y.ld(site, dir);
  Dual<R> r;
  if (!dagger) {
    r.v = u;
    r.d = mul(y, u);
  } else {
    r.v = adj(u);
    r.d = scale(R(-1), mul(r.v, y));
  }
  return r;
}

// [A, B]
template <typename R>
__device__ __forceinline__ M3<R> commutator(const M3<R>& a, const M3<R>& b)
{
  M3<R> r = mul(a, b);
  const M3<R> t = mul(b, a);
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    r.e[i].re -= t.e[i].re;
    r.e[i].im -= t.e[i].im;
  }
  return r;
}

// The links of the staple paths at signed direction e = s nu as dual
// matrices (positions x + a mu + b e, as SignedDir in force_impl.cuh): hop is
// the link from there along +e, back the one along -e, umu U_mu there.
template <typename R>
struct DualDir {
  const CField<R>& U;
  const CField<R>& Y;
  const Geo& g;
  const Coord& x;
  int mu, nu, s;
  __device__ __forceinline__ Dual<R> umu(int a, int b, bool dagger = false) const
  {
    return dlink(U, Y, site_rt(g, x, mu, a, nu, b * s), mu, dagger);
  }
  __device__ __forceinline__ Dual<R> hop(int a, int b) const
  {
    return dlink(U, Y, site_rt(g, x, mu, a, nu, b * s + (s < 0 ? -1 : 0)), nu, s < 0);
  }
  __device__ __forceinline__ Dual<R> back(int a, int b) const
  {
    return dlink(U, Y, site_rt(g, x, mu, a, nu, b * s + (s < 0 ? 0 : -1)), nu, s > 0);
  }
};

template <typename R>
__device__ __forceinline__ void dual_acc(M3<R>& S, M3<R>& dS, R w, const Dual<R>& P)
{
  axpy(S, w, P.v);
  axpy(dS, w, P.d);
}

// The staple sums S and dS of a thread, kept in shared memory (entry k at
// [k][threadIdx.x]) while its paths are walked: the dual matrices of a path
// then have the registers to themselves.
template <typename R>
struct SmemAcc {
  Cx<R> (*s)[128];
  Cx<R> (*ds)[128];
  __device__ __forceinline__ void zero()
  {
#pragma unroll
    for (int k = 0; k < 9; ++k) s[k][threadIdx.x] = ds[k][threadIdx.x] = cx<R>(R(0), R(0));
  }
  __device__ __forceinline__ void add(R w, const Dual<R>& P)
  {
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      Cx<R> a = s[k][threadIdx.x], b = ds[k][threadIdx.x];
      a.re = fma(w, P.v.e[k].re, a.re);
      a.im = fma(w, P.v.e[k].im, a.im);
      b.re = fma(w, P.d.e[k].re, b.re);
      b.im = fma(w, P.d.e[k].im, b.im);
      s[k][threadIdx.x] = a;
      ds[k][threadIdx.x] = b;
    }
  }
  __device__ __forceinline__ M3<R> S() const
  {
    M3<R> m;
#pragma unroll
    for (int k = 0; k < 9; ++k) m.e[k] = s[k][threadIdx.x];
    return m;
  }
  __device__ __forceinline__ M3<R> dS() const
  {
    M3<R> m;
#pragma unroll
    for (int k = 0; k < 9; ++k) m.e[k] = ds[k][threadIdx.x];
    return m;
  }
};

// ---- the plaquette force's pull-back ------------------------------------------
//
// With V = H W, W = M K^+ the staple of direction +nu (H = U_nu(x), M = U_mu(x+nu), K = U_nu(x+mu)) and
// W = M K, V = H^+ W that of -nu (H = U_nu(x-nu), M = U_mu(x-nu), K = U_nu(x-nu+mu)), the tangents Y of the
// links give
//   +nu: dV = Y_H V + H (Y_M W - W Y_K)
//   -nu: dV = H^+ ((Y_M - Y_H) W + M (Y_K K))
// 6 products per direction, 3 of them with an anti-Hermitian factor along +nu and 2 along -nu, where dual
// matrices (k_force_vjp_rect) take 9 full ones: the kernel is bound by the FP64 pipe, 3900 multiply-adds per link
// instead of 6600.  S and dS accumulate in shared memory, which leaves the registers to the products
// (3 blocks of 128 threads per SM).  The four directions of a site block run back to back and meet in L2.
// 16^4 FP64: 0.188 -> 0.112 ms a launch.

// An su(3) matrix by its diagonal and upper triangle; the products use that the diagonal is imaginary.
template <typename R>
struct AntiH {
  R d[3];
  Cx<R> o[3];  // (0,1), (0,2), (1,2)
};

template <typename R>
__device__ __forceinline__ Cx<R> ah_entry(const AntiH<R>& a, int i, int j)  // i != j
{
  const Cx<R> v = a.o[i + j - 1];
  return i < j ? v : cx<R>(-v.re, v.im);
}

template <typename R, typename I>
__device__ __forceinline__ AntiH<R> ld_ah(const CompLd<R, I>& Y, I site)
{
  const Cx<R>* q = Y.p + ((site >> 5) * 288 + (site & 31));
  AntiH<R> a;
  a.d[0] = ldg_cx(q).im;
  a.o[0] = ldg_cx(q + 32);
  a.o[1] = ldg_cx(q + 64);
  a.d[1] = ldg_cx(q + 32 * 4).im;
  a.o[2] = ldg_cx(q + 32 * 5);
  a.d[2] = ldg_cx(q + 32 * 8).im;
  return a;
}

// s + a b
template <typename R>
__device__ __forceinline__ M3<R> add_ah_mul(const M3<R>& s, const AntiH<R>& a, const M3<R>& b)
{
  M3<R> c;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      R re = fma(-a.d[i], b.e[3 * i + j].im, s.e[3 * i + j].re);
      R im = fma(a.d[i], b.e[3 * i + j].re, s.e[3 * i + j].im);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (k == i) continue;
        const Cx<R> v = ah_entry(a, i, k);
        re = fma(v.re, b.e[3 * k + j].re, fma(-v.im, b.e[3 * k + j].im, re));
        im = fma(v.re, b.e[3 * k + j].im, fma(v.im, b.e[3 * k + j].re, im));
      }
      c.e[3 * i + j] = cx<R>(re, im);
    }
  return c;
}

// -(b a)
template <typename R>
__device__ __forceinline__ M3<R> minus_mul_ah(const M3<R>& b, const AntiH<R>& a)
{
  M3<R> c;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      R re = a.d[j] * b.e[3 * i + j].im;
      R im = -a.d[j] * b.e[3 * i + j].re;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (k == j) continue;
        const Cx<R> v = ah_entry(a, k, j);
        re = fma(-v.re, b.e[3 * i + k].re, fma(v.im, b.e[3 * i + k].im, re));
        im = fma(-v.re, b.e[3 * i + k].im, fma(-v.im, b.e[3 * i + k].re, im));
      }
      c.e[3 * i + j] = cx<R>(re, im);
    }
  return c;
}

template <typename R>
__device__ __forceinline__ AntiH<R> ah_sub(AntiH<R> a, const AntiH<R>& b)
{
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    a.d[i] -= b.d[i];
    a.o[i].re -= b.o[i].re;
    a.o[i].im -= b.o[i].im;
  }
  return a;
}

template <typename R>
__device__ __forceinline__ M3<R> sm_ld(Cx<R> (*m)[128])
{
  M3<R> r;
#pragma unroll
  for (int k = 0; k < 9; ++k) r.e[k] = m[k][threadIdx.x];
  return r;
}

template <typename R>
__device__ __forceinline__ void sm_st(Cx<R> (*m)[128], const M3<R>& r)
{
#pragma unroll
  for (int k = 0; k < 9; ++k) m[k][threadIdx.x] = r.e[k];
}

// lambda_out = lambda_local + a (DF[Y] + [F, Y]), F the plaquette action's force; Y and lambda_local in su(3).
template <typename R, typename I>
__global__ void __launch_bounds__(128, sizeof(R) == 8 ? 3 : 4)
    k_force_vjp_plaq(Geo g, const Cx<R>* Up, const Cx<R>* Yp, const Cx<R>* lam_local, Cx<R>* lam_out, double beta, double a)
{
  const long w = (long)(blockIdx.x >> 2) * 128 + threadIdx.x;
  if (w >= g.V) return;
  const int mu = blockIdx.x & 3;
  const I s = (I)w;
  const I comp = (I)site_blocks(g.V) * 288;
  const Coord x = coord_of(g, w);
  const CompLd<R, I> Um{Up + mu * comp}, Ym{Yp + mu * comp};
  const I smu = site_stride<I>(g, mu);
  const I dmu = nb_offset<I>(sel4(x.c, mu), 1, sel4(g.d, mu), smu);
  __shared__ Cx<R> sh_s[9][128], sh_ds[9][128];
  sm_st(sh_s, m3_zero<R>());
  sm_st(sh_ds, m3_zero<R>());
#pragma unroll 1
  for (int i = 1; i < 4; ++i) {
    const int nu = (mu + i) & 3;
    const I snu = site_stride<I>(g, nu);
    const CompLd<R, I> Un{Up + nu * comp}, Yn{Yp + nu * comp};
    {
      const I y = s + nb_offset<I>(sel4(x.c, nu), 1, sel4(g.d, nu), snu);
      const M3<R> W = mul_adj(Um(y), Un(s + dmu));
      const M3<R> T = add_ah_mul(minus_mul_ah(W, ld_ah(Yn, s + dmu)), ld_ah(Ym, y), W);
      const M3<R> H = Un(s);
      sm_st(sh_ds, add_mul(sm_ld(sh_ds), H, T));
      const M3<R> V = mul(H, W);
      sm_st(sh_ds, add_ah_mul(sm_ld(sh_ds), ld_ah(Yn, s), V));
      M3<R> S = sm_ld(sh_s);
      add_to(S, V);
      sm_st(sh_s, S);
    }
    {
      const I y = s + nb_offset<I>(sel4(x.c, nu), -1, sel4(g.d, nu), snu);
      const M3<R> K = Un(y + dmu), M = Um(y);
      const M3<R> W = mul(M, K);
      M3<R> T = mul(M, add_ah_mul(m3_zero<R>(), ld_ah(Yn, y + dmu), K));
      T = add_ah_mul(T, ah_sub(ld_ah(Ym, y), ld_ah(Yn, y)), W);
      const M3<R> H = Un(y);
      sm_st(sh_ds, add_adj_mul(sm_ld(sh_ds), H, T));
      sm_st(sh_s, add_adj_mul(sm_ld(sh_s), H, W));
    }
  }
  // DF[Y] = c TA(Y (U S^+) + U dS^+), and [F, Y] by structure constants
  const M3<R> u = Um(s);
  const AntiH<R> y = ld_ah(Ym, s);
  const M3<R> P = mul_adj(u, sm_ld(sh_s));
  const M3<R> D = traceless_antiherm(add_ah_mul(mul_adj(u, sm_ld(sh_ds)), y, P));
  R f[8], d[8], yb[8], out[8], l[8];
  su3_coefs(traceless_antiherm(P), f);
  su3_coefs(D, d);
  M3<R> ym;
  ym.e[0].im = y.d[0];
  ym.e[4].im = y.d[1];
  ym.e[1] = y.o[0];
  ym.e[2] = y.o[1];
  ym.e[5] = y.o[2];
  su3_coefs(ym, yb);
  minus_ad(out, yb, f);
  su3_coefs(CField<R>{lam_local, g.V}.ld(w, mu), l);
  const R c = R(-beta / 3.0) * R(a);
#pragma unroll
  for (int k = 0; k < 8; ++k) out[k] = fma(c, out[k] + d[k], l[k]);
  WField<R>{lam_out, g.V}.st(w, mu, su3_matrix(out));
}

// ---- the same with rectangles: every path as a product of dual matrices --------

// lambda_out = lambda_local + a (DF[Y] + [F, Y]) at every link, F the force
// of GaugeAction(beta, c1) (hmc.cpp:48-75: staples (1 - 8 c1) plaq + c1 rect,
// the paths of hmc.cpp:27-46), DF[Y] its derivative along Y.
template <typename R>
__global__ void __launch_bounds__(128) k_force_vjp_rect(Geo g, const Cx<R>* Up, const Cx<R>* Yp, const Cx<R>* lam_local,
                                                        Cx<R>* lam_out, double beta, double c1, double a)
{
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= g.V) return;
  const int mu = blockIdx.y;
  const CField<R> U{Up, g.V}, Y{Yp, g.V};
  const Coord x = coord_of(g, s);
  const R cp = R(1.0 - 8.0 * c1), cr = R(c1);
  __shared__ Cx<R> sh_s[9][128], sh_ds[9][128];
  SmemAcc<R> acc{sh_s, sh_ds};
  acc.zero();
#pragma unroll 1
  for (int k = 0; k < 6; ++k) {
    const DualDir<R> d{U, Y, g, x, mu, (mu + 1 + (k >> 1)) & 3, (k & 1) ? -1 : 1};
    // plaq (nu, mu, -nu) = hop(x) U_mu(x+e) back(x+e+mu)
    acc.add(cp, dmul(dmul(d.hop(0, 0), d.umu(0, 1)), d.back(1, 1)));
    // rect1 (nu, nu, mu, -nu, -nu)
    Dual<R> C = dmul(d.hop(0, 0), d.hop(0, 1));
    C = dmul(C, d.umu(0, 2));
    C = dmul(C, d.back(1, 2));
    acc.add(cr, dmul(C, d.back(1, 1)));
    // rect2 (nu, mu, mu, -nu, -mu)
    C = dmul(d.hop(0, 0), d.umu(0, 1));
    C = dmul(C, d.umu(1, 1));
    C = dmul(C, d.back(2, 1));
    acc.add(cr, dmul(C, d.umu(1, 0, true)));
    // rect3 (-mu, nu, mu, mu, -nu)
    C = dmul(d.umu(-1, 0, true), d.hop(-1, 0));
    C = dmul(C, d.umu(-1, 1));
    C = dmul(C, d.umu(0, 1));
    acc.add(cr, dmul(C, d.back(1, 1)));
  }
  const M3<R> S = acc.S(), dS = acc.dS();
  const M3<R> u = U.ld(s, mu);
  const M3<R> y = Y.ld(s, mu);
  const M3<R> du = mul(y, u);
  const R c = R(-beta / 3.0);
  const M3<R> F = scale(c, traceless_antiherm(mul_adj(u, S)));
  const M3<R> dF = scale(c, traceless_antiherm(add_mul(mul_adj(du, S), u, adj(dS))));
  M3<R> out = CField<R>{lam_local, g.V}.ld(s, mu);
  axpy(out, R(a), dF);
  axpy(out, R(a), commutator(F, y));
  WField<R>{lam_out, g.V}.st(s, mu, traceless_antiherm(out));
}

// dexp_A(B) = sum_{k>=0} ad_A^k B / (k+1)!
template <typename R>
__device__ __forceinline__ M3<R> dexp_apply(const M3<R>& A, const M3<R>& B)
{
  M3<R> out = B, term = B;
#pragma unroll 1
  for (int k = 1; k <= 16; ++k) {
    term = scale(R(1) / R(k + 1), commutator(A, term));
    add_to(out, term);
  }
  return out;
}

// Link-local part of a stage's pull-back:
//   mu_out = eps dexp_{-eps Z}(lambda) + carry * mu_carry,   lam_local = e^{-eps Z} lambda e^{eps Z}.
// lambda counts by its su(3) part (ad_Z of the rest has none); Z and mu_carry are in su(3).  In su(3)
// coefficients a nested commutator takes 54 multiply-adds instead of 216, so the kernel is bound by
// memory: five fields, 189 MB at 16^4 in FP64:
// 0.062 -> 0.027 ms.
template <typename R>
__global__ void __launch_bounds__(128) k_flow_adj_local(long V, const Cx<R>* lam, const Cx<R>* Z, const Cx<R>* mu_carry,
                                                        double carry, double eps, Cx<R>* mu_out, Cx<R>* lam_local)
{
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  const int mu = blockIdx.y;
  R l[8], A[8], ad[8], d[8], c[8], t[8];
  su3_coefs(traceless_antiherm(CField<R>{lam, V}.ld(s, mu)), l);
  su3_coefs(CField<R>{Z, V}.ld(s, mu), A);
  // Both parts from one series of nested commutators c_k = ad_A^k lambda, A = -eps Z:
  // dexp_A(lambda) = sum_k c_k / (k+1)! and e^A lambda e^-A = sum_k c_k / k!,
  // cut once |c_k| / k! (Frobenius norms, |ad_A| <= 2 |A|) falls below
  // 2^-60 |lambda| (2^-30 in FP32), under the rounding of either sum.
  R na2 = R(0), nl2 = R(0);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    A[i] *= R(eps);  // minus_ad changes the sign
    na2 = fma(A[i], A[i], na2);
    nl2 = fma(l[i], l[i], nl2);
    c[i] = ad[i] = d[i] = l[i];
  }
  const R nad = R(2) * sqrt(R(2) * na2);
  const R tol = (sizeof(R) == 4 ? R(9.313225746154785e-10) : R(8.673617379884035e-19)) * sqrt(nl2);
  R bound = sqrt(nl2);  // bound on |c_k| / k!
#pragma unroll 1
  for (int k = 1; k <= 30 && bound > tol; ++k) {
    const R inv = R(1) / R(k), inv1 = R(1) / R(k + 1);
    minus_ad(t, A, c);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      c[i] = t[i] * inv;  // c_k / k!
      ad[i] += c[i];
      d[i] = fma(inv1, c[i], d[i]);
    }
    bound *= nad * inv;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) d[i] *= R(eps);
  if (mu_carry != nullptr && carry != 0.0) {
    su3_coefs(CField<R>{mu_carry, V}.ld(s, mu), t);
#pragma unroll
    for (int i = 0; i < 8; ++i) d[i] = fma(R(carry), t[i], d[i]);
  }
  WField<R>{mu_out, V}.st(s, mu, su3_matrix(d));
  WField<R>{lam_local, V}.st(s, mu, su3_matrix(ad));
}

// out = dexp_{-Omega}(lambda): the gradient with respect to omega of a function
// of exp(Omega) U, given its left-trivialised gradient lambda at exp(Omega) U.
template <typename R>
__global__ void k_dexp_adjoint(long V, int m, const Cx<R>* omega, const Cx<R>* lam, Cx<R>* out)
{
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  for (int mu = 0; mu < m; ++mu) {
    const M3<R> A = scale(R(-1), CField<R>{omega, V}.ld(s, mu));
    WField<R>{out, V}.st(s, mu, traceless_antiherm(dexp_apply(A, CField<R>{lam, V}.ld(s, mu))));
  }
}

// fc[x, m] = sum_a T_a basis[x, 8 m + a] and back (hmc.cpp:647-697,
// matrix-hmc.h:76-123); basis is a real field with multiplicity 8 m.
template <typename R>
__global__ void k_basis_to_matrix(long V, int m, const R* basis, Cx<R>* fc)
{
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  for (int mu = 0; mu < m; ++mu) {
    R b[8];
#pragma unroll
    for (int a = 0; a < 8; ++a) b[a] = basis[lay_index<1>(V, 8 * mu + a, 0, s)];
    const R s3 = R(0.57735026918962584) * b[7];
    M3<R> r;
    r.e[0] = cx<R>(R(0), b[2] + s3);
    r.e[4] = cx<R>(R(0), -b[2] + s3);
    r.e[8] = cx<R>(R(0), R(-2) * s3);
    r.e[1] = cx<R>(b[1], b[0]);
    r.e[2] = cx<R>(b[4], b[3]);
    r.e[3] = cx<R>(-b[1], b[0]);
    r.e[5] = cx<R>(b[6], b[5]);
    r.e[6] = cx<R>(-b[4], b[3]);
    r.e[7] = cx<R>(-b[6], b[5]);
    WField<R>{fc, V}.st(s, mu, r);
  }
}

template <typename R>
__global__ void k_matrix_to_basis(long V, int m, const Cx<R>* fc, R* basis)
{
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  for (int mu = 0; mu < m; ++mu) {
    const M3<R> x = CField<R>{fc, V}.ld(s, mu);
    R b[8];
    b[0] = x.e[1].im;
    b[1] = x.e[1].re;
    b[2] = R(0.5) * (x.e[0].im - x.e[4].im);
    b[3] = x.e[2].im;
    b[4] = x.e[2].re;
    b[5] = x.e[5].im;
    b[6] = x.e[5].re;
    b[7] = R(0.86602540378443865) * (x.e[0].im + x.e[4].im);
#pragma unroll
    for (int a = 0; a < 8; ++a) basis[lay_index<1>(V, 8 * mu + a, 0, s)] = b[a];
  }
}

template <typename R>
cudaError_t launch_force_vjp(const Geo& g, const void* U, const void* Y, const void* lam_local, void* lam_out,
                             double beta, double c1, double a, cudaStream_t st)
{
  const unsigned nb = (unsigned)((g.V + 127) / 128);
  const Cx<R>*u = (const Cx<R>*)U, *y = (const Cx<R>*)Y, *l = (const Cx<R>*)lam_local;
  if (c1 != 0.0) k_force_vjp_rect<R><<<dim3(nb, 4), 128, 0, st>>>(g, u, y, l, (Cx<R>*)lam_out, beta, c1, a);
  else if (small_offsets(g, 4)) k_force_vjp_plaq<R, int><<<4 * nb, 128, 0, st>>>(g, u, y, l, (Cx<R>*)lam_out, beta, a);
  else k_force_vjp_plaq<R, long><<<4 * nb, 128, 0, st>>>(g, u, y, l, (Cx<R>*)lam_out, beta, a);
  return cudaGetLastError();
}

template <typename R>
cudaError_t launch_flow_adj_local(long V, const void* lam, const void* Z, const void* mu_carry, double carry, double eps,
                                  void* mu_out, void* lam_local, cudaStream_t st)
{
  dim3 grid((unsigned)((V + 127) / 128), 4);
  k_flow_adj_local<R><<<grid, 128, 0, st>>>(V, (const Cx<R>*)lam, (const Cx<R>*)Z, (const Cx<R>*)mu_carry, carry, eps,
                                            (Cx<R>*)mu_out, (Cx<R>*)lam_local);
  return cudaGetLastError();
}

template <typename R>
cudaError_t launch_dexp_adjoint(long V, int m, const void* omega, const void* lam, void* out, cudaStream_t st)
{
  k_dexp_adjoint<R><<<(unsigned)((V + 127) / 128), 128, 0, st>>>(V, m, (const Cx<R>*)omega, (const Cx<R>*)lam,
                                                                 (Cx<R>*)out);
  return cudaGetLastError();
}

template <typename R>
cudaError_t launch_basis_to_matrix(long V, int m, const void* basis, void* fc, cudaStream_t st)
{
  k_basis_to_matrix<R><<<(unsigned)((V + 127) / 128), 128, 0, st>>>(V, m, (const R*)basis, (Cx<R>*)fc);
  return cudaGetLastError();
}

template <typename R>
cudaError_t launch_matrix_to_basis(long V, int m, const void* fc, void* basis, cudaStream_t st)
{
  k_matrix_to_basis<R><<<(unsigned)((V + 127) / 128), 128, 0, st>>>(V, m, (const Cx<R>*)fc, (R*)basis);
  return cudaGetLastError();
}

#define QGB_ADJ_INST(R)                                                                                          \
  template cudaError_t launch_force_vjp<R>(const Geo&, const void*, const void*, const void*, void*, double, double, \
                                           double, cudaStream_t);                                               \
  template cudaError_t launch_flow_adj_local<R>(long, const void*, const void*, const void*, double, double, void*, \
                                                void*, cudaStream_t);                                           \
  template cudaError_t launch_dexp_adjoint<R>(long, int, const void*, const void*, void*, cudaStream_t);        \
  template cudaError_t launch_basis_to_matrix<R>(long, int, const void*, void*, cudaStream_t);                  \
  template cudaError_t launch_matrix_to_basis<R>(long, int, const void*, void*, cudaStream_t);
QGB_ADJ_INST(double)
QGB_ADJ_INST(float)

}  // namespace qgb
