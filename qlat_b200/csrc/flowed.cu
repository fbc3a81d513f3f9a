// flowed.cu -- flowed HMC with masked invertible flows (the reference's
// flowed-hmc.cpp / flowed-hmc.h), FP64 on the GPU.
//
// A flow is a list of steps (mask, mu, epsilon, flow_size).  A step updates
// the links U_mu(x) of the sites x of one mask -- even/odd sites for
// flow_size 1, even/odd 2^4 blocks for flow_size 2 -- by
//   U_mu(x) <- exp(-eps TA(U_mu(x) C(x)^+)) U_mu(x)        (exp unitarized)
// with C the plaquette staple (flow_size 1) or the staple of the rectangles
// whose short edge is the link (flow_size 2).  No updated link enters another
// updated link's staple, so a step is invertible link by link (50
// fixed-point iterations) and its Jacobian is block diagonal: per flowed link
// the 8 x 8 matrix M' = 1 - eps J(X) N in the su(3) basis, J the differential
// of exp at X = -eps TA(U C^+) and N the derivative of TA(U C^+) with respect
// to the link.  The flowed-HMC action is S(flow(U)) - sum ln det M', and its
// force is propagated back through the steps (the transpose of each step's
// Jacobian) with the force of the log-determinants added at each step.
//
// A step is one launch over the flowed links (k_flow_step).  On the way back
// that launch also forms, per flowed link, the one 3 x 3 matrix that carries
// its part of the force and of the determinant's force to the links of its
// staples, and a second launch over the links (k_flow_force_step) gathers it
// over the pairs of the reference's set_xl_nu_from_mask_mu_yl_m.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <string>
#include <utility>
#include <vector>

#include "../../include/qlat_b200.h"
#include "gauge_common.cuh"
#include "kernels.h"
#include "work_pool.h"

namespace qgb
{
void set_last_error(const std::string& msg);
void* field_data(const qgb_field* f);
int library_stream(cudaStream_t* st);
int force_on(const Geo& g, const void* U, void* out, double beta, double c1);
}

namespace
{
using namespace qgb;

// ---- masks and lattice walks (flowed-hmc.cpp:71-110) ----------------------

// Sites of mask 2 have an even sum of (x_k / size), those of mask 1 an odd one.
// The i-th masked site, x fastest (extents are multiples of 2 size).
template <int SZ>
__device__ __forceinline__ Coord masked_site(const Geo& g, long i, int mask)
{
  const int hx = g.d[0] >> 1;
  Coord x;
  const int h = (int)(i % hx);
  i /= hx;
  x.c[1] = (int)(i % g.d[1]);
  i /= g.d[1];
  x.c[2] = (int)(i % g.d[2]);
  x.c[3] = (int)(i / g.d[2]);
  const int p = (x.c[1] / SZ + x.c[2] / SZ + x.c[3] / SZ + mask) & 1;
  x.c[0] = SZ == 1 ? 2 * h + p : 4 * (h >> 1) + 2 * p + (h & 1);
  return x;
}

// whether x + a mu + b nu (nu != mu) is in the mask; a, b >= -2
template <int SZ>
__device__ __forceinline__ bool in_mask(const Coord& x, int mu, int a, int nu, int b, int mask)
{
  int p = mask;
#pragma unroll
  for (int k = 0; k < 4; ++k) p += (x.c[k] + (k == mu ? a : 0) + (k == nu ? b : 0) + 4) / SZ;
  return (p & 1) == 0;
}

// The links of the staple path (e, [e,] mu, -e, [-e]) from x, e = s nu: link i's stored site and
// direction; returns whether the path runs along it (else it enters as its adjoint).
template <int SZ>
__device__ __forceinline__ bool path_link(int i, int s, int& a, int& b, bool& along_mu)
{
  along_mu = i == SZ;
  a = i > SZ ? 1 : 0;
  if (i < SZ) {
    b = s > 0 ? i : -i - 1;
    return s > 0;
  }
  if (i == SZ) {
    b = s * SZ;
    return true;
  }
  const int j = 2 * SZ - i;  // links back: j = SZ - 1 .. 0
  b = s > 0 ? j : -j - 1;
  return s < 0;
}

// One staple of the link (x, mu): gf_plaq_staple_no_comm (qcd-acc.h:152-165) or
// gf_srect_staple_no_comm (flowed-hmc.cpp:363-380), the path of direction s nu.
template <int SZ>
__device__ __forceinline__ M3<double> path_staple(const CField<double>& U, const Geo& g, const Coord& x, int mu, int nu,
                                                  int s)
{
  M3<double> r = m3_unit<double>();
#pragma unroll 1
  for (int i = 0; i < 2 * SZ + 1; ++i) {
    int a, b;
    bool am;
    const bool fwd = path_link<SZ>(i, s, a, b, am);
    M3<double> l = U.ld(site_rt(g, x, mu, a, nu, b), am ? mu : nu);
    if (!fwd) l = adj(l);
    r = i == 0 ? l : mul(r, l);
  }
  return r;
}

// ---- kernels ----------------------------------------------------------------

// What k_flow_step does with the masked links after forming their staples C.
enum FlowMode {
  FLOW_FORWARD = 0,   // U <- exp(-eps TA(U C^+)) U (flowed-hmc.cpp:424-454), the old links kept in `old`
  FLOW_INVERSE = 1,   // the inverse, by fixed-point iterations (flowed-hmc.cpp:456-490); with `old` the staples
                      // go there and U stays (k_flow_invert)
  FLOW_LN_DET = 2,    // FLOW_FORWARD, and ln det M' of each link
  FLOW_PULL = 3,      // U <- old, then the link's part of the force's pull-back
  FLOW_PULL_DET = 4   // the same with the force of the log-determinant
};

struct FlowArgs {
  Geo g;
  Cx<double>* U;
  Cx<double>* old;  // a matrix per masked link, i fastest: old[(i / 32 * 9 + k) * 32 + i % 32]
  int mask, mu;
  double eps;
  long n;  // masked links
  int n_iter;
  double* ln_det;         // FLOW_LN_DET: one value per masked link
  const Cx<double>* Fin;  // FLOW_PULL*: the force after the step
  Cx<double>* Fout;       // FLOW_PULL*: the force before it; the masked links' entries are written here
  Cx<double>* Y;          // FLOW_PULL*: Z U of each masked link (k_flow_force_step), multiplicity 1
};

// matrix i of FlowArgs::old
__device__ __forceinline__ M3<double> ld_link(const Cx<double>* old, long i)
{
  const Cx<double>* q = old + ((i >> 5) * 9) * 32 + (i & 31);
  M3<double> m;
#pragma unroll
  for (int k = 0; k < 9; ++k) m.e[k] = q[32 * k];
  return m;
}
__device__ __forceinline__ void st_link(Cx<double>* old, long i, const M3<double>& m)
{
  Cx<double>* q = old + ((i >> 5) * 9) * 32 + (i & 31);
#pragma unroll
  for (int k = 0; k < 9; ++k) q[32 * k] = m.e[k];
}

// unitarize(exp(e TA(u c^+))) v, and the solution u of u = unitarize(exp(e TA(u c^+))) u1 by n_iter iterations
__device__ __forceinline__ M3<double> moved_link(const M3<double>& u, const M3<double>& v, const M3<double>& c, double e)
{
  M3<double> ex = exp_su3(scale(e, traceless_antiherm(mul_adj(u, c))));
  unitarize(ex);
  return mul(ex, v);
}
__device__ __forceinline__ M3<double> inverse_link(const M3<double>& u1, const M3<double>& c, double e, int n_iter)
{
  M3<double> u0 = u1;
#pragma unroll 1
  for (int it = 0; it < n_iter; ++it) u0 = moved_link(u0, u1, c, e);
  return u0;
}

constexpr int FLOW_BS = 256, FLOW_LINKS = FLOW_BS / 8, INV_BS = 32;
constexpr int PAD = 66;  // doubles between two links' 8 x 8 matrices: the four links of a warp in distinct banks

// y = A v for the 8 x 8 matrix at `a` (column-major)
__device__ __forceinline__ void mat_vec(double (&y)[8], const double* a, const double (&v)[8])
{
#pragma unroll
  for (int i = 0; i < 8; ++i) y[i] = 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k)
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const double2 t = *reinterpret_cast<const double2*>(a + 8 * k + i);
      y[i] = fma(t.x, v[k], y[i]);
      y[i + 1] = fma(t.y, v[k], y[i + 1]);
    }
}

__device__ __forceinline__ void store_col(double* a, int b, const double (&v)[8])
{
#pragma unroll
  for (int i = 0; i < 8; i += 2) *reinterpret_cast<double2*>(a + 8 * b + i) = make_double2(v[i], v[i + 1]);
}

template <int N>
__device__ __forceinline__ void sum8(double (&v)[N])  // over the 8 lanes of a link
{
#pragma unroll
  for (int k = 0; k < N; ++k)
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
}

__device__ __forceinline__ void sum8(M3<double>& m)
{
#pragma unroll
  for (int k = 0; k < 9; ++k)
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      m.e[k].re += __shfl_xor_sync(0xffffffffu, m.e[k].re, o);
      m.e[k].im += __shfl_xor_sync(0xffffffffu, m.e[k].im, o);
    }
}

// Inverse and determinant of the 8 x 8 matrix whose column b is lane b's `m` (Gauss-Jordan with
// partial pivoting over the 8 lanes of a link; the pivot order of the reference's LU, matrix.h:275-420,
// may differ, which changes only rounding).  inv: column b of the inverse.
template <bool INV>
__device__ __forceinline__ double gauss8(double (&m)[8], double (&inv)[8], int b)
{
  double det = 1.0;
  if (INV) {
#pragma unroll
    for (int i = 0; i < 8; ++i) inv[i] = i == b ? 1.0 : 0.0;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    double col[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) col[i] = __shfl_sync(0xffffffffu, m[i], j, 8);
    int p = j;
    double best = fabs(col[j]);
#pragma unroll
    for (int i = j + 1; i < 8; ++i)
      if (fabs(col[i]) > best) {
        best = fabs(col[i]);
        p = i;
      }
    if (p != j) det = -det;
#pragma unroll
    for (int i = j + 1; i < 8; ++i)
      if (i == p) {
        double t = col[j];
        col[j] = col[i];
        col[i] = t;
        t = m[j];
        m[j] = m[i];
        m[i] = t;
        if (INV) {
          t = inv[j];
          inv[j] = inv[i];
          inv[i] = t;
        }
      }
    det *= col[j];
    // a zero pivot is a zero determinant (and no inverse)
    const double r = !INV && col[j] == 0.0 ? 0.0 : 1.0 / col[j];
    m[j] *= r;
    if (INV) inv[j] *= r;
#pragma unroll
    for (int i = INV ? 0 : j + 1; i < 8; ++i) {
      if (i == j) continue;
      m[i] = fma(-col[i], m[j], m[i]);
      if (INV) inv[i] = fma(-col[i], inv[j], inv[i]);
    }
  }
  return det;
}

// One step of a flow, one launch.  Eight lanes per masked link, 32 links per block.
//
// The six staples of a link go to six of its lanes (a link's path is a chain of 2 or 4 dependent
// products; one thread per link left 4096 links on 8^3 x 16 far short of filling the GPU) and are
// added by shuffles.  No updated link enters another updated link's staple, so the update is in place.
//
// The 8 x 8 matrices of the Jacobian M' = 1 - eps J(X) N (flowed-hmc.cpp:926-955, 1011-1025,
// 1117-1162) live one column per lane in registers.  With B = -ad X, applied by minus_ad:
//   J(X) = sum_k B^k / (k+1)!  from the powers B^k e_b of each lane's own unit vector,
//   the derivative of J along f[e] traced with W = eps^2 N M'^-1: tr(f[e] G),
//     G = sum_k S_k / (k+1)!, S_{k+1} = B S_k + W B^k, S_1 = W, also column by column,
// both the reference's order-20 polynomials, cut once the omitted terms are below 2^-58 of the sum.
// One thread per link held all of it in local memory and differentiated J eight times over: 2.57 ms
// a step on 8^3 x 16 (with the staple's own launch, 2.58), against 35 us (size 1) and 27 us (size 2) here.
// At 4096 links (1024 warps: 8 on each of 128 SMs) it is bound by the latency of its chains, not by FP64 rate.
template <int SZ, int MODE>
__global__ void __launch_bounds__(FLOW_BS) k_flow_step(FlowArgs a)
{
  constexpr bool PULL = MODE == FLOW_PULL || MODE == FLOW_PULL_DET;
  constexpr bool DET = MODE == FLOW_LN_DET || MODE == FLOW_PULL_DET;
  __shared__ __align__(16) double sA[DET ? FLOW_LINKS * PAD : 2], sB[DET ? FLOW_LINKS * PAD : 2];
  __shared__ Cx<double> sC[PULL ? 1 : 9][FLOW_LINKS];
  const int b = threadIdx.x & 7, w = threadIdx.x >> 3;
  const long i0 = (long)blockIdx.x * FLOW_LINKS + w;
  const long i = i0 < a.n ? i0 : a.n - 1;  // every lane stays for the shuffles
  const Geo& g = a.g;
  const int mu = a.mu;
  const Coord x = masked_site<SZ>(g, i, a.mask);
  const long s = site_rt(g, x, 0, 0, 1, 0);
  const CField<double> U{a.U, g.V};
  const WField<double> Uw{a.U, g.V};
  M3<double> c = m3_zero<double>();
  if (b < 6) c = path_staple<SZ>(U, g, x, mu, (mu + 1 + (b >> 1)) & 3, b & 1 ? -1 : 1);
  sum8(c);
  M3<double> u;
  if (PULL) {
    u = ld_link(a.old, i);
    if (b == 0 && i0 < a.n) Uw.st(s, mu, u);  // nobody's staple of this step reads it
  } else {
    u = Uw.ld(s, mu);
  }
  if constexpr (DET || PULL) {
    const M3<double> uc = mul_adj(u, c);
    const M3<double> xm = scale(-a.eps, traceless_antiherm(uc));
    double xb[8];
    su3_coefs(xm, xb);
    double nrm = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) nrm = fma(xb[k], xb[k], nrm);
    nrm = 2.8284271247461903 * sqrt(nrm);  // |ad X| <= 2 |X| <= 2 sqrt(2) |x| (Frobenius)
    double eb[8], q[8], jb[8], xp[8], t[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) q[k] = jb[k] = xp[k] = eb[k] = k == b ? 1.0 : 0.0;
    // columns of J(X) and of exp(-ad X)
    double bound = 1.0;
#pragma unroll 1
    for (int k = 1; k <= 20; ++k) {
      const double inv = 1.0 / k, inv1 = 1.0 / (k + 1);
      minus_ad(t, xb, q);
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        q[m] = t[m] * inv;
        xp[m] += q[m];
        jb[m] = fma(q[m], inv1, jb[m]);
      }
      bound *= nrm * inv;
      if (2.0 * bound * nrm < 3.4e-18 * (k + 1) && nrm < 0.5 * (k + 2)) break;
    }
    double nb[8], mp[8], minv[8], ft[8];
    M3<double> Q = m3_zero<double>();
    if constexpr (DET) {
      su3_coefs(traceless_antiherm(mul(su3_matrix(eb), uc)), nb);
      double* A = sA + w * PAD;
      double* Bm = sB + w * PAD;
      store_col(A, b, jb);
      store_col(Bm, b, nb);
      __syncwarp();
      mat_vec(t, A, nb);
#pragma unroll
      for (int k = 0; k < 8; ++k) mp[k] = fma(-a.eps, t[k], eb[k]);
      const double det = gauss8<MODE == FLOW_PULL_DET>(mp, minv, b);
      if constexpr (MODE == FLOW_LN_DET) {
        if (b == 0 && i0 < a.n) a.ln_det[i] = log(det);
      } else {
        __syncwarp();
        store_col(A, b, minv);
        __syncwarp();
        double wb[8], sb[8], gb[8], kb[8];
        mat_vec(wb, Bm, minv);
        mat_vec(kb, A, jb);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          wb[k] *= a.eps * a.eps;
          kb[k] *= -a.eps;
        }
        __syncwarp();
        store_col(Bm, b, wb);
        __syncwarp();
        // s_k = S_k / (k+1)! e_b and q_k = B^k / k! e_b
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          gb[k] = sb[k] = 0.5 * wb[k];
          q[k] = eb[k];
        }
        bound = 1.0;
#pragma unroll 1
        for (int k = 1; k < 20; ++k) {
          const double inv = 1.0 / k, i1 = 1.0 / (k + 1), i2 = 1.0 / (k + 2);
          minus_ad(t, xb, q);
#pragma unroll
          for (int m = 0; m < 8; ++m) q[m] = t[m] * inv;
          minus_ad(t, xb, sb);
          double v[8];
          mat_vec(v, Bm, q);
#pragma unroll
          for (int m = 0; m < 8; ++m) {
            sb[m] = fma(t[m], i2, v[m] * (i1 * i2));
            gb[m] += sb[m];
          }
          // |S_{k+1}| / (k+2)! <= (k+1) |B|^k |W| / (k+2)!
          bound *= nrm * inv;
          if (2.0 * bound * nrm < 3.4e-18 * (k + 1) && nrm < 0.5 * (k + 2)) break;
        }
        // e2dj[e] = tr(f[e] G) = -sum_b (2 f (e_b, G e_b))_e
        minus_ad(ft, eb, gb);
#pragma unroll
        for (int k = 0; k < 8; ++k) ft[k] *= -0.5;
        Q = scale(0.5, mul(su3_matrix(eb), su3_matrix(kb)));
      }
    }
    if constexpr (PULL) {
      // Z = -W + (E + Q) / 2: W = eps (J(X) F) . T, E = e2dj . T, Q = sum_cb K_cb T_b T_c with K = -eps M'^-1 J(X)
      double fb[8];
      su3_coefs(CField<double>{a.Fin, g.V}.ld(s, mu), fb);
      double fbb = 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k) fbb = k == b ? fb[k] : fbb;
      double z[8], r[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        z[k] = -a.eps * jb[k] * fbb;
        if (DET) z[k] += ft[k];
        r[k] = xp[k] * fbb;
      }
      sum8(z);
      sum8(r);
      M3<double> Z = su3_matrix(z);
      if constexpr (DET) {
        sum8(Q);
        add_to(Z, Q);
      }
      // the link's own entry: Ad_{exp(-X)} F + TA(U C^+ Z); Y = Z U for the links of its staples
      if (i0 < a.n) {
        if (b == 0) WField<double>{a.Y, g.V}.st(s, 0, mul(Z, u));
        if (b == 1) {
          M3<double> f = su3_matrix(r);
          add_to(f, traceless_antiherm(mul(uc, Z)));
          WField<double>{a.Fout, g.V}.st(s, mu, f);
        }
      }
    }
  }
  if constexpr (!PULL) {
    // the block's links, one per lane of its first warp
    if (b == 0) {
#pragma unroll
      for (int k = 0; k < 9; ++k) sC[k][w] = c.e[k];
    }
    __syncthreads();
    if (threadIdx.x >= FLOW_LINKS) return;
    const long j = (long)blockIdx.x * FLOW_LINKS + threadIdx.x;
    if (j >= a.n) return;
    const Coord xj = masked_site<SZ>(g, j, a.mask);
    const long sj = site_rt(g, xj, 0, 0, 1, 0);
    M3<double> cj;
#pragma unroll
    for (int k = 0; k < 9; ++k) cj.e[k] = sC[k][threadIdx.x];
    if (MODE == FLOW_INVERSE && a.old != nullptr) {
      st_link(a.old, j, cj);
      return;
    }
    const M3<double> u1 = Uw.ld(sj, mu);
    if (a.old != nullptr) st_link(a.old, j, u1);
    Uw.st(sj, mu, MODE == FLOW_INVERSE ? inverse_link(u1, cj, a.eps, a.n_iter) : moved_link(u1, u1, cj, -a.eps));
  }
}

// The inverse of a step from the staples in a.old: one thread per masked link, in a launch of its own
// (qgb_gf_flow_inv).
template <int SZ>
__global__ void __launch_bounds__(INV_BS) k_flow_invert(FlowArgs a)
{
  const long j = (long)blockIdx.x * INV_BS + threadIdx.x;
  if (j >= a.n) return;
  const long s = site_rt(a.g, masked_site<SZ>(a.g, j, a.mask), 0, 0, 1, 0);
  const WField<double> Uw{a.U, a.g.V};
  Uw.st(s, a.mu, inverse_link(Uw.ld(s, a.mu), ld_link(a.old, j), a.eps, a.n_iter));
}

// The part of the force's pull-back that reaches the link (y, nu) through a staple (flowed-hmc.cpp:596-777,
// 1059-1091, 1164-1232, 1366-1427): a masked link (x, mu) whose staple path l_1 ... l_n holds (y, nu) as
// its n-th link gives TA(uc_post Z uc_pre), which with Y = Z U is
//   -(l_1 .. l_{n-1})^+ Y (l_n .. )^+ for a link the path runs along, +(l_1 .. l_n)^+ Y (l_{n+1} ..)^+ else.
// (In the su(3) basis this is the sum over a of w_a n_mat(a, .) of the reference, with basis_a(TA(M)) =
// -tr(T_a M)/2 moving the two factors around the trace.)  x = y + a mu + b nu in the staple's plane.
template <int SZ>
__device__ __forceinline__ void pull_path(M3<double>& acc, const CField<double>& U, const CField<double>& Y,
                                          const Geo& g, const Coord& y, int mu, int nu, int a0, int b0, int s, int n)
{
  M3<double> m = Y.ld(site_rt(g, y, mu, a0, nu, b0), 0);
  int a, b;
  bool am;
  const bool along = path_link<SZ>(n, s, a, b, am);
  const int cut = along ? n : n + 1;
  auto link = [&](int i) {  // l_i^+
    const bool fwd = path_link<SZ>(i, s, a, b, am);
    M3<double> l = U.ld(site_rt(g, y, mu, a0 + a, nu, b0 + b), am ? mu : nu);
    return fwd ? adj(l) : l;
  };
#pragma unroll 1
  for (int i = 0; i < cut; ++i) m = mul(link(i), m);
#pragma unroll 1
  for (int i = 2 * SZ; i >= cut; --i) m = mul(m, link(i));
  axpy(acc, along ? -1.0 : 1.0, m);
}

// Fout at every link but the masked ones (k_flow_step writes those): Fin plus what the staples pull back.
// One thread per link; the pairs of set_xl_nu_from_mask_mu_yl_m (flowed-hmc.cpp:191-360) as the two masked
// sites among the 2 SZ positions each side of the link allows.  2 SZ + 1 products of 3 x 3 matrices per
// pair, no 8 x 8 ones: 761 us a step on 8^3 x 16 before, 16 us (size 1) and 34 us (size 2) now.
template <int SZ>
__global__ void __launch_bounds__(128) k_flow_force_step(Geo g, const Cx<double>* Up, const Cx<double>* Yp,
                                                         const Cx<double>* Finp, Cx<double>* Foutp, int mask, int mu)
{
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= g.V) return;
  const int nu = blockIdx.y;
  const Coord y = coord_of(g, s);
  const CField<double> U{Up, g.V}, Y{Yp, g.V};
  M3<double> acc = m3_zero<double>();
  if (nu == mu) {
    if (in_mask<SZ>(y, 0, 0, 1, 0, mask)) return;
#pragma unroll 1
    for (int k = 0; k < 6; ++k) {
      const int d = (mu + 1 + (k >> 1)) & 3, e = k & 1 ? -1 : 1;
      pull_path<SZ>(acc, U, Y, g, y, mu, d, 0, -SZ * e, e, SZ);
    }
  } else {
#pragma unroll 1
    for (int side = 0; side < 2; ++side) {
      // the path leaves along (links 0 .. SZ - 1, from x) or returns to (links SZ + 1 .. 2 SZ, at x + mu) this link
      int left = SZ;
#pragma unroll 1
      for (int d = 1 - SZ; d <= SZ && left > 0; ++d) {
        if (!in_mask<SZ>(y, mu, -side, nu, d, mask)) continue;
        --left;
        const int s2 = d <= 0 ? 1 : -1;
        const int r = d <= 0 ? -d : d - 1;  // links between x and this one
        pull_path<SZ>(acc, U, Y, g, y, mu, nu, -side, d, s2, side == 0 ? r : 2 * SZ - r);
      }
    }
  }
  M3<double> f = traceless_antiherm(acc);
  add_to(f, CField<double>{Finp, g.V}.ld(s, nu));
  WField<double>{Foutp, g.V}.st(s, nu, f);
}

__global__ void __launch_bounds__(1024) k_sum_links(long n, const double* v, double* out)
{
  // one block per step: fixed-order sum of its links' values
  v += (size_t)blockIdx.x * n;
  out += blockIdx.x;
  __shared__ double sm[1024];
  double t[4] = {0.0, 0.0, 0.0, 0.0};
  for (long i = threadIdx.x; i < n; i += 4096)
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (i + 1024 * k < n) t[k] += v[i + 1024 * k];
  sm[threadIdx.x] = (t[0] + t[1]) + (t[2] + t[3]);
  __syncthreads();
  for (int w = 512; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) sm[threadIdx.x] += sm[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sm[0];
}

// ---- host side --------------------------------------------------------------

int ffail(int code, const std::string& m)
{
  qgb::set_last_error(m);
  return code;
}

#define FL_CUDA(expr)                                                                                        \
  do {                                                                                                       \
    cudaError_t e_ = (expr);                                                                                 \
    if (e_ != cudaSuccess) return ffail(QGB_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e_)); \
  } while (0)
#define FL_RC(expr)              \
  do {                           \
    int r_ = (expr);             \
    if (r_ != QGB_OK) return r_; \
  } while (0)

struct FlowCtx {
  Geo g;
  cudaStream_t st = nullptr;
  long V = 0;
  size_t bytes = 0;      // one gauge field
  long links = 0;        // links that one step moves
  size_t old_bytes = 0;  // those links of one step, kept (FlowArgs::old)
};

int check_steps(const Geo& g, const qgb_flow_step* steps, int n)
{
  if (n < 0 || (n > 0 && !steps)) return ffail(QGB_ERR_INVALID_ARG, "flowed: bad flow-step list");
  for (int i = 0; i < n; ++i) {
    const qgb_flow_step& f = steps[i];
    if ((f.mask != 1 && f.mask != 2) || f.mu < 0 || f.mu > 3 || (f.flow_size != 1 && f.flow_size != 2))
      return ffail(QGB_ERR_INVALID_ARG, "flowed: a flow step needs mask 1 or 2, mu 0..3, flow_size 1 or 2");
    for (int k = 0; k < 4; ++k)
      if (g.d[k] % (2 * f.flow_size) != 0)
        return ffail(QGB_ERR_BAD_GEOMETRY, "flowed: each lattice extent must be a multiple of 2 * flow_size");
  }
  return QGB_OK;
}

int setup(FlowCtx& c, const qgb_field* gf, int32_t n, const qgb_flow_step* steps)
{
  int32_t ts[4], mult = 0, kind = 0, prec = 0;
  FL_RC(qgb_field_info(gf, ts, &mult, &kind, &prec));
  if (kind != QGB_KIND_COLOR_MATRIX || mult != 4 || prec != QGB_F64)
    return ffail(QGB_ERR_MISMATCH, "flowed: the gauge field must be an FP64 color-matrix field of multiplicity 4");
  for (int k = 0; k < 4; ++k) c.g.d[k] = ts[k];
  c.g.V = (long)ts[0] * ts[1] * ts[2] * ts[3];
  c.V = c.g.V;
  c.bytes = (size_t)padded_sites(c.V) * 72 * sizeof(double);
  c.links = c.V / 2;
  c.old_bytes = (size_t)padded_sites(c.links) * 18 * sizeof(double);
  FL_RC(qgb::library_stream(&c.st));
  return check_steps(c.g, steps, n);
}

int check_output(const qgb_field* gf)
{
  int32_t prec = 0;
  FL_RC(qgb_field_info(gf, nullptr, nullptr, nullptr, &prec));
  if (prec != QGB_F64) return ffail(QGB_ERR_MISMATCH, "flowed: the flowed gauge field must be FP64");
  return QGB_OK;
}

FlowArgs flow_args(const FlowCtx& c, void* U, const qgb_flow_step& f)
{
  FlowArgs a;
  memset((void*)&a, 0, sizeof(a));
  a.g = c.g;
  a.U = (Cx<double>*)U;
  a.mask = f.mask;
  a.mu = f.mu;
  a.eps = f.epsilon;
  a.n = c.links;
  a.n_iter = 50;
  return a;
}

template <int MODE>
int launch_flow_step(const FlowCtx& c, const FlowArgs& a, int flow_size)
{
  const unsigned grid = (unsigned)((c.links + FLOW_LINKS - 1) / FLOW_LINKS);
  if (flow_size == 1) k_flow_step<1, MODE><<<grid, FLOW_BS, 0, c.st>>>(a);
  else k_flow_step<2, MODE><<<grid, FLOW_BS, 0, c.st>>>(a);
  FL_CUDA(cudaGetLastError());
  return QGB_OK;
}

}  // namespace

extern "C" {

int qgb_flow_info_step(const uint32_t rs[24], double epsilon, double epsilon2, int32_t two_eps, qgb_flow_step* out,
                       int32_t* n_out)
{
  if (!rs || !out || !n_out) return ffail(QGB_ERR_INVALID_ARG, "qgb_flow_info_step: null argument");
  // mk_flow_info_step (flowed-hmc.cpp:21-69); random_permute (rng-state.h:85-97)
  auto permute = [](std::vector<qgb_flow_step>& v, const uint32_t* r) {
    uint32_t st[24];
    memcpy(st, r, sizeof(st));
    const long size = (long)v.size();
    for (long k = 0; k < size; ++k) {
      const long kk = (long)(qgb::rng_host_rand_gen(st) % (uint64_t)(size - k));
      std::swap(v[k], v[k + kk]);
    }
  };
  auto split = [&](const char* s, uint32_t* o) { return qgb::rng_host_split(o, rs, s); };
  std::vector<qgb_flow_step> fi;
  if (!two_eps) {
    for (int mu = 3; mu >= 0; --mu) {
      fi.push_back({2, mu, epsilon, 1});
      fi.push_back({1, mu, epsilon, 1});
    }
    permute(fi, rs);
  } else {
    std::vector<std::vector<qgb_flow_step>> g1(4), g2(4);
    for (int mu = 3; mu >= 0; --mu) {
      if (epsilon != 0.0) {
        g1[mu].push_back({2, mu, epsilon, 1});
        g1[mu].push_back({1, mu, epsilon, 1});
      }
      if (epsilon2 != 0.0) {
        g2[mu].push_back({2, mu, epsilon2, 2});
        g2[mu].push_back({1, mu, epsilon2, 2});
      }
    }
    for (int i = 0; i < 4; ++i) {
      uint32_t r1[24], r2[24];
      const std::string s1 = "fi1s-" + std::to_string(i), s2 = "fi2s-" + std::to_string(i);
      if (!split(s1.c_str(), r1) || !split(s2.c_str(), r2)) return ffail(QGB_ERR_INVALID_ARG, "qgb_flow_info_step: split");
      permute(g1[i], r1);
      permute(g2[i], r2);
      g1[i].insert(g1[i].end(), g2[i].begin(), g2[i].end());
    }
    // random_permute of the four groups with rs itself
    uint32_t st[24];
    memcpy(st, rs, sizeof(st));
    for (long k = 0; k < 4; ++k) {
      const long kk = (long)(qgb::rng_host_rand_gen(st) % (uint64_t)(4 - k));
      std::swap(g1[k], g1[k + kk]);
    }
    for (int i = 0; i < 4; ++i) fi.insert(fi.end(), g1[i].begin(), g1[i].end());
  }
  if ((int)fi.size() > 16) return ffail(QGB_ERR_INVALID_ARG, "qgb_flow_info_step: too many steps");
  for (size_t i = 0; i < fi.size(); ++i) out[i] = fi[i];
  *n_out = (int32_t)fi.size();
  return QGB_OK;
}

int qgb_gf_flow(qgb_field* gf, const qgb_field* gf0, const qgb_flow_step* steps, int32_t n)
{
  FlowCtx c;
  FL_RC(setup(c, gf0, n, steps));
  FL_RC(check_output(gf));
  FL_RC(qgb_field_copy(gf, gf0));
  void* U = qgb::field_data(gf);
  for (int i = 0; i < n; ++i) FL_RC(launch_flow_step<FLOW_FORWARD>(c, flow_args(c, U, steps[i]), steps[i].flow_size));
  return QGB_OK;
}

int qgb_gf_flow_inv(qgb_field* gf, const qgb_field* gf1, const qgb_flow_step* steps, int32_t n)
{
  FlowCtx c;
  FL_RC(setup(c, gf1, n, steps));
  FL_RC(check_output(gf));
  FL_RC(qgb_field_copy(gf, gf1));
  void* U = qgb::field_data(gf);
  // 50 exponentials a link.  In the tail of k_flow_step they are one warp's work of a block's eight, which holds as
  // long as no SM has a second block (8 steps of 4096 links: 0.84 ms, and 0.94 with a launch of their own); beyond
  // that they go one thread per link in warps of their own (6144 links: 0.91 ms against 1.61, 16^4: 1.46 against
  // 5.52).
  int dev = 0, sms = 0;
  FL_CUDA(cudaGetDevice(&dev));
  FL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  WorkBuf C;
  if (c.links > (long)FLOW_LINKS * sms) FL_CUDA(C.alloc(c.old_bytes, c.st));
  for (int i = n - 1; i >= 0; --i) {
    FlowArgs a = flow_args(c, U, steps[i]);
    a.old = (Cx<double>*)C.p;
    FL_RC(launch_flow_step<FLOW_INVERSE>(c, a, steps[i].flow_size));
    if (C.p == nullptr) continue;
    const unsigned grid = (unsigned)((c.links + INV_BS - 1) / INV_BS);
    if (steps[i].flow_size == 1) k_flow_invert<1><<<grid, INV_BS, 0, c.st>>>(a);
    else k_flow_invert<2><<<grid, INV_BS, 0, c.st>>>(a);
    FL_CUDA(cudaGetLastError());
  }
  return QGB_OK;
}

int qgb_gf_flow_and_ln_det_node(qgb_field* gf, const qgb_field* gf0, const qgb_flow_step* steps, int32_t n,
                                double* ln_det)
{
  FlowCtx c;
  FL_RC(setup(c, gf0, n, steps));
  if (!ln_det) return ffail(QGB_ERR_INVALID_ARG, "qgb_gf_flow_and_ln_det_node: null output");
  FL_RC(check_output(gf));
  FL_RC(qgb_field_copy(gf, gf0));
  WorkBuf L, S;
  FL_CUDA(L.alloc((size_t)c.links * sizeof(double) * (n > 0 ? n : 1), c.st));
  FL_CUDA(S.alloc((size_t)(n > 0 ? n : 1) * sizeof(double), c.st));
  void* U = qgb::field_data(gf);
  for (int i = 0; i < n; ++i) {
    FlowArgs a = flow_args(c, U, steps[i]);
    a.ln_det = (double*)L.p + (size_t)i * c.links;
    FL_RC(launch_flow_step<FLOW_LN_DET>(c, a, steps[i].flow_size));
  }
  std::vector<double> sums((size_t)(n > 0 ? n : 1), 0.0);
  if (n > 0) {
    k_sum_links<<<n, 1024, 0, c.st>>>(c.links, (const double*)L.p, (double*)S.p);
    FL_CUDA(cudaGetLastError());
    FL_CUDA(cudaMemcpyAsync(sums.data(), S.p, n * sizeof(double), cudaMemcpyDeviceToHost, c.st));
  }
  FL_CUDA(cudaStreamSynchronize(c.st));
  double t = 0.0;
  for (int i = 0; i < n; ++i) t += sums[i];
  *ln_det = t;
  return QGB_OK;
}

int qgb_gf_hamilton_flowed_node(const qgb_field* gf0, double beta, double c1, const qgb_flow_step* steps, int32_t n,
                                double* flowed_action, double* ln_det)
{
  int32_t ts[4];
  FL_RC(qgb_field_info(gf0, ts, nullptr, nullptr, nullptr));
  qgb_field* gf = nullptr;
  FL_RC(qgb_field_create(&gf, ts, 4, QGB_KIND_COLOR_MATRIX, QGB_F64));
  double ld = 0.0, act = 0.0;
  int rc = qgb_gf_flow_and_ln_det_node(gf, gf0, steps, n, &ld);
  if (rc == QGB_OK) rc = qgb_gf_hamilton_node(gf, beta, c1, &act);
  qgb_field_destroy(gf);
  if (rc != QGB_OK) return rc;
  if (flowed_action) *flowed_action = act;
  if (ln_det) *ln_det = ld;
  return QGB_OK;
}

}  // extern "C"

namespace
{
// The force on gf0 of a force F on the flowed field, propagated back through
// the steps with (with_det) or without the log-determinants' force.  F is the
// action's force on the flowed field (pre == nullptr) or the given field.
int flowed_force(qgb_field* gm_force, const qgb_field* gf0, const qgb_field* pre, double beta, double c1,
                 const qgb_flow_step* steps, int32_t n, int32_t with_det)
{
  FlowCtx c;
  FL_RC(setup(c, gf0, n, steps));
  int32_t ts[4], mult = 0, kind = 0, prec = 0;
  FL_RC(qgb_field_info(gm_force, ts, &mult, &kind, &prec));
  if (kind != QGB_KIND_COLOR_MATRIX || mult != 4 || prec != QGB_F64 || ts[0] != c.g.d[0] || ts[1] != c.g.d[1] ||
      ts[2] != c.g.d[2] || ts[3] != c.g.d[3])
    return ffail(QGB_ERR_MISMATCH, "flowed: the force must be an FP64 color-matrix field of multiplicity 4 on the "
                                   "gauge field's lattice");
  // one work field: the flow runs in it and keeps the links that each step replaces (an eighth of the field), and
  // the way back puts them in place again
  WorkBuf G, old, Y, F2;
  FL_CUDA(G.alloc(c.bytes, c.st));
  FL_CUDA(old.alloc(c.old_bytes * n, c.st));
  FL_CUDA(Y.alloc(c.bytes / 4, c.st));
  FL_CUDA(F2.alloc(c.bytes, c.st));
  auto old_of = [&](int i) { return (Cx<double>*)((char*)old.p + c.old_bytes * i); };
  FL_CUDA(cudaMemcpyAsync(G.p, qgb::field_data(gf0), c.bytes, cudaMemcpyDeviceToDevice, c.st));
  for (int i = 0; i < n; ++i) {
    FlowArgs a = flow_args(c, G.p, steps[i]);
    a.old = old_of(i);
    FL_RC(launch_flow_step<FLOW_FORWARD>(c, a, steps[i].flow_size));
  }
  // The steps alternate between the caller's force and F2 so that the last one writes the caller's: F2 holds
  // words of earlier calls in its padding, and a field's padding is zero.
  void* F = qgb::field_data(gm_force);
  void *in = n % 2 == 0 ? F : F2.p, *out = n % 2 == 0 ? F2.p : F;
  if (pre) {
    FL_RC(qgb_field_copy(gm_force, pre));
    if (in != F) FL_CUDA(cudaMemcpyAsync(in, F, c.bytes, cudaMemcpyDeviceToDevice, c.st));
  } else {
    FL_RC(qgb::force_on(c.g, G.p, in, beta, c1));  // the action's force on the flowed field (hmc.cpp:466-490)
  }
  // back through the steps (set_gm_force_propagated_det_from_flow, flowed-hmc.cpp:1456-1477)
  for (int i = n - 1; i >= 0; --i) {
    FlowArgs a = flow_args(c, G.p, steps[i]);
    a.old = old_of(i);
    a.Fin = (const Cx<double>*)in;
    a.Fout = (Cx<double>*)out;
    a.Y = (Cx<double>*)Y.p;
    if (with_det) FL_RC(launch_flow_step<FLOW_PULL_DET>(c, a, steps[i].flow_size));
    else FL_RC(launch_flow_step<FLOW_PULL>(c, a, steps[i].flow_size));
    const dim3 grid((unsigned)((c.V + 127) / 128), 4);
    if (steps[i].flow_size == 1)
      k_flow_force_step<1><<<grid, 128, 0, c.st>>>(c.g, a.U, a.Y, a.Fin, a.Fout, a.mask, a.mu);
    else
      k_flow_force_step<2><<<grid, 128, 0, c.st>>>(c.g, a.U, a.Y, a.Fin, a.Fout, a.mask, a.mu);
    FL_CUDA(cudaGetLastError());
    std::swap(in, out);
  }
  return QGB_OK;
}
}  // namespace

extern "C" {

int qgb_set_gm_force_flowed(qgb_field* gm_force, const qgb_field* gf0, double beta, double c1,
                            const qgb_flow_step* steps, int32_t n, int32_t with_det)
{
  return flowed_force(gm_force, gf0, nullptr, beta, c1, steps, n, with_det);
}

int qgb_set_gm_force_flowed_no_det(qgb_field* gm_force, const qgb_field* gm_force_pre, const qgb_field* gf0,
                                   const qgb_flow_step* steps, int32_t n)
{
  if (!gm_force_pre) return ffail(QGB_ERR_INVALID_ARG, "qgb_set_gm_force_flowed_no_det: null force");
  return flowed_force(gm_force, gf0, gm_force_pre, 0.0, 0.0, steps, n, 0);
}

}  // extern "C"
