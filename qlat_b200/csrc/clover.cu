// clover.cu -- field-strength observables: the clover energy density and
// topological charge (wilson-flow.cpp:99-129, qcd.cpp:64-79) and the 5-loop
// improved charge (qcd.cpp:425-489, hep-lat/9701012).
//
// Leaves.  With A and B the straight lines of m links along a and n links
// along b, the four m x n leaves at x sum to C, and only C - C^+ enters.  Two
// of them start with A(x) and two end with A(x - m a), so with
//   D(y) = B(y+ma) A(y+nb)^+ B(y)^+ - B(y+ma-nb)^+ A(y-nb)^+ B(y-nb)
// (the upper minus the lower staple of A(y))
//   C - C^+ = G - G^+,   G = A(x) D(x) + D(x-ma) A(x-ma):
// 10 matrix products per plane instead of the 12 of walking four plaquettes,
// and for the larger loops 10 instead of 28 to 44, the lines of two and three
// links coming from a pass that forms them once per site (k_lines).
//
// Work split.  A block holds 64 sites and three groups of 64 threads; group p
// forms the two planes of one term of the charge, (02,13), (03,12), (23,01),
// so a thread's chain is a third of a site's work and the groups' loads of
// the same links meet in L1.  Sums are in FP64 in a fixed order.
#include <cuda_runtime.h>

#include <type_traits>

#include "gauge_common.cuh"
#include "kernels.h"

namespace qgb
{

namespace
{

constexpr int SITES = 64, GROUPS = 3, BS = SITES * GROUPS;

// An anti-Hermitian matrix: imaginary diagonal and upper triangle.
template <typename R>
struct AntiH {
  R d[3];
  Cx<R> o[3];  // (0,1), (0,2), (1,2)
};

// f (g - g^+)
template <typename R>
__device__ __forceinline__ AntiH<R> antiherm(R f, const M3<R>& g)
{
  AntiH<R> h;
#pragma unroll
  for (int i = 0; i < 3; ++i) h.d[i] = R(2) * f * g.e[4 * i].im;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int i = q == 2 ? 1 : 0, j = q == 0 ? 1 : 2;
    h.o[q] = cx<R>(f * (g.e[3 * i + j].re - g.e[3 * j + i].re), f * (g.e[3 * i + j].im + g.e[3 * j + i].im));
  }
  return h;
}

// -tr(a b)
template <typename R>
__device__ __forceinline__ R minus_tr(const AntiH<R>& a, const AntiH<R>& b)
{
  R s = R(0);
#pragma unroll
  for (int q = 0; q < 3; ++q) s = fma(a.o[q].re, b.o[q].re, fma(a.o[q].im, b.o[q].im, s));
  s *= R(2);
#pragma unroll
  for (int i = 0; i < 3; ++i) s = fma(a.d[i], b.d[i], s);
  return s;
}

// -tr(G^2) with G the traceless part of f (matrix-hmc.h:202-213)
template <typename R>
__device__ __forceinline__ R energy_of(AntiH<R> f)
{
  const R t = (f.d[0] + f.d[1] + f.d[2]) / R(3);
#pragma unroll
  for (int i = 0; i < 3; ++i) f.d[i] -= t;
  return minus_tr(f, f);
}

// s - a^+ b
template <typename R>
__device__ __forceinline__ M3<R> sub_adj_mul(const M3<R>& s, const M3<R>& a, const M3<R>& b)
{
  M3<R> c;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      R re = s.e[3 * i + j].re, im = s.e[3 * i + j].im;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        re = fma(-a.e[3 * k + i].re, b.e[3 * k + j].re, re);
        re = fma(-a.e[3 * k + i].im, b.e[3 * k + j].im, re);
        im = fma(-a.e[3 * k + i].re, b.e[3 * k + j].im, im);
        im = fma(a.e[3 * k + i].im, b.e[3 * k + j].re, im);
      }
      c.e[3 * i + j] = cx<R>(re, im);
    }
  }
  return c;
}

// acc += G at site s; m and n links: am, bn (and amm, bnn) lead m links along a (n along b) forward (backward).
// A, B: CompLd, or LineWalk.
template <typename R, typename I, typename Line>
__device__ __forceinline__ void add_leaves(M3<R>& acc, const Line& A, const Line& B, I s, I am, I amm, I bn, I bnn)
{
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    const I y = h == 0 ? s : s + amm, ya = h == 0 ? s + am : s;  // y and y + m a
    M3<R> T = mul(B(y), A(y + bn));
    M3<R> D = mul_adj(B(ya), T);
    T = mul(A(y + bnn), B(ya + bnn));
    D = sub_adj_mul(D, T, B(y + bnn));
    acc = h == 0 ? add_mul(acc, A(y), D) : add_mul(acc, D, A(y));
  }
}

// The first plane's matrix of each thread waits in shared memory while the second is formed.
template <typename R>
__device__ __forceinline__ void park(R (*sm)[BS], const AntiH<R>& f)
{
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    sm[i][threadIdx.x] = f.d[i];
    sm[3 + 2 * i][threadIdx.x] = f.o[i].re;
    sm[4 + 2 * i][threadIdx.x] = f.o[i].im;
  }
}
template <typename R>
__device__ __forceinline__ AntiH<R> parked(R (*sm)[BS])
{
  AntiH<R> f;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    f.d[i] = sm[i][threadIdx.x];
    f.o[i] = cx<R>(sm[3 + 2 * i][threadIdx.x], sm[4 + 2 * i][threadIdx.x]);
  }
  return f;
}

// The planes (a, b) of group p: 02, 13 | 03, 12 | 23, 01.
__device__ __forceinline__ void plane_of(int p, int i, int& a, int& b)
{
  a = i == 0 ? (p == 2 ? 2 : 0) : (p == 2 ? 0 : 1);
  b = i == 0 ? (p == 0 ? 2 : 3) : (p == 0 ? 3 : (p == 1 ? 2 : 1));
}

// Sum over the first 64 threads in a fixed order; thread 0 returns it.
__device__ __forceinline__ double sum_sites(double x)
{
  __shared__ double sm[2];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  if (threadIdx.x == 32) sm[1] = x;
  __syncthreads();
  const double r = threadIdx.x == 0 ? x + sm[1] : 0.0;
  __syncthreads();
  return r;
}

// E(x) = sum over planes of -tr(TA(C/4)^2) and the charge density -1/(4 pi^2) [-tr(F02 F13) + tr(F03 F12) +
// tr(F23 F01)], F = (C - C^+)/8; partials: their sums per block.
// Bound by the FP64 pipe (60 products per site) at 12 warps per SM; at most 168 registers (FP64), the first
// plane's matrix parked in shared memory.  24^3 x 48: FP64 0.56 -> 0.49 ms, FP32 0.33 -> 0.28 ms.
template <typename R, typename I>
__global__ void __launch_bounds__(BS, sizeof(R) == 8 ? 2 : 3) k_clover(Geo g, const Cx<R>* Up, R* ef, R* qf,
                                                                       double* partials)
{
  __shared__ double se[GROUPS][SITES], sq[GROUPS][SITES];
  __shared__ R sF[9][BS];
  const int p = threadIdx.x / SITES, t = threadIdx.x % SITES;
  const long w = (long)blockIdx.x * SITES + t;
  const bool valid = w < g.V;
  const long site = site_of_work(g, valid ? w : g.V - 1, SITES);
  {
    const Coord x = coord_of(g, site);
    const I comp = (I)site_blocks(g.V) * 288, s = (I)site;
    double e = 0.0, q = 0.0;
#pragma unroll 1
    for (int i = 0; i < 2; ++i) {
      int a, b;
      plane_of(p, i, a, b);
      const int xa = sel4(x.c, a), xb = sel4(x.c, b), La = sel4(g.d, a), Lb = sel4(g.d, b);
      const I sa = site_stride<I>(g, a), sb = site_stride<I>(g, b);
      M3<R> G = m3_zero<R>();
      add_leaves(G, CompLd<R, I>{Up + a * comp}, CompLd<R, I>{Up + b * comp}, s, nb_offset<I>(xa, 1, La, sa),
                       nb_offset<I>(xa, -1, La, sa), nb_offset<I>(xb, 1, Lb, sb), nb_offset<I>(xb, -1, Lb, sb));
      const AntiH<R> f = antiherm(R(0.125), G);
      e += (double)energy_of(f);
      if (i == 0) park(sF, f);
      else q = (double)minus_tr(parked(sF), f);
    }
    se[p][t] = e;
    sq[p][t] = p == 0 ? q : -q;
  }
  __syncthreads();
  double ve = 0.0, vq = 0.0;
  if (threadIdx.x < SITES) {
    const double e = se[0][t] + se[1][t] + se[2][t];
    const double q = (sq[0][t] + sq[1][t] + sq[2][t]) * (-1.0 / (4.0 * 3.141592653589793 * 3.141592653589793));
    if (valid) {
      if (ef) ef[site] = (R)e;
      if (qf) qf[site] = (R)q;
      if (in_reduce(g, site)) {
        ve = e;
        vq = q;
      }
    }
  }
  ve = sum_sites(ve);
  vq = sum_sites(vq);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = ve;
    partials[gridDim.x + blockIdx.x] = vq;
  }
}

// lines[a] = U_a(x) U_a(x+a) and lines[4 + a] = lines[a] U_a(x+2a): one thread per (site, a).
template <typename R, typename I>
__global__ void __launch_bounds__(128) k_lines(Geo g, const Cx<R>* Up, Cx<R>* lines)
{
  const long s = (long)blockIdx.x * 128 + threadIdx.x;
  if (s >= g.V) return;
  const int a = blockIdx.y;
  const I comp = (I)site_blocks(g.V) * 288;
  const CompLd<R, I> U{Up + a * comp};
  const Coord x = coord_of(g, s);
  const int xa = sel4(x.c, a), La = sel4(g.d, a);
  const I sa = site_stride<I>(g, a);
  const M3<R> d = mul(U((I)s), U((I)s + nb_offset<I>(xa, 1, La, sa)));
  const WField<R> L{lines, g.V};
  L.st(s, a, d);
  L.st(s, 4 + a, mul(d, U((I)s + nb_offset<I>(xa, 2, La, sa))));
}

// The line of m links along a direction of extent L from site y, formed from its links as k_lines does: what
// k_topology_5li reads where the device has no room for the lines (1.2 KB a site in FP64).  1092 links a site from L2
// instead of 588 lines, and the products of each line again: 16^3 x 32 2.22 ms in FP64 against 0.64, 24^3 x 48 23.2
// against 3.24.
template <typename R, typename I>
struct LineWalk {
  CompLd<R, I> U;
  int m, L;
  I stride;
  __device__ __forceinline__ M3<R> operator()(I y) const
  {
    const int x = (int)((y / stride) % L);
    M3<R> r = U(y);
#pragma unroll 1
    for (int i = 1; i < m; ++i) r = mul(r, U(y + nb_offset<I>(x, i, L, stride)));
    return r;
  }
};

// The five terms c_k / (m n)^2 q_{m x n} of the improved charge, (m, n) = (1,1), (2,2), (1,2), (1,3), (3,3), the
// unequal ones averaged with their transposes (qcd.cpp:536-568): terms (multiplicity 5) and total (multiplicity
// 1) fields, each optional, and the block sums of the terms.
// 420 products per site and the 8 of k_lines, where walking every loop link by link took 1080; 16^3 x 32,
// FP64: 2.71 -> 0.60 ms, and 0.04 ms for the lines.
template <typename R, typename I, bool LINES>
__global__ void __launch_bounds__(BS, sizeof(R) == 8 ? 2 : 3)
    k_topology_5li(Geo g, const Cx<R>* Up, const Cx<R>* lines, R* terms, R* total, double* partials)
{
  __shared__ double sq[5][GROUPS][SITES];
  __shared__ R sF[9][BS];
  const int p = threadIdx.x / SITES, t = threadIdx.x % SITES;
  const long w = (long)blockIdx.x * SITES + t;
  const bool valid = w < g.V;
  const long site = valid ? w : g.V - 1;
  {
    const Coord x = coord_of(g, site);
    const I comp = (I)site_blocks(g.V) * 288, s = (I)site;
    auto line = [&](int a, int m) {
      if constexpr (LINES) return CompLd<R, I>{(m == 1 ? Up : lines + (m == 3 ? 4 * comp : (I)0)) + a * comp};
      else return LineWalk<R, I>{CompLd<R, I>{Up + a * comp}, m, sel4(g.d, a), site_stride<I>(g, a)};
    };
#pragma unroll 1
    for (int k = 0; k < 5; ++k) {
      const int m0 = k == 1 ? 2 : (k == 4 ? 3 : 1), n0 = k == 0 ? 1 : (k == 1 || k == 2 ? 2 : 3);
      double q = 0.0;
#pragma unroll 1
      for (int i = 0; i < 2; ++i) {
        int a, b;
        plane_of(p, i, a, b);
        const int xa = sel4(x.c, a), xb = sel4(x.c, b), La = sel4(g.d, a), Lb = sel4(g.d, b);
        const I sa = site_stride<I>(g, a), sb = site_stride<I>(g, b);
        M3<R> G = m3_zero<R>();
#pragma unroll 1
        for (int h = 0; h <= (m0 != n0); ++h) {
          const int m = h == 0 ? m0 : n0, n = h == 0 ? n0 : m0;
          add_leaves(G, line(a, m), line(b, n), s, nb_offset<I>(xa, m, La, sa), nb_offset<I>(xa, -m, La, sa),
                           nb_offset<I>(xb, n, Lb, sb), nb_offset<I>(xb, -n, Lb, sb));
        }
        const AntiH<R> f = antiherm(m0 == n0 ? R(0.125) : R(0.0625), G);
        if (i == 0) park(sF, f);
        else q = (double)minus_tr(parked(sF), f);
      }
      sq[k][p][t] = p == 0 ? q : -q;
    }
  }
  __syncthreads();
  double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  if (threadIdx.x < SITES && valid) {
    const double c5 = 1.0 / 20.0;
    const double coef[5] = {(19.0 - 55.0 * c5) / 9.0, (1.0 - 64.0 * c5) / 9.0 / 16.0,
                            (-64.0 + 640.0 * c5) / 45.0 / 4.0, (1.0 / 5.0 - 2.0 * c5) / 9.0, c5 / 81.0};
    const double fac = -1.0 / (4.0 * 3.141592653589793 * 3.141592653589793);
    double tot = 0.0;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      v[k] = coef[k] * (fac * (sq[k][0][t] + sq[k][1][t] + sq[k][2][t]));
      tot += v[k];
      if (terms) terms[lay_index<1>(g.V, k, 0, site)] = (R)v[k];
    }
    if (total) total[site] = (R)tot;
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const double r = sum_sites(v[k]);
    if (threadIdx.x == 0) partials[(long)k * gridDim.x + blockIdx.x] = r;
  }
}

}  // namespace

int clover_blocks(const Geo& g) { return (int)((g.V + SITES - 1) / SITES); }

template <typename R>
cudaError_t launch_clover(const Geo& g, const void* U, void* e_field, void* q_field, double* partials,
                          cudaStream_t st)
{
  // the grid covers every site of the field: a domain's owned-box traversal does not apply here
  if (has_box(g)) return cudaErrorInvalidValue;
  Geo gk = g;  // z slabs on large lattices (the leaves reach one slice either way)
  set_slab_order(gk, SITES, (int)(18 * sizeof(R)));
  if (small_offsets(g, 4))
    k_clover<R, int><<<clover_blocks(g), BS, 0, st>>>(gk, (const Cx<R>*)U, (R*)e_field, (R*)q_field, partials);
  else
    k_clover<R, long><<<clover_blocks(g), BS, 0, st>>>(gk, (const Cx<R>*)U, (R*)e_field, (R*)q_field, partials);
  return cudaGetLastError();
}

size_t lines_bytes(const Geo& g, size_t real) { return (size_t)padded_sites(g.V) * 8 * 18 * real; }

template <typename R>
cudaError_t launch_topology_5li(const Geo& g, const void* U, void* lines, void* terms, void* total, double* partials,
                                cudaStream_t st)
{
  const dim3 grid((unsigned)((g.V + 127) / 128), 4);
  const Cx<R>* u = (const Cx<R>*)U;
  Cx<R>* l = (Cx<R>*)lines;
  auto sums = [&](auto kernel) {
    kernel<<<clover_blocks(g), BS, 0, st>>>(g, u, (const Cx<R>*)l, (R*)terms, (R*)total, partials);
  };
  if (lines == nullptr && small_offsets(g, 4)) {
    sums(k_topology_5li<R, int, false>);
  } else if (lines == nullptr) {
    sums(k_topology_5li<R, long, false>);
  } else if (small_offsets(g, 8)) {
    k_lines<R, int><<<grid, 128, 0, st>>>(g, u, l);
    sums(k_topology_5li<R, int, true>);
  } else {
    k_lines<R, long><<<grid, 128, 0, st>>>(g, u, l);
    sums(k_topology_5li<R, long, true>);
  }
  return cudaGetLastError();
}

#define QGB_CLOVER_INST(R)                                                                                        \
  template cudaError_t launch_clover<R>(const Geo&, const void*, void*, void*, double*, cudaStream_t);           \
  template cudaError_t launch_topology_5li<R>(const Geo&, const void*, void*, void*, void*, double*, cudaStream_t);
QGB_CLOVER_INST(double)
QGB_CLOVER_INST(float)

}  // namespace qgb
