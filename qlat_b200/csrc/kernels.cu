// kernels.cu -- CUDA kernels of the pure-gauge hot path for sm_100a.
//
// Memory layout in HBM (gauge_common.cuh): sites in the reference's order (x
// fastest, coordinate.h:182-188) cut into blocks of 32; entry k of the 3x3
// matrix of component mu at site s is Cx<R>[((mu * nblk + s / 32) * 9 + k) *
// 32 + s % 32].  A warp touching 32 consecutive sites reads one fully coalesced
// 512-byte (FP64) or 256-byte (FP32) segment per matrix entry.  Neighbour
// links come through L1/L2; the lattice is periodic.
//
// Kernels use one thread per link (site, mu) for link-local work and force
// evaluation, and one thread per site for the site reductions.  Reductions
// accumulate in FP64 whatever the storage precision, then reduce in a fixed
// order (warp shuffles, block, then one block over the partials), so results
// are deterministic run to run.
#include <cuda_runtime.h>
#include <type_traits>
#include <stdint.h>
#include <string.h>

#include "gauge_common.cuh"
#include "kernels.h"
#include "rng.cuh"
#include "su3.cuh"

namespace qgb
{

ShaConst qgb_sha_host;

// ------------------------------------------------------------------------
// constants

static void sha_const_compute(ShaConst& c)
{
  int primes[64];
  int n = 0;
  for (int v = 2; n < 64; ++v) {
    bool p = true;
    for (int d = 2; d * d <= v; ++d)
      if (v % d == 0) {
        p = false;
        break;
      }
    if (p) primes[n++] = v;
  }
  // first 32 fractional bits of cube roots (k) and square roots (h0) of primes
  for (int i = 0; i < 64; ++i) {
    const unsigned __int128 target = ((unsigned __int128)primes[i]) << 96;
    uint64_t lo = 0, hi = (uint64_t)1 << 36;
    while (hi - lo > 1) {
      const uint64_t mid = (lo + hi) / 2;
      if ((unsigned __int128)mid * mid * mid <= target) lo = mid; else hi = mid;
    }
    c.k[i] = (uint32_t)lo;
  }
  for (int i = 0; i < 8; ++i) {
    const unsigned __int128 target = ((unsigned __int128)primes[i]) << 64;
    uint64_t lo = 0, hi = (uint64_t)1 << 36;
    while (hi - lo > 1) {
      const uint64_t mid = (lo + hi) / 2;
      if ((unsigned __int128)mid * mid <= target) lo = mid; else hi = mid;
    }
    c.h0[i] = (uint32_t)lo;
  }
}

struct HostConstInit {
  HostConstInit() { sha_const_compute(qgb_sha_host); }
};
static HostConstInit host_const_init;

void init_constants()
{
  cudaMemcpyToSymbol(qgb_sha_dev, &qgb_sha_host, sizeof(ShaConst));
  cudaMemcpyToSymbol(qgb_logtab_dev, qgb_logtab_host, sizeof(qgb_logtab_host));
}

// ------------------------------------------------------------------------
// gf_evolve: W = unitarize(exp(eps P) U) (hmc.cpp:311-328, matrix-hmc.h:179-188); W may be U

template <typename R>
__global__ void __launch_bounds__(256) k_evolve(Geo g, Cx<R>* U, Cx<R>* W, const Cx<R>* P, double eps, int unit,
                                                int taylor)
{
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= g.V) return;
  const int mu = blockIdx.y;
  const WField<R> Uf{U, g.V}, Wf{W, g.V};
  const CField<R> Pf{P, g.V};
  const M3<R> a = scale(R(eps), Pf.ld(s, mu));
  const M3<R> e = taylor ? exp_taylor(a, 20) : exp_ch(a);
  M3<R> un = mul(e, Uf.ld(s, mu));
  if (unit) unitarize(un);
  Wf.st(s, mu, un);
}

template <typename R>
cudaError_t launch_evolve(const Geo& g, void* U, const void* P, double eps, int unitarize, int taylor,
                          cudaStream_t st, void* W)
{
  const int bs = 256;
  dim3 grid((unsigned)((g.V + bs - 1) / bs), 4);
  k_evolve<R><<<grid, bs, 0, st>>>(g, (Cx<R>*)U, (Cx<R>*)(W ? W : U), (const Cx<R>*)P, eps, unitarize, taylor);
  return cudaGetLastError();
}

template <typename R, typename C>
__global__ void k_unitarize(long V, int m, Cx<R>* U)
{
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  const WField<R> Uf{U, V};
  for (int mu = 0; mu < m; ++mu) {
    M3<R> u = Uf.ld(s, mu);
    unitarize_as<C, R>(u);
    Uf.st(s, mu, u);
  }
}

template <typename R, typename C>
cudaError_t launch_unitarize(const Geo& g, int m, void* U, cudaStream_t st)
{
  const int bs = 256;
  k_unitarize<R, C><<<(unsigned)((g.V + bs - 1) / bs), bs, 0, st>>>(g.V, m, (Cx<R>*)U);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------
// deterministic reductions

static const int RED_BS = 256;

int reduce_blocks(const Geo& g) { return (int)((g.V + RED_BS - 1) / RED_BS); }

// Reduce NV values across the block in a fixed order; thread 0 writes
// partials[k * gridDim.x + blockIdx.x].
template <int NV>
__device__ __forceinline__ void block_reduce_store(double (&v)[NV], double* partials)
{
  __shared__ double sm[NV][RED_BS / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double x = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) sm[k][w] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double t = 0.0;
      for (int i = 0; i < RED_BS / 32; ++i) t += sm[k][i];
      partials[(long)k * gridDim.x + blockIdx.x] = t;
    }
  }
}

template <typename R>
__global__ void __launch_bounds__(RED_BS) k_gm_hamilton(Geo g, const Cx<R>* P, double* partials)
{
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  double v[1] = {0.0};
  if (s < g.V && in_reduce(g, s)) {
    const CField<R> Pf{P, g.V};
#pragma unroll
    for (int mu = 0; mu < 4; ++mu) v[0] += neg_half_tr_square(Pf.ld(s, mu));
  }
  block_reduce_store<1>(v, partials);
}

template <typename R>
cudaError_t launch_gm_hamilton(const Geo& g, const void* P, double* partials, cudaStream_t st)
{
  k_gm_hamilton<R><<<reduce_blocks(g), RED_BS, 0, st>>>(g, (const Cx<R>*)P, partials);
  return cudaGetLastError();
}

// Threads cover the padded sites too (reduce_blocks(g) blocks of RED_BS span
// padded_sites(V), RED_BS being a multiple of 32), so Q's padding is written
// (with the zeros of P's).  The sum uses the FP64 one of the two matrices, so
// it equals k_gm_hamilton<double> on the FP64 field bit for bit.
template <typename RI, typename RO>
__global__ void __launch_bounds__(RED_BS) k_gm_hamilton_convert(Geo g, const Cx<RI>* P, Cx<RO>* Q, double* partials)
{
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  double v[1] = {0.0};
  if (s < padded_sites(g.V)) {
    const CField<RI> Pf{P, g.V};
    const WField<RO> Qf{Q, g.V};
    const bool sum = s < g.V && in_reduce(g, s);
#pragma unroll 1
    for (int mu = 0; mu < 4; ++mu) {
      const M3<RI> p = Pf.ld(s, mu);
      M3<RO> q;
      M3<double> d;
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        q.e[k] = cx<RO>((RO)p.e[k].re, (RO)p.e[k].im);
        d.e[k] = sizeof(RI) == 8 ? cx<double>((double)p.e[k].re, (double)p.e[k].im)
                                 : cx<double>((double)q.e[k].re, (double)q.e[k].im);
      }
      Qf.st(s, mu, q);
      if (sum) v[0] += neg_half_tr_square(d);
    }
  }
  block_reduce_store<1>(v, partials);
}

template <typename RI, typename RO>
cudaError_t launch_gm_hamilton_convert(const Geo& g, const void* P, void* Q, double* partials, cudaStream_t st)
{
  k_gm_hamilton_convert<RI, RO><<<reduce_blocks(g), RED_BS, 0, st>>>(g, (const Cx<RI>*)P, (Cx<RO>*)Q, partials);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(256) k_unitarize_to_f64(long V, const Cx<float>* P, Cx<double>* Q)
{
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= padded_sites(V)) return;
  const CField<float> Pf{P, V};
  const WField<double> Qf{Q, V};
#pragma unroll 1
  for (int mu = 0; mu < 4; ++mu) {
    const M3<float> p = Pf.ld(s, mu);
    M3<double> u;
#pragma unroll
    for (int k = 0; k < 9; ++k) u.e[k] = cx<double>((double)p.e[k].re, (double)p.e[k].im);
    if (s < V) unitarize_as<double, double>(u);
    Qf.st(s, mu, u);
  }
}

cudaError_t launch_unitarize_to_f64(const Geo& g, const void* P, void* Q, cudaStream_t st)
{
  const int bs = 256;
  k_unitarize_to_f64<<<(unsigned)((padded_sites(g.V) + bs - 1) / bs), bs, 0, st>>>(g.V, (const Cx<float>*)P,
                                                                                  (Cx<double>*)Q);
  return cudaGetLastError();
}

// Sums over the 6 planes mu < nu at x of (Re tr plaq - 3) and, with RECT, of
// (Re tr rect - 3) for both rectangle orientations (hmc.cpp:9-25,203-252):
// plaq = A B^+ with A = U_mu(x) U_nu(x+mu), B = U_nu(x) U_mu(x+nu);
// rect (mu, mu, nu, -mu, -mu, -nu) = A B^+ with A = U_mu(x) U_mu(x+mu) U_nu(x+2mu),
// B = U_nu(x) U_mu(x+nu) U_mu(x+mu+nu).
template <typename R, bool RECT>
__global__ void __launch_bounds__(RED_BS) k_action(Geo g, const Cx<R>* Up, double* partials)
{
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  double v[2] = {0.0, 0.0};
  if (s < g.V && in_reduce(g, s)) {
    const CField<R> U{Up, g.V};
    const Coord x = coord_of(g, s);
#pragma unroll 1
    for (int p = 0; p < 6; ++p) {
      const int mu = p < 3 ? 0 : (p < 5 ? 1 : 2);
      const int nu = p < 3 ? p + 1 : (p < 5 ? p - 1 : 3);
      {
        const M3<R> A = mul(U.ld(s, mu), U.ld(site_rt(g, x, mu, 1, nu, 0), nu));
        const M3<R> B = mul(U.ld(s, nu), U.ld(site_rt(g, x, mu, 0, nu, 1), mu));
        v[0] += (double)re_tr_mul_adj(A, B) - 3.0;
      }
      if (RECT) {
#pragma unroll 1
        for (int o = 0; o < 2; ++o) {
          const int a = o == 0 ? mu : nu, b = o == 0 ? nu : mu;  // long side along a
          M3<R> A = mul(U.ld(s, a), U.ld(site_rt(g, x, a, 1, b, 0), a));
          A = mul(A, U.ld(site_rt(g, x, a, 2, b, 0), b));
          M3<R> B = mul(U.ld(s, b), U.ld(site_rt(g, x, a, 0, b, 1), a));
          B = mul(B, U.ld(site_rt(g, x, a, 1, b, 1), a));
          v[1] += (double)re_tr_mul_adj(A, B) - 3.0;
        }
      }
    }
  }
  block_reduce_store<2>(v, partials);
}

// The same sums with each loop walked as one running product (two 3x3
// matrices live instead of four; at most 128 registers, two blocks per SM),
// neighbours as the site plus per-direction offsets (LinkLd):
// plaq = Re tr(U_mu(x) U_nu(x+mu) U_mu(x+nu)^+ U_nu(x)^+),
// rect = Re tr(U_a(x) U_a(x+a) U_b(x+2a) U_a(x+a+b)^+ U_a(x+b)^+ U_b(x)^+)
// over the 12 ordered pairs (a, b), i.e. both orientations of every plane.
// In FP32 the double link U_a(x) U_a(x+a) is formed once for the three
// rectangles whose long side runs along a (52 instead of 60 products per
// site); in FP64 the extra live matrix costs more than the products it saves
// (24^3 x 64 on B200: FP64 0.56 ms with the double link recomputed against
// 0.59 ms shared, FP32 0.31 ms shared against 0.34 ms; 0.79 / 0.53 ms for
// k_action).
// With copy != nullptr each thread also writes its site's links, converted to
// FP32, into copy (padded sites included, with zeros).
template <typename R, bool RECT>
__global__ void __launch_bounds__(RED_BS, 2) k_action_loops(Geo g, const Cx<R>* Up, double* partials,
                                                            Cx<float>* copy)
{
  constexpr bool SHARE = sizeof(R) == 4;
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (copy != nullptr && s < padded_sites(g.V)) {
    const CField<R> Uf{Up, g.V};
    const WField<float> Cf{copy, g.V};
#pragma unroll 1
    for (int mu = 0; mu < 4; ++mu) {
      const M3<R> u = Uf.ld(s, mu);
      M3<float> c;
#pragma unroll
      for (int k = 0; k < 9; ++k) c.e[k] = cx<float>((float)u.e[k].re, (float)u.e[k].im);
      Cf.st(s, mu, c);
    }
  }
  double v[2] = {0.0, 0.0};
  if (s < g.V && in_reduce(g, s)) {
    const LinkLd<R> L{Up, (int)site_blocks(g.V)};
    const Coord x = coord_of(g, s);
    const int si = (int)s;
    const int st[4] = {1, g.d[0], g.d[0] * g.d[1], g.d[0] * g.d[1] * g.d[2]};
    int d1[4], d2[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      d1[k] = nb_delta(x.c[k], 1, g.d[k], st[k]);
      d2[k] = nb_delta(x.c[k], 2, g.d[k], st[k]);
    }
#pragma unroll 1
    for (int p = 0; p < 6; ++p) {
      const int mu = p < 3 ? 0 : (p < 5 ? 1 : 2);
      const int nu = p < 3 ? p + 1 : (p < 5 ? p - 1 : 3);
      M3<R> M = mul(L(mu, si), L(nu, si + sel4(d1, mu)));
      M = mul_adj(M, L(mu, si + sel4(d1, nu)));
      v[0] += (double)re_tr_mul_adj(M, L(nu, si)) - 3.0;
    }
    if (RECT) {
#pragma unroll 1
      for (int a = 0; a < 4; ++a) {
        const int a1 = sel4(d1, a), a2 = sel4(d2, a);
        M3<R> D;
        if constexpr (SHARE) D = mul(L(a, si), L(a, si + a1));
#pragma unroll 1
        for (int i = 1; i < 4; ++i) {
          const int b = (a + i) & 3;
          const int b1 = sel4(d1, b);
          M3<R> M;
          if constexpr (SHARE) {
            M = mul(D, L(b, si + a2));
          } else {
            M = mul(L(a, si), L(a, si + a1));
            M = mul(M, L(b, si + a2));
          }
          M = mul_adj(M, L(a, si + a1 + b1));
          M = mul_adj(M, L(a, si + b1));
          v[1] += (double)re_tr_mul_adj(M, L(b, si)) - 3.0;
        }
      }
    }
  }
  block_reduce_store<2>(v, partials);
}

// The same sums with the two corners of each plane (a, b) shared by its
// plaquette and its two rectangles (FP64; one thread per site, up to 255
// registers):
//   Pa = U_a(x) U_b(x+a), Pb = U_b(x) U_a(x+b):   plaq = Re tr(Pa Pb^+)
//   rect, long side a = Re tr([U_a(x) U_a(x+a) U_b(x+2a)] [Pb U_a(x+a+b)]^+)
//   rect, long side b = Re tr([U_b(x) U_b(x+b) U_a(x+2b)] [Pa U_b(x+a+b)]^+)
// 8 products, 3 traces and 10 link loads per plane instead of 10, 3 and 16:
// the loops of hmc.cpp:203-252, grouped differently.  The plaquette-only sum
// (gf_avg_plaq, Wilson actions) fits 128 registers and runs two blocks per SM.
template <typename R, bool RECT>
__global__ void __launch_bounds__(RED_BS, RECT ? 1 : 2) k_action_corners(Geo g, const Cx<R>* Up, double* partials,
                                                              Cx<float>* copy)
{
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (copy != nullptr && s < padded_sites(g.V)) {
    const CField<R> Uf{Up, g.V};
    const WField<float> Cf{copy, g.V};
#pragma unroll 1
    for (int mu = 0; mu < 4; ++mu) {
      const M3<R> u = Uf.ld(s, mu);
      M3<float> c;
#pragma unroll
      for (int k = 0; k < 9; ++k) c.e[k] = cx<float>((float)u.e[k].re, (float)u.e[k].im);
      Cf.st(s, mu, c);
    }
  }
  double v[2] = {0.0, 0.0};
  if (s < g.V && in_reduce(g, s)) {
    const LinkLd<R> L{Up, (int)site_blocks(g.V)};
    const Coord x = coord_of(g, s);
    const int si = (int)s;
    const int st[4] = {1, g.d[0], g.d[0] * g.d[1], g.d[0] * g.d[1] * g.d[2]};
    int d1[4], d2[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      d1[k] = nb_delta(x.c[k], 1, g.d[k], st[k]);
      d2[k] = nb_delta(x.c[k], 2, g.d[k], st[k]);
    }
#pragma unroll 1
    for (int p = 0; p < 6; ++p) {
      const int a = p < 3 ? 0 : (p < 5 ? 1 : 2);
      const int b = p < 3 ? p + 1 : (p < 5 ? p - 1 : 3);
      const int a1 = sel4(d1, a), b1 = sel4(d1, b);
      const M3<R> ua = L(a, si), ub = L(b, si);
      const M3<R> Pa = mul(ua, L(b, si + a1));
      const M3<R> Pb = mul(ub, L(a, si + b1));
      v[0] += (double)re_tr_mul_adj(Pa, Pb) - 3.0;
      if (RECT) {
        {
          const M3<R> A = mul(mul(ua, L(a, si + a1)), L(b, si + sel4(d2, a)));
          v[1] += (double)re_tr_mul_adj(A, mul(Pb, L(a, si + a1 + b1))) - 3.0;
        }
        {
          const M3<R> A = mul(mul(ub, L(b, si + b1)), L(a, si + sel4(d2, b)));
          v[1] += (double)re_tr_mul_adj(A, mul(Pa, L(b, si + a1 + b1))) - 3.0;
        }
      }
    }
  }
  block_reduce_store<2>(v, partials);
}

template <typename R>
cudaError_t launch_action(const Geo& g, const void* U, int rect, double* partials, cudaStream_t st, void* copy_f32)
{
  const Cx<R>* u = (const Cx<R>*)U;
  Cx<float>* c = (Cx<float>*)copy_f32;
  if (sizeof(R) == 8 && padded_sites(g.V) * 36 < 2147483647L) {
    if (rect) k_action_corners<R, true><<<reduce_blocks(g), RED_BS, 0, st>>>(g, u, partials, c);
    else k_action_corners<R, false><<<reduce_blocks(g), RED_BS, 0, st>>>(g, u, partials, c);
  } else if (padded_sites(g.V) * 36 < 2147483647L) {
    if (rect) k_action_loops<R, true><<<reduce_blocks(g), RED_BS, 0, st>>>(g, u, partials, c);
    else k_action_loops<R, false><<<reduce_blocks(g), RED_BS, 0, st>>>(g, u, partials, c);
  } else {  // 32-bit link offsets would overflow
    if (rect) k_action<R, true><<<reduce_blocks(g), RED_BS, 0, st>>>(g, u, partials);
    else k_action<R, false><<<reduce_blocks(g), RED_BS, 0, st>>>(g, u, partials);
    if (c != nullptr) return launch_convert<R, float>(padded_sites(g.V) * 4 * 18, U, c, st);
  }
  return cudaGetLastError();
}

template <typename R>
__global__ void __launch_bounds__(RED_BS) k_qnorm(long n, const R* x, double* partials)
{
  double v[1] = {0.0};
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const double t = (double)x[i];
    v[0] += t * t;
  }
  block_reduce_store<1>(v, partials);
}

template <typename R>
cudaError_t launch_qnorm(long n_reals, const void* x, double* partials, int blocks, cudaStream_t st)
{
  k_qnorm<R><<<blocks, RED_BS, 0, st>>>(n_reals, (const R*)x, partials);
  return cudaGetLastError();
}

// One block per value: its partial sums in a fixed order (loads in groups of 8, so that a block's latency is
// paid once per group).
__global__ void __launch_bounds__(1024) k_finalize(const double* partials, int blocks, double* results, int slot)
{
  __shared__ double sm[32];
  const int k = blockIdx.x;
  double t = 0.0;
#pragma unroll 8
  for (int i = threadIdx.x; i < blocks; i += 1024) t += partials[(long)k * blocks + i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    double r = 0.0;
    for (int i = 0; i < 32; ++i) r += sm[i];
    results[slot + k] = r;
  }
}

cudaError_t launch_finalize(const double* partials, int n_values, int blocks, double* results, int slot,
                            cudaStream_t st)
{
  k_finalize<<<n_values, 1024, 0, st>>>(partials, blocks, results, slot);
  return cudaGetLastError();
}

__global__ void k_combine(double* r, int out, int a, int b, int c) { r[out] = r[a] + r[b] - r[c]; }

cudaError_t launch_combine(double* results, int out, int a, int b, int c, cudaStream_t st)
{
  k_combine<<<1, 1, 0, st>>>(results, out, a, b, c);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------
// per-site random fields (qcd-utils.cpp:47-92)

struct RngArg {
  uint32_t v[24];
};

// One link's momentum from its 8 Gaussians (make_g_rand_anti_hermitian_matrix,
// matrix-hmc.h:125-142), stored in the field's precision.
template <typename R>
__device__ __forceinline__ void momentum_store(const WField<R>& Pf, long s, int mu, const double* b, double inv_sqrt3)
{
  const M3<double> m = x_make_anti_hermitian(b, inv_sqrt3);
  M3<R> mr;
#pragma unroll
  for (int k = 0; k < 9; ++k) mr.e[k] = cx<R>((R)m.e[k].re, (R)m.e[k].im);
  Pf.st(s, mu, mr);
}

// set_g_rand_anti_hermitian_matrix_field: per site RngState(rs, gindex),
// 4 x make_g_rand_anti_hermitian_matrix (matrix-hmc.h:125-142).
template <typename R>
__global__ void __launch_bounds__(128) k_rand_momentum(Geo g, RngArg ra, double s_sigma, double inv_sqrt3,
                                                       Cx<R>* P, int* ambiguous)
{
  // every lane of the warp stays to the end (warp-wide refills); lanes past
  // the last site draw nothing, and so do the halo sites of a domain, whose
  // momenta no force or sum reads (they are set to zero)
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool inside = s < g.V;
  const bool active = inside && (!has_box(g) || in_box(g, s));
  Rng base, rs;
  rng_import(base, ra.v);
  if (active) rng_split_long(rs, base, (int64_t)rng_index(g, s));
  int amb = 0;
  const WField<R> Pf{P, g.V};
  if (inside && !active) {
#pragma unroll 1
    for (int mu = 0; mu < 4; ++mu) Pf.st(s, mu, m3_zero<R>());
  }
  // the 8 Gaussians of a link wait in shared memory (the draw index is a
  // run-time value; a per-thread array would live in local memory)
  __shared__ double sb[8 * 128];
  rng_gaussians_converged<32>(rs, s_sigma, active, &amb, [&](int i, double v) {
    sb[(i & 7) * 128 + threadIdx.x] = v;
    if ((i & 7) == 7) {
      double b[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) b[k] = sb[k * 128 + threadIdx.x];
      momentum_store(Pf, s, i >> 3, b, inv_sqrt3);
    }
  });
  if (amb) atomicAdd(ambiguous, 1);
}

template <typename R>
cudaError_t launch_rand_momentum(const Geo& g, void* P, const uint32_t* rs24, double sigma, int* ambiguous,
                                 cudaStream_t st)
{
  RngArg ra;
  memcpy(ra.v, rs24, sizeof(ra.v));
  const double s_sigma = sigma / sqrt(2.0);
  const double inv_sqrt3 = 1.0 / sqrt(3.0);
  const int bs = 128;
  k_rand_momentum<R><<<(unsigned)((g.V + bs - 1) / bs), bs, 0, st>>>(g, ra, s_sigma, inv_sqrt3, (Cx<R>*)P,
                                                                     ambiguous);
  return cudaGetLastError();
}

// The four links of one site of a hot start (below): per link n_step factors,
// each unitarize(exp_taylor20(X)) with X made from 8 Gaussians, multiplied in
// order.  The Gaussians come from rng_gaussians_converged, 8 per factor, so a
// warp's SHA-256 refills run together; the values are those of 8 successive
// g_rand_gen calls.  Called by all 32 lanes of a warp.
template <typename R>
__device__ __forceinline__ void hot_start_links(Rng& rs, bool active, double s_sigma, double inv_sqrt3, int n_step,
                                                const WField<R>& Uf, long s, int* amb)
{
  __shared__ double sb[8 * 128];  // the 8 Gaussians of a factor (run-time draw index)
  const int nk = n_step > 1 ? n_step : 1;  // the reference always draws at least one factor
  for (int mu = 0; mu < 4; ++mu) {
    M3<double> v;
    for (int k = 0; k < nk; ++k) {
      rng_gaussians_converged<8>(rs, s_sigma, active, amb,
                                 [&](int i, double x) { sb[i * 128 + threadIdx.x] = x; });
      double b[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) b[i] = active ? sb[i * 128 + threadIdx.x] : 0.0;
      M3<double> e = x_exp_taylor20(x_make_anti_hermitian(b, inv_sqrt3));
      x_unitarize(e);
      v = (k == 0) ? e : xm_mul(v, e);
    }
    if (active) {
      M3<R> vr;
#pragma unroll
      for (int k = 0; k < 9; ++k) vr.e[k] = cx<R>((R)v.e[k].re, (R)v.e[k].im);
      Uf.st(s, mu, vr);
    }
  }
}

// set_g_rand_color_matrix_field: per link n_step products of
// unitarize(exp_taylor20(X)) with X from make_g_rand_anti_hermitian_matrix.
template <typename R>
__global__ void __launch_bounds__(128) k_hot_start(Geo g, RngArg ra, double s_sigma, double inv_sqrt3, int n_step,
                                                   Cx<R>* U, int* ambiguous)
{
  // every lane of the warp stays to the end (warp-wide refills); lanes past
  // the last site draw nothing and store nothing
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = s < g.V;
  Rng base, rs;
  rng_import(base, ra.v);
  if (active) rng_split_long(rs, base, (int64_t)rng_index(g, s));
  int amb = 0;
  hot_start_links<R>(rs, active, s_sigma, inv_sqrt3, n_step, WField<R>{U, g.V}, s, &amb);
  if (amb) atomicAdd(ambiguous, 1);
}

template <typename R>
cudaError_t launch_hot_start(const Geo& g, void* U, const uint32_t* rs24, double sigma, int n_step, int* ambiguous,
                             cudaStream_t st)
{
  RngArg ra;
  memcpy(ra.v, rs24, sizeof(ra.v));
  const double s_sigma = sigma / sqrt(2.0);
  const double inv_sqrt3 = 1.0 / sqrt(3.0);
  const int bs = 128;
  k_hot_start<R><<<(unsigned)((g.V + bs - 1) / bs), bs, 0, st>>>(g, ra, s_sigma, inv_sqrt3, n_step, (Cx<R>*)U,
                                                                 ambiguous);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------
// batches of independent chains (all chains in one launch)

// Per-site random momenta of every chain: chain c uses RngState rs24[24 c ..]
// split by the site's index within its chain.
template <typename R>
__global__ void __launch_bounds__(128) k_rand_momentum_batch(long Vtot, int nchain, const long* __restrict__ offs,
                                                             const uint32_t* __restrict__ rs24, double s_sigma,
                                                             double inv_sqrt3, Cx<R>* P, int* ambiguous)
{
  const long sg = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = sg < Vtot;
  Rng rs;
  if (active) {
    const int c = chain_of(offs, nchain, sg);
    Rng base;
    rng_import(base, rs24 + 24 * c);
    rng_split_long(rs, base, (int64_t)(sg - offs[c]));
  }
  int amb = 0;
  const WField<R> Pf{P, Vtot};
  double b[8];
  rng_gaussians_converged<32>(rs, s_sigma, active, &amb, [&](int i, double v) {
    b[i & 7] = v;
    if ((i & 7) == 7) momentum_store(Pf, sg, i >> 3, b, inv_sqrt3);
  });
  if (amb) atomicAdd(ambiguous, 1);
}

template <typename R>
__global__ void __launch_bounds__(128) k_hot_start_batch(long Vtot, int nchain, const long* __restrict__ offs,
                                                         const uint32_t* __restrict__ rs24, double s_sigma,
                                                         double inv_sqrt3, int n_step, Cx<R>* U, int* ambiguous)
{
  const long sg = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = sg < Vtot;
  Rng rs;
  if (active) {
    const int c = chain_of(offs, nchain, sg);
    Rng base;
    rng_import(base, rs24 + 24 * c);
    rng_split_long(rs, base, (int64_t)(sg - offs[c]));
  }
  int amb = 0;
  hot_start_links<R>(rs, active, s_sigma, inv_sqrt3, n_step, WField<R>{U, Vtot}, sg, &amb);
  if (amb) atomicAdd(ambiguous, 1);
}

// Site values for the per-chain Hamiltonians.

// vals[sg] = sum_mu -tr(P^2)/2, and with COPY the momenta converted to RO into Q in the same pass (padded sites
// included, with the zeros of P's).  Memory-bound: 1.69 M sites (256 chains of 4^4 to 12^4) in a trajectory, 0.220 ms
// with the copy (1.47 GB) and 0.062 ms from FP32 (0.50 GB, of which the L2 still holds what the last force wrote).
template <typename RI, typename RO, bool COPY>
__global__ void __launch_bounds__(256) k_batch_kinetic(long Vtot, const Cx<RI>* P, Cx<RO>* Q, double* vals)
{
  const long sg = (long)blockIdx.x * 256 + threadIdx.x;
  if (sg >= padded_sites(Vtot)) return;
  const CField<RI> Pf{P, Vtot};
  double v = 0.0;
#pragma unroll 1
  for (int mu = 0; mu < 4; ++mu) {
    const M3<RI> p = Pf.ld(sg, mu);
    M3<double> d;
#pragma unroll
    for (int k = 0; k < 9; ++k) d.e[k] = cx<double>((double)p.e[k].re, (double)p.e[k].im);
    if (COPY) {
      M3<RO> q;
#pragma unroll
      for (int k = 0; k < 9; ++k) q.e[k] = cx<RO>((RO)p.e[k].re, (RO)p.e[k].im);
      WField<RO>{Q, Vtot}.st(sg, mu, q);
    }
    v += neg_half_tr_square(d);
  }
  if (sg < Vtot) vals[sg] = v;
}

// Plaquette sums into vals[sg] and, with RECT, rectangle sums into vals[Vtot + sg], as k_action_corners within
// each site's chain (8 products per plane instead of 10 from 64-bit index walks); with copy != nullptr also the
// links in FP32 (padded sites included).  Blocks of 64 sites, so that a small batch spreads over the SMs: one chain of
// 4^4 8.9 -> 7.8 us, three of 4^4 to 8^4 with rectangles 23.7 -> 17.7 (blocks of 256 before), 256 chains as before.
constexpr int ACT_BS = 64;

template <bool RECT>
__global__ void __launch_bounds__(ACT_BS, RECT ? 4 : 8)
    k_batch_action(long Vtot, int nchain, const long* __restrict__ offs, const ChainInfo* __restrict__ chains,
                   const Cx<double>* U, Cx<float>* copy, double* vals)
{
  const long sg = (long)blockIdx.x * ACT_BS + threadIdx.x;
  if (copy != nullptr && sg < padded_sites(Vtot)) {
    const CField<double> Uf{U, Vtot};
#pragma unroll 1
    for (int mu = 0; mu < 4; ++mu) {
      const M3<double> u = Uf.ld(sg, mu);
      M3<float> c;
#pragma unroll
      for (int k = 0; k < 9; ++k) c.e[k] = cx<float>((float)u.e[k].re, (float)u.e[k].im);
      WField<float>{copy, Vtot}.st(sg, mu, c);
    }
  }
  if (sg >= Vtot) return;
  const Geo g = chain_geo(chains[chain_of(offs, nchain, sg)]);
  const Coord x = coord_of(g, sg - g.off);
  const LinkLd<double> L{U, (int)site_blocks(Vtot)};
  const int si = (int)sg;
  const int st[4] = {1, g.d[0], g.d[0] * g.d[1], g.d[0] * g.d[1] * g.d[2]};
  int d1[4], d2[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    d1[k] = nb_delta(x.c[k], 1, g.d[k], st[k]);
    d2[k] = nb_delta(x.c[k], 2, g.d[k], st[k]);
  }
  double sp = 0.0, sr = 0.0;
#pragma unroll 1
  for (int p = 0; p < 6; ++p) {
    const int a = p < 3 ? 0 : (p < 5 ? 1 : 2);
    const int b = p < 3 ? p + 1 : (p < 5 ? p - 1 : 3);
    const int a1 = sel4(d1, a), b1 = sel4(d1, b);
    const M3<double> ua = L(a, si), ub = L(b, si);
    const M3<double> Pa = mul(ua, L(b, si + a1));
    const M3<double> Pb = mul(ub, L(a, si + b1));
    sp += re_tr_mul_adj(Pa, Pb) - 3.0;
    if (RECT) {
      {
        const M3<double> A = mul(mul(ua, L(a, si + a1)), L(b, si + sel4(d2, a)));
        sr += re_tr_mul_adj(A, mul(Pb, L(a, si + a1 + b1))) - 3.0;
      }
      {
        const M3<double> A = mul(mul(ub, L(b, si + b1)), L(a, si + sel4(d2, b)));
        sr += re_tr_mul_adj(A, mul(Pa, L(b, si + a1 + b1))) - 3.0;
      }
    }
  }
  vals[sg] = sp;
  if (RECT) vals[Vtot + sg] = sr;
}

// The action sums where 32-bit link offsets would overflow.
template <typename R>
__global__ void __launch_bounds__(128) k_batch_action_large(long Vtot, int nchain, const long* __restrict__ offs,
                                                            const ChainInfo* __restrict__ chains, int rect,
                                                            const Cx<R>* F, double* vals)
{
  const long sg = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (sg >= Vtot) return;
  const CField<R> Ff{F, Vtot};
  const int c = chain_of(offs, nchain, sg);
  const Geo g = chain_geo(chains[c]);
  const Coord x = coord_of(g, sg - g.off);
  double sp = 0.0, sr = 0.0;
#pragma unroll 1
  for (int p = 0; p < 6; ++p) {
    const int mu = p < 3 ? 0 : (p < 5 ? 1 : 2);
    const int nu = p < 3 ? p + 1 : (p < 5 ? p - 1 : 3);
    const M3<R> A = mul(Ff.ld(sg, mu), Ff.ld(site_rt(g, x, mu, 1, nu, 0), nu));
    const M3<R> B = mul(Ff.ld(sg, nu), Ff.ld(site_rt(g, x, mu, 0, nu, 1), mu));
    sp += (double)re_tr_mul_adj(A, B) - 3.0;
    if (rect) {
#pragma unroll 1
      for (int o = 0; o < 2; ++o) {
        const int a = o == 0 ? mu : nu, b = o == 0 ? nu : mu;
        M3<R> A2 = mul(Ff.ld(sg, a), Ff.ld(site_rt(g, x, a, 1, b, 0), a));
        A2 = mul(A2, Ff.ld(site_rt(g, x, a, 2, b, 0), b));
        M3<R> B2 = mul(Ff.ld(sg, b), Ff.ld(site_rt(g, x, a, 0, b, 1), a));
        B2 = mul(B2, Ff.ld(site_rt(g, x, a, 1, b, 1), a));
        sr += (double)re_tr_mul_adj(A2, B2) - 3.0;
      }
    }
  }
  vals[sg] = sp;
  if (rect) vals[Vtot + sg] = sr;
}

// out[c] = sum of vals over chain c's sites, one block per chain, fixed order.
__global__ void __launch_bounds__(256) k_segment_sum(int nchain, const long* __restrict__ offs,
                                                     const double* __restrict__ vals, double* out)
{
  const int c = blockIdx.x;
  const long a = offs[c], b = offs[c + 1];
  double t = 0.0;
  for (long i = a + threadIdx.x; i < b; i += blockDim.x) t += vals[i];
  __shared__ double sm[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    double r = 0.0;
    for (int i = 0; i < 8; ++i) r += sm[i];
    out[c] = r;
  }
}

// dst = src on the sites of chains whose flag is set (4 links per site).
template <typename R>
__global__ void k_accept_batch(long Vtot, int nchain, const long* __restrict__ offs, const int* __restrict__ flags,
                               Cx<R>* dst, const Cx<R>* src)
{
  const long sg = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (sg >= Vtot) return;
  const int c = chain_of(offs, nchain, sg);
  if (!flags[c]) return;
  const CField<R> S{src, Vtot};
  const WField<R> D{dst, Vtot};
  for (int mu = 0; mu < 4; ++mu) D.st(sg, mu, S.ld(sg, mu));
}

template <typename R>
cudaError_t launch_rand_momentum_batch(long Vtot, int nchain, const long* offs, const uint32_t* rs24, double sigma,
                                       void* P, int* ambiguous, cudaStream_t st)
{
  k_rand_momentum_batch<R><<<(unsigned)((Vtot + 127) / 128), 128, 0, st>>>(Vtot, nchain, offs, rs24, sigma / sqrt(2.0),
                                                                          1.0 / sqrt(3.0), (Cx<R>*)P, ambiguous);
  return cudaGetLastError();
}

template <typename R>
cudaError_t launch_hot_start_batch(long Vtot, int nchain, const long* offs, const uint32_t* rs24, double sigma,
                                   int n_step, void* U, int* ambiguous, cudaStream_t st)
{
  k_hot_start_batch<R><<<(unsigned)((Vtot + 127) / 128), 128, 0, st>>>(Vtot, nchain, offs, rs24, sigma / sqrt(2.0),
                                                                      1.0 / sqrt(3.0), n_step, (Cx<R>*)U, ambiguous);
  return cudaGetLastError();
}

template <typename RI>
cudaError_t launch_batch_kinetic(long Vtot, const void* P, void* copy_f32, double* vals, cudaStream_t st)
{
  const unsigned grid = (unsigned)((padded_sites(Vtot) + 255) / 256);
  if (copy_f32) k_batch_kinetic<RI, float, true><<<grid, 256, 0, st>>>(Vtot, (const Cx<RI>*)P, (Cx<float>*)copy_f32, vals);
  else k_batch_kinetic<RI, float, false><<<grid, 256, 0, st>>>(Vtot, (const Cx<RI>*)P, nullptr, vals);
  return cudaGetLastError();
}

cudaError_t launch_batch_action(long Vtot, int nchain, const long* offs, const ChainInfo* chains, int rect,
                                const void* U, void* copy_f32, double* vals, cudaStream_t st)
{
  const Cx<double>* u = (const Cx<double>*)U;
  Cx<float>* c = (Cx<float>*)copy_f32;
  if (padded_sites(Vtot) * 36 < 2147483647L) {
    const unsigned grid = (unsigned)((padded_sites(Vtot) + ACT_BS - 1) / ACT_BS);
    if (rect) k_batch_action<true><<<grid, ACT_BS, 0, st>>>(Vtot, nchain, offs, chains, u, c, vals);
    else k_batch_action<false><<<grid, ACT_BS, 0, st>>>(Vtot, nchain, offs, chains, u, c, vals);
    return cudaGetLastError();
  }
  k_batch_action_large<double><<<(unsigned)((Vtot + 127) / 128), 128, 0, st>>>(Vtot, nchain, offs, chains, rect, u, vals);
  if (c != nullptr) return launch_convert<double, float>(padded_sites(Vtot) * 72, U, c, st);
  return cudaGetLastError();
}

cudaError_t launch_segment_sum(int nchain, const long* offs, const double* vals, double* out, cudaStream_t st)
{
  k_segment_sum<<<nchain, 256, 0, st>>>(nchain, offs, vals, out);
  return cudaGetLastError();
}

template <typename R>
cudaError_t launch_accept_batch(long Vtot, int nchain, const long* offs, const int* flags, void* dst, const void* src,
                                cudaStream_t st)
{
  k_accept_batch<R><<<(unsigned)((Vtot + 127) / 128), 128, 0, st>>>(Vtot, nchain, offs, flags, (Cx<R>*)dst,
                                                                    (const Cx<R>*)src);
  return cudaGetLastError();
}

template cudaError_t launch_rand_momentum_batch<double>(long, int, const long*, const uint32_t*, double, void*, int*,
                                                        cudaStream_t);
template cudaError_t launch_hot_start_batch<double>(long, int, const long*, const uint32_t*, double, int, void*, int*,
                                                    cudaStream_t);
template cudaError_t launch_batch_kinetic<double>(long, const void*, void*, double*, cudaStream_t);
template cudaError_t launch_batch_kinetic<float>(long, const void*, void*, double*, cudaStream_t);
template cudaError_t launch_accept_batch<double>(long, int, const long*, const int*, void*, const void*, cudaStream_t);

// ------------------------------------------------------------------------
// elementwise field operations

template <typename R>
__global__ void k_set_unit(long V, int m, Cx<R>* U)
{
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  const WField<R> Uf{U, V};
  for (int mu = 0; mu < m; ++mu) Uf.st(s, mu, m3_unit<R>());
}

template <typename R>
cudaError_t launch_set_unit(const Geo& g, int m, void* U, cudaStream_t st)
{
  k_set_unit<R><<<(unsigned)((g.V + 255) / 256), 256, 0, st>>>(g.V, m, (Cx<R>*)U);
  return cudaGetLastError();
}

template <typename R>
__global__ void k_axpby(long n, R* y, R a, const R* x, R b)
{
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const R xv = x ? x[i] : R(0);
    y[i] = (b == R(0)) ? a * xv : fma(a, xv, b * y[i]);
  }
}

template <typename R>
cudaError_t launch_axpby(long n, void* y, double a, const void* x, double b, cudaStream_t st)
{
  const long blocks = (n + 255) / 256;
  k_axpby<R><<<(unsigned)(blocks < 148 * 32 ? blocks : 148 * 32), 256, 0, st>>>(n, (R*)y, (R)a, (const R*)x, (R)b);
  return cudaGetLastError();
}

// reference image [site][m][k] (doubles) <-> device layout (gauge_common.cuh).
// Sites [off, off + n) of a field of Vf sites; the image holds those n sites.
// One thread per (component, site), sites fastest, so the device-side accesses
// of a warp are coalesced.
template <typename R>
__global__ void k_aos_to_store(long Vf, long off, long n, int m, int k_per, const double* __restrict__ aos,
                               R* __restrict__ store)
{
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * m) return;
  const int mm = (int)(i / n);
  const long s = i % n;
  const double* src = aos + (s * m + mm) * k_per;
  if (k_per == 1) {
    store[lay_index<1>(Vf, mm, 0, off + s)] = (R)src[0];
  } else {
    Cx<R>* dst = (Cx<R>*)store + lay_index<9>(Vf, mm, 0, off + s);
#pragma unroll
    for (int c = 0; c < 9; ++c) dst[32 * c] = cx<R>((R)src[2 * c], (R)src[2 * c + 1]);
  }
}

template <typename R>
__global__ void k_store_to_aos(long Vf, long off, long n, int m, int k_per, const R* __restrict__ store,
                               double* __restrict__ aos)
{
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * m) return;
  const int mm = (int)(i / n);
  const long s = i % n;
  double* dst = aos + (s * m + mm) * k_per;
  if (k_per == 1) {
    dst[0] = (double)store[lay_index<1>(Vf, mm, 0, off + s)];
  } else {
    const Cx<R>* src = (const Cx<R>*)store + lay_index<9>(Vf, mm, 0, off + s);
#pragma unroll
    for (int c = 0; c < 9; ++c) {
      const Cx<R> v = src[32 * c];
      dst[2 * c] = (double)v.re;
      dst[2 * c + 1] = (double)v.im;
    }
  }
}

// The same for gauge fields (four color matrices per site), a block of 32 sites through shared memory, so that
// both sides move whole lines: the image as one contiguous run of 18 KB, the device layout entry by entry.  Site
// s of the image starts at 37 s sixteen-byte units there (36 and one of padding): any 8 lanes of an access on
// consecutive sites meet 8 different bank groups.  One thread per component and site wrote 16 bytes every 576: a
// gauge field of 24^3 x 48 took 272 us from FP32 (573 MB) and 139 us to it, 91 and 97 us here.  Needs a range that starts at a block of 32
// sites and a 16-byte aligned image.
constexpr int AOS_PITCH = 37;

template <typename R>
__global__ void __launch_bounds__(128) k_store_to_aos4(long Vf, long off, long n, const Cx<R>* __restrict__ store,
                                                       double2* __restrict__ aos)
{
  __shared__ double2 sm[32 * AOS_PITCH];
  const long s0 = (long)blockIdx.x * 32;
  const int lane = threadIdx.x & 31, mu = threadIdx.x >> 5;
  if (s0 + lane < n) {
    const Cx<R>* src = store + lay_index<9>(Vf, mu, 0, off + s0 + lane);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const Cx<R> v = ldg_cx(src + 32 * k);
      sm[lane * AOS_PITCH + mu * 9 + k] = make_double2((double)v.re, (double)v.im);
    }
  }
  __syncthreads();
  const int count = (int)(n - s0 < 32 ? n - s0 : 32) * 36;
  double2* dst = aos + s0 * 36;
#pragma unroll
  for (int j = threadIdx.x; j < 32 * 36; j += 128)
    if (j < count) dst[j] = sm[(j / 36) * AOS_PITCH + j % 36];
}

template <typename R>
__global__ void __launch_bounds__(128) k_aos4_to_store(long Vf, long off, long n, const double2* __restrict__ aos,
                                                       Cx<R>* __restrict__ store)
{
  __shared__ double2 sm[32 * AOS_PITCH];
  const long s0 = (long)blockIdx.x * 32;
  const int count = (int)(n - s0 < 32 ? n - s0 : 32) * 36;
  const double2* src = aos + s0 * 36;
#pragma unroll
  for (int j = threadIdx.x; j < 32 * 36; j += 128)
    if (j < count) sm[(j / 36) * AOS_PITCH + j % 36] = __ldg(src + j);
  __syncthreads();
  const int lane = threadIdx.x & 31, mu = threadIdx.x >> 5;
  if (s0 + lane >= n) return;
  Cx<R>* dst = store + lay_index<9>(Vf, mu, 0, off + s0 + lane);
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const double2 v = sm[lane * AOS_PITCH + mu * 9 + k];
    dst[32 * k] = cx<R>((R)v.x, (R)v.y);
  }
}

static bool aos_by_blocks(long off, int m, int k_per, const void* aos)
{
  return m == 4 && k_per == 18 && off % 32 == 0 && (uintptr_t)aos % 16 == 0;
}

template <typename R>
cudaError_t launch_aos_to_store(long Vf, long off, long n, int m, int k_per, const double* aos, void* store,
                                cudaStream_t st)
{
  if (aos_by_blocks(off, m, k_per, aos)) {
    k_aos4_to_store<R><<<(unsigned)((n + 31) / 32), 128, 0, st>>>(Vf, off, n, (const double2*)aos, (Cx<R>*)store);
    return cudaGetLastError();
  }
  const long t = n * m;
  k_aos_to_store<R><<<(unsigned)((t + 255) / 256), 256, 0, st>>>(Vf, off, n, m, k_per, aos, (R*)store);
  return cudaGetLastError();
}

template <typename R>
cudaError_t launch_store_to_aos(long Vf, long off, long n, int m, int k_per, const void* store, double* aos,
                                cudaStream_t st)
{
  if (aos_by_blocks(off, m, k_per, aos)) {
    k_store_to_aos4<R><<<(unsigned)((n + 31) / 32), 128, 0, st>>>(Vf, off, n, (const Cx<R>*)store, (double2*)aos);
    return cudaGetLastError();
  }
  const long t = n * m;
  k_store_to_aos<R><<<(unsigned)((t + 255) / 256), 256, 0, st>>>(Vf, off, n, m, k_per, (const R*)store, aos);
  return cudaGetLastError();
}

template <typename RI, typename RO>
__global__ void k_convert(long n, const RI* in, RO* out)
{
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    out[i] = (RO)in[i];
}

// four elements per thread: 16- or 32-byte loads and stores (n % 4 == 0, 16-byte aligned buffers)
template <typename RI, typename RO>
__global__ void k_convert4(long n4, const RI* __restrict__ in, RO* __restrict__ out)
{
  using I2 = typename std::conditional<sizeof(RI) == 8, double2, float2>::type;
  using O2 = typename std::conditional<sizeof(RO) == 8, double2, float2>::type;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (long)gridDim.x * blockDim.x) {
    const I2 a = reinterpret_cast<const I2*>(in)[2 * i], b = reinterpret_cast<const I2*>(in)[2 * i + 1];
    O2 c, d;
    c.x = (decltype(c.x))a.x;
    c.y = (decltype(c.y))a.y;
    d.x = (decltype(d.x))b.x;
    d.y = (decltype(d.y))b.y;
    reinterpret_cast<O2*>(out)[2 * i] = c;
    reinterpret_cast<O2*>(out)[2 * i + 1] = d;
  }
}

template <typename RI, typename RO>
cudaError_t launch_convert(long n, const void* in, void* out, cudaStream_t st)
{
  const bool vec = n % 4 == 0 && ((uintptr_t)in % 16) == 0 && ((uintptr_t)out % 16) == 0;
  const long work = vec ? n / 4 : n;
  const long blocks = (work + 255) / 256;
  const unsigned grid = (unsigned)(blocks < 148 * 16 ? blocks : 148 * 16);
  if (vec) k_convert4<RI, RO><<<grid, 256, 0, st>>>(work, (const RI*)in, (RO*)out);
  else k_convert<RI, RO><<<grid, 256, 0, st>>>(n, (const RI*)in, (RO*)out);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------
// explicit instantiations

#define QGB_INST(R)                                                                                          \
  template cudaError_t launch_evolve<R>(const Geo&, void*, const void*, double, int, int, cudaStream_t, void*); \
  template cudaError_t launch_gm_hamilton<R>(const Geo&, const void*, double*, cudaStream_t);              \
  template cudaError_t launch_action<R>(const Geo&, const void*, int, double*, cudaStream_t, void*);       \
  template cudaError_t launch_qnorm<R>(long, const void*, double*, int, cudaStream_t);                    \
  template cudaError_t launch_rand_momentum<R>(const Geo&, void*, const uint32_t*, double, int*, cudaStream_t); \
  template cudaError_t launch_hot_start<R>(const Geo&, void*, const uint32_t*, double, int, int*, cudaStream_t); \
  template cudaError_t launch_set_unit<R>(const Geo&, int, void*, cudaStream_t);                          \
  template cudaError_t launch_axpby<R>(long, void*, double, const void*, double, cudaStream_t);           \
  template cudaError_t launch_aos_to_store<R>(long, long, long, int, int, const double*, void*, cudaStream_t); \
  template cudaError_t launch_store_to_aos<R>(long, long, long, int, int, const void*, double*, cudaStream_t);

QGB_INST(double)
QGB_INST(float)
template cudaError_t launch_unitarize<double, double>(const Geo&, int, void*, cudaStream_t);
template cudaError_t launch_unitarize<float, float>(const Geo&, int, void*, cudaStream_t);
template cudaError_t launch_unitarize<float, double>(const Geo&, int, void*, cudaStream_t);
template cudaError_t launch_gm_hamilton_convert<double, float>(const Geo&, const void*, void*, double*, cudaStream_t);
template cudaError_t launch_gm_hamilton_convert<float, double>(const Geo&, const void*, void*, double*, cudaStream_t);
template cudaError_t launch_convert<double, float>(long, const void*, void*, cudaStream_t);
template cudaError_t launch_convert<float, double>(long, const void*, void*, cudaStream_t);
template cudaError_t launch_convert<double, double>(long, const void*, void*, cudaStream_t);
template cudaError_t launch_convert<float, float>(long, const void*, void*, cudaStream_t);

}  // namespace qgb

namespace qgb
{
// ------------------------------------------------------------------------
// host RngState API

void rng_host_seed(uint32_t out[24], const char* seed)
{
  Rng r;
  memset(&r, 0, sizeof(r));
  memcpy(r.hash, qgb_sha_host.h0, 32);
  r.type = RNG_NO_TYPE;
  if (!seed) {  // RngState(): reset(rs) only
    rng_export(out, r);
    return;
  }
  Rng o;
  rng_split_bytes(o, r, (const uint8_t*)seed, (int)strlen(seed));
  rng_export(out, o);
}

bool rng_host_split(uint32_t out[24], const uint32_t rs[24], const char* sindex)
{
  Rng r, o;
  rng_import(r, rs);
  if (!rng_split_bytes(o, r, (const uint8_t*)sindex, (int)strlen(sindex))) return false;
  rng_export(out, o);
  return true;
}

uint64_t rng_host_rand_gen(uint32_t rs[24])
{
  Rng r;
  rng_import(r, rs);
  const uint64_t v = rng_rand_gen(r);
  rng_export(rs, r);
  return v;
}

double rng_host_u_rand_gen(uint32_t rs[24], double upper, double lower)
{
  Rng r;
  rng_import(r, rs);
  const double v = rng_u_rand_gen(r, upper, lower);
  rng_export(rs, r);
  return v;
}

double rng_host_g_rand_gen(uint32_t rs[24], double center, double sigma)
{
  Rng r;
  rng_import(r, rs);
  const double v = rng_g_rand_gen<false>(r, center, sigma, nullptr);
  rng_export(rs, r);
  return v;
}
// ------------------------------------------------------------------------
// box pack / unpack (halo exchange of a domain-decomposed field)

template <typename E>
__global__ void k_box_copy(Geo g, int K, int lo0, int lo1, int lo2, int lo3, int n0, int n1, int n2, long nbox,
                           E* field, E* buf, bool unpack)
{
  const long w = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= nbox) return;
  const int c = blockIdx.y;  // component * K + entry
  const int m = c / K, k = c - m * K;
  long r = w;
  const long x0 = r % n0 + lo0;
  r /= n0;
  const long x1 = r % n1 + lo1;
  r /= n1;
  const long x2 = r % n2 + lo2;
  const long x3 = r / n2 + lo3;
  const long s = x0 + (long)g.d[0] * (x1 + (long)g.d[1] * (x2 + (long)g.d[2] * x3));
  const long fi = ((m * site_blocks(g.V) + (s >> 5)) * K + k) * 32 + (s & 31);
  const long bi = (long)c * nbox + w;
  if (unpack) field[fi] = buf[bi];
  else buf[bi] = field[fi];
}

template <typename E>
cudaError_t launch_box_copy(const Geo& g, int m, int K, const int lo[4], const int n[4], void* field, void* buf,
                            bool unpack, cudaStream_t st)
{
  const long nbox = (long)n[0] * n[1] * n[2] * n[3];
  if (nbox == 0) return cudaSuccess;
  dim3 grid((unsigned)((nbox + 255) / 256), (unsigned)(m * K));
  k_box_copy<E><<<grid, 256, 0, st>>>(g, K, lo[0], lo[1], lo[2], lo[3], n[0], n[1], n[2], nbox, (E*)field, (E*)buf,
                                      unpack);
  return cudaGetLastError();
}

template cudaError_t launch_box_copy<double2>(const Geo&, int, int, const int*, const int*, void*, void*, bool,
                                              cudaStream_t);
template cudaError_t launch_box_copy<float2>(const Geo&, int, int, const int*, const int*, void*, void*, bool,
                                             cudaStream_t);
template cudaError_t launch_box_copy<double>(const Geo&, int, int, const int*, const int*, void*, void*, bool,
                                             cudaStream_t);
template cudaError_t launch_box_copy<float>(const Geo&, int, int, const int*, const int*, void*, void*, bool,
                                            cudaStream_t);

}  // namespace qgb
