// force_pair.cu -- the FP32 force and its fused consumers on pairs of sites.
//
// Two sites half a lattice apart along one direction p (t, or z where t is odd
// or short) share a thread: every operation on a link's reals acts on both
// (pair.cuh).  The fields of molecular dynamics and of the flow are kept in a
// packed layout meanwhile: a color-matrix field of the blocked layout whose
// entries hold both sites' reals, over the lattice with extent L_p / 2 along p
// plus two sites on either side.  Those borders hold the partners' links,
// swapped (x + L_p/2 wraps to the other half), so the neighbours of a pair are
// a pair at a constant offset everywhere; a kernel that writes links writes
// the borders' copies too (4 / (L_p / 2) of the links).
//
// At 255 registers a thread carries the staple's matrices of both sites
// without spills, 8 warps per SM.  Iwasaki force + momentum + link update at
// 24^3 x 48: 675 M warp instructions and 1.2 no_instruction stalls per issue in
// the scalar two-row form, 345 M and 0.06 here; at 24^3 x 64 a force launch of
// a trajectory takes 1.16 against 1.03 ms (both kinds of launch of the
// force-gradient step averaged), and 8 such steps 38.9 against 35.0 ms.  Three
// or four blocks per SM spill or take shared memory from L1: 1.19 to 2.0 ms a
// launch.  The plaquette force gains 4% and stays scalar.  capi.cu:pairs_pay
// says which runs go in pairs.
#include "force_impl.cuh"
#include "pair.cuh"

namespace qgb
{

namespace
{

constexpr int PAIR_BS = 128;

// packed position along p of the pair (0 .. half - 1), -2 .. half + 1 with the borders
__device__ __forceinline__ int along(const PairGeo& pg, const Coord& x) { return sel4(x.c, pg.p) - 2; }

__device__ __forceinline__ long pair_site(const PairGeo& pg, long w)
{
  return pg.p == 3 ? w + 2 * pg.stride : box_site(pg.g, w);
}

// W = m at packed site s, and its swapped copies in the borders
__device__ __forceinline__ void store_links(const WField<Pair>& W, const PairGeo& pg, long s, int mu, const M3<Pair>& m)
{
  W.st(s, mu, m);
  const int c = along(pg, coord_of(pg.g, s));
  if (c < 2 || c >= pg.half - 2) {
    M3<Pair> t;
#pragma unroll
    for (int k = 0; k < 9; ++k) t.e[k] = cx<Pair>(swapped(m.e[k].re), swapped(m.e[k].im));
    if (c < 2) W.st(s + pg.half * pg.stride, mu, t);
    if (c >= pg.half - 2) W.st(s - pg.half * pg.stride, mu, t);
  }
}

// The modes of force_epilogue that the packed fields are used for, with the same meaning.
template <int MODE, bool RECT>
__global__ void __launch_bounds__(PAIR_BS, 2) k_force_pair(PairGeo pg, ForceArgs a)
{
  const long w = (long)(blockIdx.x >> 2) * PAIR_BS + threadIdx.x;
  if (w >= pg.pairs) return;
  const int mu = blockIdx.x & 3;
  const long s = pair_site(pg, w), V = pg.g.V;
  const Pair cp(1.0 - 8.0 * a.c1), cr(a.c1);
  const M3<Pair> S = staple_sum_fast<Pair, RECT, true>((const Cx<Pair>*)a.U, pg.g, (int)s, mu, cp, cr);
  const CField<Pair> U{(const Cx<Pair>*)a.U, V};
  const M3<Pair> u = U.ld(s, mu);
  M3<Pair> F = traceless_antiherm(mul_adj(u, S));
  F = scale(Pair(-a.beta / 3.0), F);
  if (MODE == FORCE_UPDATE_EVOLVE) {
    const WField<Pair> P{(Cx<Pair>*)a.out, V}, W{(Cx<Pair>*)a.ev, V};
    M3<Pair> p = P.ld(s, mu);
    axpy(p, Pair(a.dt), F);
    P.st(s, mu, p);
    M3<Pair> wn = mul(exp_su3_pair(scale(Pair(a.ev_eps), p)), a.ev_from_u ? U.ld(s, mu) : W.ld(s, mu));
    if (a.ev_unit == 1) unitarize_pair<float>(wn);
    else if (a.ev_unit == 2) unitarize_pair<double>(wn);
    store_links(W, pg, s, mu, wn);
  } else {
    M3<Pair> Z = F;
    if (MODE == FORCE_FLOW) {
      Z = scale(Pair(a.a), F);
      if (a.zp != nullptr && a.b != 0.0) axpy(Z, Pair(a.b), CField<Pair>{(const Cx<Pair>*)a.zp, V}.ld(s, mu));
      if (a.z != nullptr) WField<Pair>{(Cx<Pair>*)a.z, V}.st(s, mu, Z);
    }
    M3<Pair> un = mul(exp_su3_pair(scale(Pair(a.dt), Z)), u);
    if (a.unitarize) unitarize_pair<float>(un);
    store_links(WField<Pair>{(Cx<Pair>*)a.out, V}, pg, s, mu, un);
  }
}

// Sites of the lattice g that the packed site x holds.
__device__ __forceinline__ void partners(const Geo& g, const PairGeo& pg, Coord x, long& sa, long& sb)
{
  const int L = 2 * pg.half;
  int c = along(pg, x);
  if (c < 0) c += L;
  long base = 0;
#pragma unroll
  for (int k = 3; k >= 0; --k) base = base * g.d[k] + (k == pg.p ? 0 : x.c[k]);
  sa = base + c * pg.stride;
  sb = base + (c >= pg.half ? c - pg.half : c + pg.half) * pg.stride;
}

__global__ void __launch_bounds__(128) k_pair_pack(Geo g, PairGeo pg, const Cx<float>* f, Cx<Pair>* packed)
{
  const long s = (long)blockIdx.x * 128 + threadIdx.x;
  if (s >= pg.g.V) return;
  const int mu = blockIdx.y;
  long sa, sb;
  partners(g, pg, coord_of(pg.g, s), sa, sb);
  const CField<float> F{f, g.V};
  WField<Pair>{packed, pg.g.V}.st(s, mu, joined(F.ld(sa, mu), F.ld(sb, mu)));
}

__global__ void __launch_bounds__(128) k_pair_unpack(Geo g, PairGeo pg, const Cx<Pair>* packed, Cx<float>* f)
{
  const long w = (long)blockIdx.x * 128 + threadIdx.x;
  if (w >= pg.pairs) return;
  const int mu = blockIdx.y;
  const long s = pair_site(pg, w);
  long sa, sb;
  partners(g, pg, coord_of(pg.g, s), sa, sb);
  const M3<Pair> m = CField<Pair>{packed, pg.g.V}.ld(s, mu);
  const WField<float> F{f, g.V};
  F.st(sa, mu, first(m));
  F.st(sb, mu, second(m));
}

}  // namespace

bool pair_geo(const Geo& g, PairGeo* out)
{
  PairGeo pg;
  pg.p = -1;
  // along y and x the borders scatter: 24 x 64 x 25^2 gains 2% (8 x: loses 3%), 64 x 25^3 nothing (8 x 25^3: loses 11%)
  for (int k = 3; k >= 2 && pg.p < 0; --k)
    if (g.d[k] % 2 == 0 && g.d[k] >= 6) pg.p = k;
  if (pg.p < 0 || g.off != 0 || g.r0 != 0 || g.r1 >= 0 || has_box(g) || g.gd[0] != 0) return false;
  pg.half = g.d[pg.p] / 2;
  pg.pairs = g.V / 2;
  pg.stride = 1;
  pg.g.V = 1;
  for (int k = 0; k < 4; ++k) {
    if (k < pg.p) pg.stride *= g.d[k];
    pg.g.d[k] = k == pg.p ? pg.half + 4 : g.d[k];
    pg.g.bl[k] = k == pg.p ? 2 : 0;
    pg.g.bn[k] = k == pg.p ? pg.half : g.d[k];
    pg.g.V *= pg.g.d[k];
  }
  pg.bytes = (size_t)padded_sites(pg.g.V) * 72 * sizeof(Pair);
  *out = pg;
  // the kernel's 32-bit link offsets
  return padded_sites(pg.g.V) * 36 < 2147483647L;
}

cudaError_t launch_pair_pack(const Geo& g, const PairGeo& pg, const void* f, void* packed, cudaStream_t st)
{
  k_pair_pack<<<dim3((unsigned)((pg.g.V + 127) / 128), 4), 128, 0, st>>>(g, pg, (const Cx<float>*)f, (Cx<Pair>*)packed);
  return cudaGetLastError();
}

cudaError_t launch_pair_unpack(const Geo& g, const PairGeo& pg, const void* packed, void* f, cudaStream_t st)
{
  k_pair_unpack<<<dim3((unsigned)((pg.pairs + 127) / 128), 4), 128, 0, st>>>(g, pg, (const Cx<Pair>*)packed,
                                                                            (Cx<float>*)f);
  return cudaGetLastError();
}

cudaError_t launch_force_pair(const PairGeo& pg, ForceMode mode, const ForceArgs& a, cudaStream_t st)
{
  if (a.c1 == 0.0) return cudaErrorInvalidValue;
  const unsigned grid = (unsigned)(4 * ((pg.pairs + PAIR_BS - 1) / PAIR_BS));
  switch (mode) {
    case FORCE_EVOLVE: k_force_pair<FORCE_EVOLVE, true><<<grid, PAIR_BS, 0, st>>>(pg, a); break;
    case FORCE_FLOW: k_force_pair<FORCE_FLOW, true><<<grid, PAIR_BS, 0, st>>>(pg, a); break;
    case FORCE_UPDATE_EVOLVE: k_force_pair<FORCE_UPDATE_EVOLVE, true><<<grid, PAIR_BS, 0, st>>>(pg, a); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace qgb
