// pair.cuh -- two FP32 reals in one 64-bit register pair, for kernels that
// treat two sites at once with packed arithmetic (fma.rn.f32x2 and its
// relatives): the templates of su3.cuh and force_impl.cuh with R = Pair.
//
// A packed multiply-add does the work of two scalar ones in one issue slot.
// The FP32 Iwasaki force is limited by instruction issue and fetch, not by the
// multiply-add pipe, so halving its instructions shortens it, although the
// pipe's rate is the same.
#pragma once

#include <cuda_runtime.h>

#include "gauge_common.cuh"

namespace qgb
{

struct Pair {
  float2 v;
  Pair() = default;
  __host__ __device__ __forceinline__ Pair(double x) { v.x = v.y = (float)x; }
  __host__ __device__ __forceinline__ Pair(float a, float b)
  {
    v.x = a;
    v.y = b;
  }
};

__device__ __forceinline__ Pair pair_of(float2 x)
{
  Pair p;
  p.v = x;
  return p;
}
__device__ __forceinline__ Pair operator*(Pair a, Pair b) { return pair_of(__fmul2_rn(a.v, b.v)); }
__device__ __forceinline__ Pair operator+(Pair a, Pair b) { return pair_of(__fadd2_rn(a.v, b.v)); }
__device__ __forceinline__ Pair operator-(Pair a) { return Pair(-a.v.x, -a.v.y); }
__device__ __forceinline__ Pair operator-(Pair a, Pair b) { return a + (-b); }
__device__ __forceinline__ Pair operator/(Pair a, Pair b) { return Pair(a.v.x / b.v.x, a.v.y / b.v.y); }
__device__ __forceinline__ Pair fma(Pair a, Pair b, Pair c) { return pair_of(__ffma2_rn(a.v, b.v, c.v)); }
__device__ __forceinline__ Pair& operator+=(Pair& a, Pair b) { return a = a + b; }
__device__ __forceinline__ Pair& operator-=(Pair& a, Pair b) { return a = a - b; }
__device__ __forceinline__ Pair swapped(Pair a) { return Pair(a.v.y, a.v.x); }

// 16 bytes: (re of both sites, im of both sites)
__device__ __forceinline__ Cx<Pair> ldg_cx(const Cx<Pair>* p)
{
  const float4 t = __ldg(reinterpret_cast<const float4*>(p));
  return cx<Pair>(Pair(t.x, t.y), Pair(t.z, t.w));
}

__device__ __forceinline__ M3<float> first(const M3<Pair>& m)
{
  M3<float> r;
#pragma unroll
  for (int k = 0; k < 9; ++k) r.e[k] = cx<float>(m.e[k].re.v.x, m.e[k].im.v.x);
  return r;
}
__device__ __forceinline__ M3<float> second(const M3<Pair>& m)
{
  M3<float> r;
#pragma unroll
  for (int k = 0; k < 9; ++k) r.e[k] = cx<float>(m.e[k].re.v.y, m.e[k].im.v.y);
  return r;
}
__device__ __forceinline__ M3<Pair> joined(const M3<float>& a, const M3<float>& b)
{
  M3<Pair> r;
#pragma unroll
  for (int k = 0; k < 9; ++k) r.e[k] = cx<Pair>(Pair(a.e[k].re, b.e[k].re), Pair(a.e[k].im, b.e[k].im));
  return r;
}

// exp_su3 of both matrices; the recursion stops when the larger one's omitted terms are below FP32 resolution
// (more terms than the other needs are below it too).
__device__ __forceinline__ M3<Pair> exp_su3_pair(const M3<Pair>& a)
{
  Pair h[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    Pair v(0.0);
#pragma unroll
    for (int k = 0; k < 3; ++k)
      v = fma(a.e[3 * i + k].re, a.e[3 * k + i].re, fma(-a.e[3 * i + k].im, a.e[3 * k + i].im, v));
    h[i] = v;
  }
  Cx<Pair> u[3];  // (0,1), (0,2), (1,2)
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int i = q == 2 ? 1 : 0, j = q == 0 ? 1 : 2;
    Pair re(0.0), im(0.0);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      re = fma(a.e[3 * i + k].re, a.e[3 * k + j].re, fma(-a.e[3 * i + k].im, a.e[3 * k + j].im, re));
      im = fma(a.e[3 * i + k].re, a.e[3 * k + j].im, fma(a.e[3 * i + k].im, a.e[3 * k + j].re, im));
    }
    u[q] = cx<Pair>(re, im);
  }
  const Pair s = Pair(-0.5) * (h[0] + h[1] + h[2]);
  Pair t3 = h[0] * a.e[0].im;
  t3 = fma(h[1], a.e[4].im, t3);
  t3 = fma(h[2], a.e[8].im, t3);
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int i = q == 2 ? 1 : 0, j = q == 0 ? 1 : 2;
    const Cx<Pair> aij = a.e[3 * i + j], aji = a.e[3 * j + i];
    t3 = fma(u[q].re, aji.im + aij.im, t3);
    t3 = fma(u[q].im, aji.re - aij.re, t3);
  }
  const float third = 1.0f / 3.0f;
  const Pair delta = t3 * Pair(third, third);
  const float nrm = sqrtf(fmaxf(2.0f * fmaxf(s.v.x, s.v.y), 0.0f));
  const float tol = 7.450580596923828e-9f;
  const Pair ms = -s;
  Cx<Pair> x = cx<Pair>(Pair(1.0), Pair(0.0)), y = cx<Pair>(Pair(0.0), Pair(0.0)), z = y;
  Cx<Pair> f0 = x, f1 = y, f2 = z;
  float term = 1.0f;
#pragma unroll 1
  for (int n = 1; n <= 20; ++n) {
    const float inv1 = qgb_inv_nf[n];
    const Pair inv(inv1, inv1), di = delta * inv;
    const Cx<Pair> xn = cx<Pair>(-(di * z.im), di * z.re);
    const Cx<Pair> yn = cx<Pair>(fma(ms, z.re, x.re) * inv, fma(ms, z.im, x.im) * inv);
    z = cx<Pair>(y.re * inv, y.im * inv);
    x = xn;
    y = yn;
    f0.re += x.re;
    f0.im += x.im;
    f1.re += y.re;
    f1.im += y.im;
    f2.re += z.re;
    f2.im += z.im;
    term *= nrm * inv1;
    if (2.0f * term * nrm < tol * (float)(n + 1) && nrm < 0.5f * (float)(n + 2)) break;
  }
  M3<Pair> r;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      Cx<Pair> q2;
      if (i == j) q2 = cx<Pair>(h[i], Pair(0.0));
      else if (i < j) q2 = u[i + j - 1];
      else q2 = cx<Pair>(u[i + j - 1].re, -u[i + j - 1].im);
      const Cx<Pair> ae = a.e[3 * i + j];
      Pair re = fma(f1.re, ae.re, fma(-f1.im, ae.im, fma(f2.re, q2.re, -(f2.im * q2.im))));
      Pair im = fma(f1.re, ae.im, fma(f1.im, ae.re, fma(f2.re, q2.im, f2.im * q2.re)));
      if (i == j) {
        re += f0.re;
        im += f0.im;
      }
      r.e[3 * i + j] = cx<Pair>(re, im);
    }
  return r;
}

// unitarize_as<C, float> of both matrices
template <typename C>
__device__ __forceinline__ void unitarize_pair(M3<Pair>& m)
{
  M3<float> a = first(m), b = second(m);
  unitarize_as<C, float>(a);
  unitarize_as<C, float>(b);
  m = joined(a, b);
}

}  // namespace qgb
