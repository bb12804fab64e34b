// Radial envelope and powers shared by the edge-geometry kernels.
#pragma once
#include "ictc_common.cuh"
#include "generated/harmonics_tables.cuh"

namespace ictc {

template <int A> __device__ __forceinline__ float ipw(float x) { return A == 0 ? 1.f : (A == 1 ? x : x * x); }
template <int A> __device__ __forceinline__ float dpw(float x) { return A == 0 ? 0.f : (A == 1 ? 1.f : 2.f * x); }

// polynomial cutoff envelope of order p and its derivative (mace_ictc/models/radial_basis.py:11-92)
__device__ __forceinline__ void envelope(float r, float r_max, int p, float& env, float& denv) {
  const float u = r / r_max;
  if (!(r < r_max)) { env = 0.f; denv = 0.f; return; }
  const float pf = float(p);
  const float up = powf(u, float(p - 1));   // u^(p-1)
  const float a = (pf + 1.f) * (pf + 2.f) * 0.5f, b = pf * (pf + 2.f), c = pf * (pf + 1.f) * 0.5f;
  env = 1.f - a * up * u + b * up * u * u - c * up * u * u * u;
  denv = (-a * pf * up + b * (pf + 1.f) * up * u - c * (pf + 2.f) * up * u * u) / r_max;
}

// harmonics of a unit vector, and the gradient of sum_h g[h] Y_h with respect to it
__device__ __forceinline__ void harmonics_value(float x, float y, float z, float (&val)[9]) {
#pragma unroll
  for (int h = 0; h < 9; ++h) val[h] = 0.f;
#define ICTC_T(h, aa, bb, cc, cf) val[h] = fmaf(cf, ipw<aa>(x) * ipw<bb>(y) * ipw<cc>(z), val[h]);
  ICTC_HARM_TERMS(ICTC_T)
#undef ICTC_T
}
__device__ __forceinline__ void harmonics_vjp(float x, float y, float z, const float (&g)[9], float& d0, float& d1, float& d2) {
  d0 = d1 = d2 = 0.f;
#define ICTC_T(h, aa, bb, cc, cf)                                        \
  d0 = fmaf(g[h] * (cf), dpw<aa>(x) * ipw<bb>(y) * ipw<cc>(z), d0);       \
  d1 = fmaf(g[h] * (cf), ipw<aa>(x) * dpw<bb>(y) * ipw<cc>(z), d1);       \
  d2 = fmaf(g[h] * (cf), ipw<aa>(x) * ipw<bb>(y) * dpw<cc>(z), d2);
  ICTC_HARM_TERMS(ICTC_T)
#undef ICTC_T
}

// Gradient of an edge with respect to its vector, from the gradient of its harmonics (g) and of its radial basis
// (drb, null: none).  (x, y, z) unit vector, r length.
__device__ __forceinline__ float3 edge_vector_gradient(float x, float y, float z, float r, const float (&g)[9],
                                                       const float* drb, int num_basis, int p, float r_max) {
  float d0, d1, d2;
  harmonics_vjp(x, y, z, g, d0, d1, d2);
  float dr = 0.f;
  if (drb) {
    float env, denv;
    envelope(r, r_max, p, env, denv);
    const float rs = fmaxf(r, 1e-12f);
    const float pref = sqrtf(2.f / r_max);
    const float w = 3.14159265358979323846f / r_max;
    for (int k = 0; k < num_basis; ++k) {
      const float wk = w * float(k + 1);
      float s, c;
      sincosf(r * wk, &s, &c);
      const float f = pref * s / rs;                      // bessel value
      const float df = pref * (wk * c / rs - s / (rs * rs));
      dr = fmaf(drb[k], df * env + f * denv, dr);
    }
  }
  const float rc = fmaxf(r, 1e-8f);
  const float dot = x * d0 + y * d1 + z * d2;
  return make_float3(dr * x + (d0 - dot * x) / rc, dr * y + (d1 - dot * y) / rc, dr * z + (d2 - dot * z) / rc);
}

}  // namespace ictc
