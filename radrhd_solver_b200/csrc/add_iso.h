// The isotropic part of a scattering row added to a float: compiled for the device, and by the tests for the host.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define RRHD_BOTH __host__ __device__ __forceinline__
#else
#define RRHD_BOTH inline
#endif

// v + iso, iso = hi + lo (a double split in two floats), rounded to float once but for terms of
// 2^-48 iso: conversions to double and back run at a fraction of the FP32 rate and were a third of
// the scattering drain's store phase.  The sum of v and hi is taken apart in the form that needs
// neither to be the larger (signed intensities leave an anisotropic part above the isotropic one);
// where it is not finite it is the result.  Additions only: there is nothing to contract.
RRHD_BOTH float add_iso(float v, float hi, float lo) {
  const float s = hi + v;
  const float b = s - hi;
  const float e = (hi - (s - b)) + (v - b);
  return fabsf(s) < INFINITY ? s + (e + lo) : s;
}

#ifdef __CUDACC__
// The same for two columns of a row: the same operations, two to an instruction (a - b as the fused
// b (-1) + a, which rounds once as well).
__device__ __forceinline__ void add_iso2(float &v0, float &v1, float hi, float lo) {
  const float2 v = make_float2(v0, v1), h = make_float2(hi, hi), m = make_float2(-1.f, -1.f);
  const float2 s = __fadd2_rn(h, v);
  const float2 b = __ffma2_rn(h, m, s);
  const float2 e = __fadd2_rn(__ffma2_rn(__ffma2_rn(b, m, s), m, h), __ffma2_rn(b, m, v));
  const float2 r = __fadd2_rn(s, __fadd2_rn(e, make_float2(lo, lo)));
  v0 = fabsf(s.x) < INFINITY ? r.x : s.x;
  v1 = fabsf(s.y) < INFINITY ? r.y : s.y;
}
#endif
