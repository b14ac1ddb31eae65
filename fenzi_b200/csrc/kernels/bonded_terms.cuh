// Force terms among the atoms of one molecule, shared by the bonded kernel (a thread per
// term) and the integrator's pass over rigid waters (a thread per water).
#pragma once
#include "common.cuh"

namespace fzk {

// minimum-image difference a - b of two FP32 positions, formed in FP64 and rounded once:
// two atoms of a term split by the periodic boundary are about L apart before the image
// shift, and an FP32 difference would round at the ulp of L (up to 3.8e-6 A for
// L = 130 A), a 1e-4 relative error in the force of a stiff bond
__device__ __forceinline__ float3 image_diff(float4 a, float4 b, const SysParams& p) {
  double d[3] = {(double)a.x - (double)b.x, (double)a.y - (double)b.y, (double)a.z - (double)b.z};
  min_image_d(d, p);
  return make_float3((float)d[0], (float)d[1], (float)d[2]);
}
__device__ __forceinline__ float dot(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float3 cross(float3 a, float3 b) {
  return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

// harmonic bond along d = ri - rj (k, r0): force / r on i; *dr the elongation
__device__ __forceinline__ float bond_force(float3 d, float2 prm, float* dr) {
  const float rr = sqrtf(dot(d, d));
  *dr = rr - prm.y;
  return rr > 0.f ? -2.f * prm.x * *dr / rr : 0.f;
}

// harmonic angle between u and v (k, theta0): forces on the ends; *dth the opening
__device__ __forceinline__ void angle_force(float3 u, float3 v, float2 prm, float3* fi, float3* fk, float* dth) {
  const float uu = dot(u, u), vv = dot(v, v), uv = dot(u, v);
  const float3 uxv = cross(u, v);
  const float ruv = rsqrtf(uu * vv);
  const float c = uv * ruv;
  const float s = sqrtf(dot(uxv, uxv)) * ruv;
  *dth = atan2f(s, c) - prm.y;
  const float dE = 2.f * prm.x * *dth;
  const float sf = fmaxf(s, 1e-6f);
  const float k1 = -dE / sf;
  // dtheta/du = -(v/(|u||v|) - c u/|u|^2)/sin ; force = -dE * dtheta/du
  const float3 gu = make_float3(v.x * ruv - c * u.x / uu, v.y * ruv - c * u.y / uu, v.z * ruv - c * u.z / uu);
  const float3 gv = make_float3(u.x * ruv - c * v.x / vv, u.y * ruv - c * v.y / vv, u.z * ruv - c * v.z / vv);
  *fi = make_float3(-k1 * gu.x, -k1 * gu.y, -k1 * gu.z);
  *fk = make_float3(-k1 * gv.x, -k1 * gv.y, -k1 * gv.z);
}

// Ewald exclusion correction E = -CC qq erf(beta r)/r of a pair r2 apart, FP64 (it
// cancels against the self term and the reciprocal sum): force / r on the first atom
__device__ __forceinline__ double excl_force(double r2, double qq, double beta, double* rr, double* erfv) {
  *rr = sqrt(r2);
  *erfv = erf(beta * *rr);
  return kCC * qq * (1.1283791670955126 * beta * *rr * exp(-beta * beta * r2) - *erfv) / (r2 * *rr);
}

// The terms among the three atoms of a rigid water (apex 0, base 1 and 2) that the
// integrator evaluates itself: bonds and exclusion pairs (0,1), (0,2), (1,2), and the
// angle at the apex.
struct UnitTerms {
  float2 bond[3];  // k, r0
  float2 angle;    // k, theta0
  int has;         // bits 0-2 bonds, 3 angle (4: its first atom is base atom 2), 5-7 exclusion pairs
  int pad[3];
};

}  // namespace fzk
