// Input features of the value surrogate: relative 5D states (6 features) and
// 8D world nodes (10), each car's position over the extent, heading as cosine
// and sine, speed mapped to [-1, 1].  Shared by the encode kernels (mlp.cu)
// and the fused inference kernel (mlp_fused.cu).
#pragma once
#include <cuda_bf16.h>

#include <cstdint>

namespace pe {

constexpr int kMaxFeatures = 16;  // features are padded to the 16 of one MMA step

struct RelFeatureScale {
  float inv_extent, vp_mid, vp_inv_half, ve_mid, ve_inv_half;
};

inline RelFeatureScale feature_scale(float extent, float vp_lo, float vp_hi, float ve_lo,
                                     float ve_hi) {
  RelFeatureScale f;
  f.inv_extent = 1.f / extent;
  f.vp_mid = 0.5f * (vp_lo + vp_hi);
  f.vp_inv_half = 2.f / (vp_hi - vp_lo);
  f.ve_mid = 0.5f * (ve_lo + ve_hi);
  f.ve_inv_half = 2.f / (ve_hi - ve_lo);
  return f;
}

// Grid of a dense table: relative [vP, vE, psi, y, x] (np unused) or world
// [xP, yP, thP, vP, xE, yE, thE, vE].
struct NodeGrid {
  int n, nh, np, ne;
  float extent, dx, dh, vp_lo, dvp, ve_lo, dve;
  RelFeatureScale f;
};

inline NodeGrid node_grid(int positions, int headings, int p_speeds, int e_speeds,
                          double extent, double p_min, double p_max, double e_min,
                          double e_max) {
  const double pi = 3.14159265358979323846;
  return NodeGrid{positions,
                  headings,
                  p_speeds,
                  e_speeds,
                  (float)extent,
                  (float)(2 * extent / (positions - 1)),
                  (float)(2 * pi / headings),
                  (float)p_min,
                  (float)((p_max - p_min) / (p_speeds - 1)),
                  (float)e_min,
                  (float)((e_max - e_min) / (e_speeds - 1)),
                  feature_scale((float)extent, (float)p_min, (float)p_max, (float)e_min,
                                (float)e_max)};
}

__device__ __forceinline__ void state_features(float v[kMaxFeatures], const RelFeatureScale &f,
                                               float x, float y, float psi, float vp,
                                               float ve) {
  float s, c;
  sincosf(psi, &s, &c);
  v[0] = x * f.inv_extent;
  v[1] = y * f.inv_extent;
  v[2] = c;
  v[3] = s;
  v[4] = (vp - f.vp_mid) * f.vp_inv_half;
  v[5] = (ve - f.ve_mid) * f.ve_inv_half;
#pragma unroll
  for (int k = 6; k < kMaxFeatures; k++) v[k] = 0.f;
}

__device__ __forceinline__ void relative_node_features(float v[kMaxFeatures],
                                                       const NodeGrid &g, int64_t j) {
  const int ix = (int)(j % g.n);
  j /= g.n;
  const int iy = (int)(j % g.n);
  j /= g.n;
  const int ip = (int)(j % g.nh);
  j /= g.nh;
  const int ie = (int)(j % g.ne);
  const int iv = (int)(j / g.ne);
  state_features(v, g.f, fmaf((float)ix, g.dx, -g.extent), fmaf((float)iy, g.dx, -g.extent),
                 fmaf((float)ip, g.dh, -3.14159265358979f), fmaf((float)iv, g.dvp, g.vp_lo),
                 fmaf((float)ie, g.dve, g.ve_lo));
}

__device__ __forceinline__ void world_node_features(float v[kMaxFeatures], const NodeGrid &g,
                                                    int64_t j) {
  const int q7 = (int)(j % g.ne);
  j /= g.ne;
  const int q6 = (int)(j % g.nh);
  j /= g.nh;
  const int q5 = (int)(j % g.n);
  j /= g.n;
  const int q4 = (int)(j % g.n);
  j /= g.n;
  const int q3 = (int)(j % g.np);
  j /= g.np;
  const int q2 = (int)(j % g.nh);
  j /= g.nh;
  const int q1 = (int)(j % g.n);
  const int q0 = (int)(j / g.n);
  float sp, cp, se, ce;
  sincosf(fmaf((float)q2, g.dh, -3.14159265358979f), &sp, &cp);
  sincosf(fmaf((float)q6, g.dh, -3.14159265358979f), &se, &ce);
  v[0] = fmaf((float)q0, g.dx, -g.extent) * g.f.inv_extent;
  v[1] = fmaf((float)q1, g.dx, -g.extent) * g.f.inv_extent;
  v[2] = cp;
  v[3] = sp;
  v[4] = (fmaf((float)q3, g.dvp, g.vp_lo) - g.f.vp_mid) * g.f.vp_inv_half;
  v[5] = fmaf((float)q4, g.dx, -g.extent) * g.f.inv_extent;
  v[6] = fmaf((float)q5, g.dx, -g.extent) * g.f.inv_extent;
  v[7] = ce;
  v[8] = se;
  v[9] = (fmaf((float)q7, g.dve, g.ve_lo) - g.f.ve_mid) * g.f.ve_inv_half;
#pragma unroll
  for (int k = 10; k < kMaxFeatures; k++) v[k] = 0.f;
}

// Eight features as one 16-byte bf16 unit.
__device__ __forceinline__ uint4 pack_features(const float *v) {
  uint4 u;
  __nv_bfloat162 p[4];
#pragma unroll
  for (int k = 0; k < 4; k++) p[k] = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
  u.x = *reinterpret_cast<uint32_t *>(&p[0]);
  u.y = *reinterpret_cast<uint32_t *>(&p[1]);
  u.z = *reinterpret_cast<uint32_t *>(&p[2]);
  u.w = *reinterpret_cast<uint32_t *>(&p[3]);
  return u;
}

}  // namespace pe
