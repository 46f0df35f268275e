// The path loop over a query policy, run from any vertex to the path's end: by the warp engine and the
// megakernel (vp_render.cu) and by the wavefront engine's tail (vp_wavefront.cu).
#pragma once

#include "vp_path.cuh"
#include "vp_traverse.cuh"

namespace vp {

struct PathStats {
  unsigned long long bounces = 0, scatters = 0, shadow = 0;
  unsigned int max_overlap = 0;
};

// Runs a path from its current vertex to its end; key: the free-flight key of this bounce, already drawn.
template <class Q>
__device__ __forceinline__ void run_path(const SceneView& S, const EnvView& E, const ParamsView& P, Q& q, PathState& s,
                                         uint64_t key, PathStats& ps) {
  while (true) {
    // Stages 1-3 of sample_scattering_event (sampling.cuh:474-540): ADT argmin over every
    // overlapped Gaussian, with the albedo of the rebuilt active set.  In a scene whose albedo
    // is 0 everywhere a scatter ends the path with zero contribution, so the camera-ray argmin
    // is skipped there (the bounce-0 direct term is the whole image).
    float tstar = kInf;
    ScatterAlbedo sa;
    sa.valid = false;
    if (!(s.bounce == 0 && S.albedo_all_zero)) tstar = q.argmin(s.o, s.d, key, &sa);
    const bool scattered = tstar < kInf;
    float3 albedo = f3(0.f, 0.f, 0.f);
    if (scattered) {
      uint32_t overlap = sa.overlap;
      if (sa.valid) {
        albedo = sa.albedo;
      } else {
        albedo = q.albedo_along(s.o, s.d, tstar, overlap);
        if (S.one_albedo) albedo = S.albedo;
      }
      if (P.measure) ps.max_overlap = max(ps.max_overlap, overlap);
    }
    if (P.measure) {
      ps.bounces++;
      if (scattered) ps.scatters++;
    }
    ShadowSet sh;
    const uint32_t gauss = scattered ? sa.gauss : kNoGauss;
    const bool alive = shade_bounce(E, P, s, scattered, tstar, albedo, sh, gauss);
#pragma unroll 1
    for (int k = 0; k < sh.n; ++k) {  // compute_transmittance_to_env (sampling.cuh:548-583)
      s.rad = add(s.rad, mul(sh.w[k], q.transmittance(sh.o[k], sh.d[k], sh.seed[k])));
      if (P.measure) ps.shadow++;
    }
    if (!alive) return;
    key = draw_bounce_key(s.rng);
  }
}

template <class Q>
__device__ float3 trace_path(const SceneView& S, const EnvView& E, const CameraView& C,
                             const ParamsView& P, Q& q, uint32_t px, uint32_t py,
                             uint64_t sample_index, PathStats& ps) {
  PathState s = start_path(C, P, px, py, sample_index);
  if (P.max_bounces > 0) {
    const uint64_t key = draw_bounce_key(s.rng);
    run_path(S, E, P, q, s, key, ps);
  }
  return finalize_sample(P, s.rad);
}

template <bool kAcc>
struct WarpQueries {
  const SceneView& S;
  const WarpSmem& W;
  uint32_t& status;
  WarpStats& ws;
  bool measure;
  __device__ float argmin(float3 o, float3 d, uint64_t key, ScatterAlbedo* sa) {
    return warp_ray_query<kAcc, kArgmin>(S, W, o, d, key, status, ws, measure, sa);
  }
  __device__ float transmittance(float3 o, float3 d, uint32_t seed = kNoGauss) {
    const float tau = warp_ray_query<kAcc, kTau>(S, W, o, d, 0ull, status, ws, measure, nullptr, seed);
    return tau >= kMaxOpticalDepth ? 0.0f : expf(-tau);
  }
  __device__ float3 albedo_along(float3 o, float3 d, float t, uint32_t& overlap) {
    return warp_scatter_albedo<kAcc>(S, W, o, d, t, overlap, status, ws, measure);
  }
};

__device__ __forceinline__ void flush_stats(Counters* c, const PathStats& ps, const WarpStats& ws,
                                            uint32_t status, bool measure) {
  if (status) atomicOr(&c->status, status);
  if (!measure) return;
  atomicAdd(&c->bounces, ps.bounces);
  atomicAdd(&c->scatters, ps.scatters);
  atomicAdd(&c->shadow_rays, ps.shadow);
  atomicAdd(&c->crossings, ws.crossings);
  atomicAdd(&c->nodes, ws.nodes);
  atomicAdd(&c->leaves, ws.leaves);
  for (int k = 0; k < 3; ++k) {
    atomicAdd(&c->kind_nodes[k], ws.kind_nodes[k]);
    atomicAdd(&c->kind_leaves[k], ws.kind_leaves[k]);
    atomicAdd(&c->kind_prims[k], ws.kind_prims[k]);
    atomicAdd(&c->kind_geo[k], ws.kind_geo[k]);
  }
  atomicMax(&c->max_hits, ws.max_hits);
  atomicMax(&c->max_overlap, ps.max_overlap);
}

}  // namespace vp
