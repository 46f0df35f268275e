// The paths in flight of the wavefront and serving engines: packing of their state (PathStore) and the work of one
// thread on one path -- shading a vertex, gathering its transmittance queries.
//
// After the first bounces a queue holds its paths in the order of their places in the scene, so a stage reads and
// writes path records at random, and DRAM and L2 traffic counts in 32-byte sectors.  With each field an array of
// its own a vertex took 17 sectors and more for 200 bytes; with the record of PathStore, whose halves are what the
// stages read together, it takes 7 and its queries 2.5 each.  12-bounce images, the stages besides extend and
// shadow (shade, gather, sort), before / after: 4.2M paths through 500k Gaussians 9.0 / 6.5 ms, 2.2M paths through 2M Gaussians 5.2 / 3.8 ms.
#pragma once
#include "vp_internal.h"
#include "vp_path.cuh"
#include "vp_traverse.cuh"

namespace vp {

constexpr uint32_t kAliveBit = 1u << 18;
constexpr uint32_t kMetaMask = (1u << 19) - 1u;  // bounce, shadow count, alive; above it the server's request
__device__ __forceinline__ uint32_t meta_bounce(uint32_t m) { return m & 0xFFFFu; }
__device__ __forceinline__ uint32_t meta_nshadow(uint32_t m) { return (m >> 16) & 3u; }
__device__ __forceinline__ uint32_t meta_request(uint32_t m) { return m >> 19; }

__device__ __forceinline__ uint32_t path_meta(const PathStore& b, uint32_t p) { return __float_as_uint(b.st[4u * p].w); }
__device__ __forceinline__ uint32_t path_gauss(const PathStore& b, uint32_t p) {
  return __float_as_uint(b.st[4u * p + 1u].w);
}
__device__ __forceinline__ float path_scatter_t(const PathStore& b, uint32_t p) { return b.st[4u * p + 3u].w; }

__device__ __forceinline__ void path_ray(const PathStore& b, uint32_t p, float3& o, float3& d, uint64_t& key) {
  const float4 o4 = b.ray[2u * p], d4 = b.ray[2u * p + 1u];
  o = f3(o4.x, o4.y, o4.z);
  d = f3(d4.x, d4.y, d4.z);
  key = ((uint64_t)__float_as_uint(d4.w) << 32) | __float_as_uint(o4.w);
}
__device__ __forceinline__ void query_ray(const PathStore& b, uint32_t slot, float3& o, float3& d, uint32_t& seed,
                                          float& seed_tau) {
  const float4 o4 = b.sq[2u * slot], d4 = b.sq[2u * slot + 1u];
  o = f3(o4.x, o4.y, o4.z);
  d = f3(d4.x, d4.y, d4.z);
  seed = __float_as_uint(d4.w);
  seed_tau = o4.w;
}
__device__ __forceinline__ void set_scatter(const PathStore& b, uint32_t p, float3 albedo, float t, uint32_t gauss) {
  b.st[4u * p + 3u] = make_float4(albedo.x, albedo.y, albedo.z, t);
  b.st[4u * p + 1u].w = __uint_as_float(gauss);
}
__device__ __forceinline__ void set_transmittance(const PathStore& b, uint32_t slot, float tau) {
  b.sw[slot].w = tau >= kMaxOpticalDepth ? 0.0f : expf(-tau);
}

__device__ __forceinline__ void store_path(const PathStore& b, uint32_t p, const PathState& s, uint64_t key,
                                           uint32_t meta, uint32_t gauss) {
  b.ray[2u * p] = make_float4(s.o.x, s.o.y, s.o.z, __uint_as_float((uint32_t)key));
  b.ray[2u * p + 1u] = make_float4(s.d.x, s.d.y, s.d.z, __uint_as_float((uint32_t)(key >> 32)));
  float4* st = b.st + 4u * p;
  st[0] = make_float4(s.thr.x, s.thr.y, s.thr.z, __uint_as_float(meta));
  st[1] = make_float4(s.rad.x, s.rad.y, s.rad.z, __uint_as_float(gauss));
  reinterpret_cast<uint4*>(st)[2] = make_uint4((uint32_t)s.rng.state, (uint32_t)(s.rng.state >> 32),
                                               (uint32_t)s.rng.inc, (uint32_t)(s.rng.inc >> 32));
}

__device__ __forceinline__ PathState load_path(const PathStore& b, uint32_t p, uint64_t& key, uint32_t& meta) {
  PathState s;
  path_ray(b, p, s.o, s.d, key);
  const float4* st = b.st + 4u * p;
  const float4 t = st[0], r = st[1];
  const uint4 g = reinterpret_cast<const uint4*>(st)[2];
  s.thr = f3(t.x, t.y, t.z);
  s.rad = f3(r.x, r.y, r.z);
  s.rng.state = ((uint64_t)g.y << 32) | g.x;
  s.rng.inc = ((uint64_t)g.w << 32) | g.z;
  meta = __float_as_uint(t.w);
  s.bounce = meta_bounce(meta);
  return s;
}

// Warp-aggregated queue append, called by all 32 lanes: returns this lane's first slot for its
// `n` (possibly 0) entries; one atomic per warp.
__device__ __forceinline__ uint32_t queue_reserve(uint32_t* counter, uint32_t n) {
  const int lane = threadIdx.x & 31;
  uint32_t incl = n;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += v;
  }
  const uint32_t total = __shfl_sync(kFull, incl, 31);
  uint32_t base = 0;
  if (lane == 31 && total) base = atomicAdd(counter, total);
  base = __shfl_sync(kFull, base, 31);
  return base + incl - n;
}

// A path's vertex, by one thread: phase sample, NEE and roulette; the path's next ray, its transmittance
// queries (sq, sw) and its meta word.  Returns which of the queries need a traversal (bit k) and sets
// ns and alive.  The shadow rays' seed chords are evaluated here, one thread per ray (seed_chord_tau): a ray
// whose seed chord alone reaches MAX_OPTICAL_DEPTH gets T = 0 at once; the others carry the seed's optical
// depth to the query.
__device__ __forceinline__ unsigned shade_path(const SceneView& S, const EnvView& E, const ParamsView& P,
                                               const PathStore& b, uint32_t p, int& ns, bool& alive,
                                               unsigned long long& opaque) {
  uint64_t key;
  uint32_t meta;
  PathState s = load_path(b, p, key, meta);
  const uint32_t gauss = path_gauss(b, p);
  const float4 a = b.st[4u * p + 3u];
  const bool scattered = a.w < kInf;
  ShadowSet sh;
  alive = shade_bounce(E, P, s, scattered, a.w, f3(a.x, a.y, a.z), sh, gauss);
  ns = sh.n;
  unsigned queued = 0u;
  for (int k = 0; k < sh.n; ++k) {
    float seed_tau = -1.0f;  // no seed
    if (sh.seed[k] != kNoGauss)
      seed_tau = P.accurate ? seed_chord_tau<true>(S, sh.seed[k], sh.o[k], sh.d[k])
                            : seed_chord_tau<false>(S, sh.seed[k], sh.o[k], sh.d[k]);
    const bool opaque_k = seed_tau >= kMaxOpticalDepth;
    const uint32_t slot = 3u * p + k;
    b.sw[slot] = make_float4(sh.w[k].x, sh.w[k].y, sh.w[k].z, 0.0f);  // T = 0, or the query's to come
    if (opaque_k) {
      opaque += 1;
      continue;
    }
    b.sq[2u * slot] = make_float4(sh.o[k].x, sh.o[k].y, sh.o[k].z, seed_tau);
    b.sq[2u * slot + 1u] = make_float4(sh.d[k].x, sh.d[k].y, sh.d[k].z, __uint_as_float(sh.seed[k]));
    queued |= 1u << k;
  }
  if (alive) key = draw_bounce_key(s.rng);
  meta = (meta & ~kMetaMask) | (s.bounce & 0xFFFFu) | ((uint32_t)sh.n << 16) | (alive ? kAliveBit : 0u);
  store_path(b, p, s, key, meta, gauss);
  return queued;
}

// radiance += weight x T over a path's queries, in their order.  True while the path lives.
__device__ __forceinline__ bool gather_radiance(const PathStore& b, uint32_t p, float3& rad) {
  const uint32_t m = path_meta(b, p);
  const int ns = (int)meta_nshadow(m);
  const float4 r = b.st[4u * p + 1u];
  rad = f3(r.x, r.y, r.z);
  for (int k = 0; k < ns; ++k) {
    const float4 w = b.sw[3u * p + k];
    rad = add(rad, mul(f3(w.x, w.y, w.z), w.w));
  }
  const bool alive = (m & kAliveBit) != 0u;
  if (alive) b.st[4u * p + 1u] = make_float4(rad.x, rad.y, rad.z, r.w);
  return alive;
}

}  // namespace vp
