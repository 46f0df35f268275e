// Wavefront engine: the path loop as a sequence of small persistent kernels over queues of
// paths, with the path state in device memory between stages.
//
//   generate  (thread per path)  camera ray, PCG32 stream, first free-flight key
//   per bounce, while any path is alive:
//     extend  (thread per path)  free-flight argmin over the 8-wide BVH + albedo at the scatter point
//     shade   (thread per path)  phase sample, NEE sampling, escape rule, roulette; compacts
//                                surviving paths into the next queue and the bounce's
//                                transmittance queries into the shadow queue
//     shadow  (thread per query) transmittance over the 8-wide BVH with early exit at tau >= 88
//     gather  (thread per path)  radiance += weight x T in query order; finished paths write
//                                their sample
//   tail      (a few paths a warp) once few paths are left: they run to their ends in one launch; then, a
//                                thread per pixel, the running mean over the batch's samples in order
//
//   extend, shadow and tail run thread per ray over the compressed 8-wide BVH (vp_trace8.cuh); the scatter-point
//   albedo is then the scene's, when all its Gaussians share one, or a second traversal.
//   Their warp-per-ray forms over the BVH32 give the same results: they count (VP_MEASURE_COUNTERS), serve scenes
//   without an 8-wide tree (too deep, or of Gaussians that fill most of it) and take the last paths where
//   Gaussians differ in albedo.
//
// Each kernel is a fraction of the fused path loop's code and registers, so more warps are
// resident per SM to hide the latency of the dependent node loads.  The reference found a
// wavefront 100x slower than its megakernel because ~352 B of per-ray sets and hit buffers
// streamed through DRAM each bounce (latex/chapters/06-optimization.tex:438-446); here no hit
// buffer or active set survives a stage (the queries rebuild them from geometry), and the ~280 B a
// path carries are laid out by what the stages read together (vp_pathstore.cuh).  Results are
// those of the warp engine: the same shading code (vp_path.cuh), the same queries, and the
// same order of radiance accumulation.
#include <algorithm>

#include <cooperative_groups.h>

#include "vp_internal.h"
#include "vp_pathloop.cuh"
#include "vp_pathstore.cuh"
#include "vp_trace8.cuh"

namespace vp {
namespace {

// Resident 256-thread blocks per SM the warp-per-ray extend / shadow kernels' register budgets are sized for:
// 4 (64 registers) for extend; 5 (48 registers, some spills) for the FP32 shadow kernel, whose
// smaller state gains more from the extra warps than it loses to the spills.  The ACCURATE shadow kernel keeps
// the extend budget.
#ifndef VP_WF_MIN_BLOCKS
#define VP_WF_MIN_BLOCKS 4
#endif
#ifndef VP_WF_SHADOW_MIN_BLOCKS
#define VP_WF_SHADOW_MIN_BLOCKS 5
#endif
// Hit-buffer entries of the extend kernel (chords retained for the scatter-point albedo plus
// one leaf's new ones); the shadow kernel retains none and uses 32.
#ifndef VP_WF_EXTEND_HIT_CAP
#define VP_WF_EXTEND_HIT_CAP 64
#endif
constexpr int kExtendHitCap = VP_WF_EXTEND_HIT_CAP;
// Queues shorter than this are not re-sorted (the sort would cost more than it saves).
#ifndef VP_WF_SORT_MIN
#define VP_WF_SORT_MIN 65536
#endif
constexpr uint32_t kSortMinPaths = VP_WF_SORT_MIN;
// At most this many paths go to the tail: as stages, a bounce of few paths is launches, polls and each stage's
// slowest ray.  64-bounce images, ms as stages / with the tail from 16k / 64k / 128k paths: 4k paths 4.4 / 1.9 /
// 1.9 / 1.8 (50k-Gaussian cloud), 5.3 / 2.5 / 2.4 / 2.4 (500k); 65k paths 5.6 / 3.5 / 3.0 / 3.2, 7.3 / 5.0 / 4.6 /
// 4.4; a 12-bounce image of 361k paths 4.4 from 64k, 5.0 from 128k.
constexpr uint32_t kTailMax = 65536;
// With a warp on each path the tail takes as many as are resident at once, so that none waits for another; in an
// image of more than kTailDeep bounces, whose paths mostly end on the way, twice as many.  12-bounce images of 4.2k / 10.8k
// paths from one / two a resident warp on: 3,000 Gaussians of differing albedos 1.27 / 1.82 and 1.47 / 1.82 ms, 100k
// ACCURATE 1.60 / 1.68 and 1.69 / 2.20; 64 bounces, 10k 1.51 / 2.16 and 1.41 / 1.87, 500k 2.79 / 5.83 and 2.61 / 5.07.
constexpr uint32_t kTailDeep = 32;
// By threads it takes two a resident warp where Gaussians fill more of the scene than kTailOverlap (vp_build.cu,
// k_overlap): its few paths a warp wait for one another's long rays.  20,000 Gaussians, scales of 0.15 in a
// box of side 2 (0.11), 11k / 30k / 60k paths: 17.0 / 29.9 / 49.6 ms from 64k on, 15.6 / 27.4 / 42.1 from 4.7k; scales of
// 0.1 (0.06) 5.2 / 9.8 / 16.2 and 5.4 / 9.6 / 15.6.  ACCURATE chords cost more, and the line lies lower: 10k Gaussians
// in clusters (0.03), 12 bounces of 11k / 60k paths 1.58 / 3.03 ms from 64k on, 1.42 / 2.16 from 4.7k, 64 bounces of 8k / 60k
// 2.10 / 4.00 from 64k, 1.97 / 3.48 from 16k.
constexpr float kTailOverlap = 0.1f, kTailOverlapAccurate = 0.02f;
constexpr uint32_t kTailMaxAccurate = 16384;
// Scenes whose Gaussians differ in albedo take their few paths with a warp on each, whose one traversal keeps
// the chords at the scatter point: extend from this many paths on by threads (two traversals, at 2 blocks an SM),
// shadow from this many.  12-bounce images of 11k / 30k / 60k paths, threads / warps / this: 3,000 Gaussians 1.15 / 1.62 /
// 1.93, 0.66 / 1.02 / 1.33 and 0.65 / 1.03 / 1.29 ms; 10k in clusters 1.88 / 2.62 / 3.58, 1.22 / 1.74 / 2.52 and 1.22 /
// 1.64 / 2.09.
constexpr uint32_t kMixedExtendMin = 65536, kMixedShadowMin = 16384;
// Resident blocks per SM of its register budget: 2 (128 registers) against 3: 4k paths 1.9 / 2.2 ms (50k), 2.4 /
// 2.8 (500k).
constexpr int kTailBlocks = 2;



// Path p is sample p % batch of pixel p / batch.  Without adaptive sampling every path starts
// and queue slot p holds path p.  With it, the host has cleared the counters and only the paths
// of pixels that have not converged join the queue (their order within a warp is kept).
__global__ void k_wf_generate(CameraView C, ParamsView P, uint32_t spp_offset, uint32_t batch, uint32_t n,
                              WfBuffers b, const float4* __restrict__ mean, const float4* __restrict__ m2,
                              const uint32_t* __restrict__ count, Counters* __restrict__ ctr) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  const bool adaptive = P.adaptive_threshold > 0.0f;
  uint32_t slot = p;
  if (!adaptive) {
    if (p == 0) {
      b.ctr[0] = P.max_bounces > 0 ? n : 0u;
      b.ctr[1] = b.ctr[2] = b.ctr[3] = b.ctr[4] = 0u;
    }
    if (p >= n) return;
  } else {
    bool live = false;
    if (p < n) {
      const uint32_t pixel = p / batch;
      live = !pixel_converged(P, count[pixel], mean[pixel], m2[pixel]);
      if (!live && p % batch == 0u) atomicAdd(&ctr->skipped, (unsigned long long)batch);
    }
    slot = queue_reserve(b.ctr + 0, live && P.max_bounces > 0 ? 1u : 0u);  // all 32 lanes: blockDim is a multiple of 32
    if (!live) return;
  }
  b.L4[p] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (P.max_bounces == 0) return;  // no vertex: the sample is black
  const uint32_t pixel = p / batch, s = p % batch;
  PathState st = start_path(C, P, pixel % P.width, pixel / P.width, (uint64_t)spp_offset + s);
  const uint64_t key = draw_bounce_key(st.rng);
  store_path(b, p, st, key, kAliveBit, kNoGauss);
  b.qa[slot] = p;
}

// kMeasure = false compiles the statistics out (their registers would otherwise stay live
// through the traversal loop).
template <bool kAcc, bool kMeasure>
__global__ void __launch_bounds__(256, VP_WF_MIN_BLOCKS) k_wf_extend(SceneView S, ParamsView P, WfBuffers b, const uint32_t* q,
                                                   const uint32_t* count, unsigned int* work, Counters* ctr) {
  extern __shared__ unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  WarpSmem W = carve(smem + kRootStageBytes + warp * warp_smem_bytes(S.argmin_cap, kExtendHitCap), S.argmin_cap,
                     kExtendHitCap);
  if constexpr (VP_STAGE_ROOT) {
    stage_root(S.wide, S.wide_root);
    W.root_staged = true;
  }
  const uint32_t n = *count;
  uint32_t status = 0, max_overlap = 0;
  unsigned long long bounces = 0, scatters = 0;
  WarpStats ws;
  const bool measure = kMeasure && P.measure != 0;
  if (measure) ws.hist = &ctr->hits_hist[0][0];
  while (true) {
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(work, 1u);
    item = __shfl_sync(kFull, item, 0);
    if (item >= n) break;
    const uint32_t p = __ldg(q + item);
    const uint32_t bounce = meta_bounce(path_meta(b, p));
    float3 of, df;
    uint64_t key;
    path_ray(b, p, of, df, key);
    float tstar = kInf;
    ScatterAlbedo sa;
    sa.valid = false;
    if (!(bounce == 0 && S.albedo_all_zero))
      tstar = warp_ray_query<kAcc, kArgmin>(S, W, of, df, key, status, ws, measure, &sa);
    float3 albedo = f3(0.f, 0.f, 0.f);
    if (tstar < kInf) {
      uint32_t ov = sa.overlap;
      albedo = sa.valid ? sa.albedo : warp_scatter_albedo<kAcc>(S, W, of, df, tstar, ov, status, ws, measure);
      if (S.one_albedo) albedo = S.albedo;
      max_overlap = max(max_overlap, ov);
      ++scatters;
    }
    ++bounces;
    if (lane == 0) set_scatter(b, p, albedo, tstar, tstar < kInf ? sa.gauss : kNoGauss);
    if (status) break;
  }
  if (lane == 0) {
    if (status) atomicOr(&ctr->status, status);
    if (measure) {
      atomicAdd(&ctr->bounces, bounces);
      atomicAdd(&ctr->scatters, scatters);
      atomicMax(&ctr->max_overlap, max_overlap);
      atomicAdd(&ctr->crossings, ws.crossings);
      atomicAdd(&ctr->nodes, ws.nodes);
      atomicAdd(&ctr->leaves, ws.leaves);
      atomicMax(&ctr->max_hits, ws.max_hits);
      for (int k = 0; k < 3; ++k) {
        atomicAdd(&ctr->kind_nodes[k], ws.kind_nodes[k]);
        atomicAdd(&ctr->kind_leaves[k], ws.kind_leaves[k]);
        atomicAdd(&ctr->kind_prims[k], ws.kind_prims[k]);
        atomicAdd(&ctr->kind_geo[k], ws.kind_geo[k]);
      }
    }
  }
}

// ---- thread-per-ray stages (vp_trace8.cuh) -----------------------------------------------------

template <bool kAcc, bool kMixed>
__global__ void __launch_bounds__(kT8Threads, kMixed ? 2 : kT8Blocks) k_wf_extend8(SceneView S, WfBuffers b, const uint32_t* q,
                                                                     const uint32_t* count, unsigned int* work,
                                                                     Counters* ctr) {
  uint32_t* smem = reinterpret_cast<uint32_t*>(vp_dyn_smem) + (threadIdx.x >> 5) * trace8_warp_words(S.depth8);
  uint32_t status = 0;
  extend8<kAcc, kMixed>(
      OneScene8{scene8_of(S)}, S.depth8, smem, *count, work, status,
      [&](uint32_t item, Ray8& ray) {
        const uint32_t p = __ldg(q + item);
        const uint32_t bounce = meta_bounce(path_meta(b, p));
        if (S.albedo_all_zero && bounce == 0u) {  // a scatter would end the path with nothing
          set_scatter(b, p, f3(0.f, 0.f, 0.f), kInf, kNoGauss);
          return false;
        }
        path_ray(b, p, ray.o, ray.d, ray.key);
        ray.seed = bounce ? path_gauss(b, p) : kNoGauss;
        return true;
      },
      [&](uint32_t item, const Ray8&, const Hit8& h) {
        const uint32_t p = __ldg(q + item);
        set_scatter(b, p, h.t < kInf ? S.albedo : f3(0.f, 0.f, 0.f), h.t, h.gauss);
      },
      [&](uint32_t item, Ray8& ray) {
        const uint32_t p = __ldg(q + item);
        ray.t = path_scatter_t(b, p);
        if (!(ray.t < kInf)) return false;
        path_ray(b, p, ray.o, ray.d, ray.key);
        return true;
      },
      [&](uint32_t item, const Ray8& ray, float3 a) {
        b.st[4u * __ldg(q + item) + 3u] = make_float4(a.x, a.y, a.z, ray.t);
      });
  if (status) atomicOr(&ctr->status, status);
}

template <bool kAcc>
__global__ void __launch_bounds__(kT8Threads, kT8Blocks) k_wf_shadow8(SceneView S, WfBuffers b, const uint32_t* count,
                                                                        unsigned int* work, Counters* ctr) {
  uint32_t* smem = reinterpret_cast<uint32_t*>(vp_dyn_smem) + (threadIdx.x >> 5) * trace8_warp_words(S.depth8);
  const uint32_t n = *count;
  uint32_t status = 0;
  trace8<kAcc, kTau8>(
      OneScene8{scene8_of(S)}, S.depth8, smem, stage_order8(), n, work, grid_warps(), rays_per_warp(n, grid_warps()), status,
      [&](uint32_t item, Ray8& ray) {
        query_ray(b, __ldg(b.qs + item), ray.o, ray.d, ray.seed, ray.seed_tau);
        return true;
      },
      [&](uint32_t item, const Ray8&, const Hit8& h) { set_transmittance(b, __ldg(b.qs + item), (float)h.w); });
  if (status) atomicOr(&ctr->status, status);
}

// Bound by the latency of its path records (DRAM: random after the first sort) at 2 resident blocks; more blocks
// only widen the set of records in L2: 3 / 4 / 5 blocks an SM took 9.6 / 10.7 / 11.9 ms against 9.0 (with gather and
// sort; 4.2M paths, 500k Gaussians), so what helps is fewer sectors a path (vp_pathstore.cuh).
__global__ void __launch_bounds__(256) k_wf_shade(SceneView S, EnvView E, ParamsView P, WfBuffers b,
                                                  const uint32_t* q, const uint32_t* count, uint32_t* qnext,
                                                  uint32_t* cnext, Counters* ctr) {
  const uint32_t n = *count;
  unsigned long long shadows = 0, opaque = 0;
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x / 32);
  const uint32_t wid = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  // warp-uniform loop: every lane runs every iteration, so the queue appends are full-warp
  for (uint32_t base = wid * 32u; base < n; base += warps * 32u) {
    const uint32_t i = base + lane;
    const bool valid = i < n;
    uint32_t p = 0;
    int ns = 0;
    unsigned queued = 0u;  // bit k: shadow ray k enters the shadow queue
    bool alive = false;
    if (valid) {
      p = q[i];
      queued = shade_path(S, E, P, b, p, ns, alive, opaque);
    }
    shadows += (unsigned)ns;
    uint32_t slot = queue_reserve(b.ctr + 2, (uint32_t)__popc(queued));
    for (int k = 0; k < ns; ++k)
      if (queued & (1u << k)) b.qs[slot++] = 3u * p + k;
    const uint32_t qslot = queue_reserve(cnext, alive ? 1u : 0u);
    if (alive) qnext[qslot] = p;
  }
  if (P.measure) {
    for (int o = 16; o > 0; o >>= 1) {
      shadows += __shfl_xor_sync(0xFFFFFFFFu, shadows, o);
      opaque += __shfl_xor_sync(0xFFFFFFFFu, opaque, o);
    }
    if ((threadIdx.x & 31) == 0 && shadows) atomicAdd(&ctr->shadow_rays, shadows);
    if ((threadIdx.x & 31) == 0 && opaque) {  // transmittance queries answered by their seed chord
      atomicAdd(&ctr->crossings, opaque);
      atomicAdd(&ctr->hits_hist[1][1], opaque);
      atomicMax(&ctr->max_hits, 1u);
    }
  }
}

template <bool kAcc, bool kMeasure>
__global__ void __launch_bounds__(256, kAcc ? VP_WF_MIN_BLOCKS : VP_WF_SHADOW_MIN_BLOCKS) k_wf_shadow(SceneView S, WfBuffers b, const uint32_t* count,
                                                   unsigned int* work, Counters* ctr, int measure_i) {
  extern __shared__ unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  WarpSmem W = carve(smem + kRootStageBytes + warp * warp_smem_bytes(S.stack_cap, 32), S.stack_cap, 32);
  if constexpr (VP_STAGE_ROOT) {
    stage_root(S.wide, S.wide_root);
    W.root_staged = true;
  }
  const uint32_t n = *count;
  uint32_t status = 0;
  WarpStats ws;
  const bool measure = kMeasure && measure_i != 0;
  if (measure) ws.hist = &ctr->hits_hist[0][0];
  while (true) {
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(work, 1u);
    item = __shfl_sync(kFull, item, 0);
    if (item >= n) break;
    const uint32_t slot = __ldg(b.qs + item);
    float3 o, d;
    uint32_t seed;
    float seed_tau;
    query_ray(b, slot, o, d, seed, seed_tau);
    const float tau = warp_ray_query<kAcc, kTau>(S, W, o, d, 0ull, status, ws, measure, nullptr, seed, seed_tau);
    if (lane == 0) set_transmittance(b, slot, tau);
    if (status) break;
  }
  if (lane == 0) {
    if (status) atomicOr(&ctr->status, status);
    if (measure) {
      atomicAdd(&ctr->crossings, ws.crossings);
      atomicAdd(&ctr->nodes, ws.nodes);
      atomicAdd(&ctr->leaves, ws.leaves);
      atomicMax(&ctr->max_hits, ws.max_hits);
      for (int k = 0; k < 3; ++k) {
        atomicAdd(&ctr->kind_nodes[k], ws.kind_nodes[k]);
        atomicAdd(&ctr->kind_leaves[k], ws.kind_leaves[k]);
        atomicAdd(&ctr->kind_prims[k], ws.kind_prims[k]);
        atomicAdd(&ctr->kind_geo[k], ws.kind_geo[k]);
      }
    }
  }
}

// radiance += weight x T over a path's queries, in their order; an ended path writes its sample.
__device__ __forceinline__ void gather_path(const ParamsView& P, const WfBuffers& b, uint32_t p) {
  float3 rad;
  if (!gather_radiance(b, p, rad)) {
    const float3 L = finalize_sample(P, rad);
    b.L4[p] = make_float4(L.x, L.y, L.z, 0.f);
  }
}

__global__ void __launch_bounds__(256) k_wf_gather(ParamsView P, WfBuffers b, const uint32_t* q,
                                                   const uint32_t* count) {
  const uint32_t n = *count;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    gather_path(P, b, q[i]);
  }
}

// Next bounce: the new queue becomes current; shadow queue and work heads restart.
__global__ void k_wf_advance(uint32_t* ctr) {
  ctr[0] = ctr[1];
  ctr[1] = 0u;
  ctr[2] = 0u;
  ctr[3] = 0u;
  ctr[4] = 0u;
}

// Welford mean over the batch's samples of one pixel, in sample order (raygen.cuh:214-242).
// With adaptive sampling it also keeps M2, and a pixel that k_wf_generate found converged (the
// same test on the same, still unchanged state) keeps its state.
__device__ __forceinline__ void welford_pixel(const ParamsView& P, const WfBuffers& b, uint32_t batch, uint32_t pix,
                                              float4* __restrict__ mean, float4* __restrict__ m2,
                                              uint32_t* __restrict__ count) {
  const bool adaptive = P.adaptive_threshold > 0.0f;
  const uint32_t prev = count[pix];
  const float4 m4 = mean[pix];
  const float4 q4 = adaptive ? m2[pix] : make_float4(0.f, 0.f, 0.f, 0.f);
  if (adaptive && pixel_converged(P, prev, m4, q4)) return;
  float3 m = f3(m4.x, m4.y, m4.z), q = f3(q4.x, q4.y, q4.z);
  for (uint32_t s = 0; s < batch; ++s) {
    const float4 L = b.L4[(size_t)pix * batch + s];
    welford_step<true>(m, q, f3(L.x, L.y, L.z), prev + s + 1u);
  }
  mean[pix] = make_float4(m.x, m.y, m.z, 0.f);
  if (adaptive) m2[pix] = make_float4(q.x, q.y, q.z, 0.f);
  count[pix] = prev + batch;
}

// The end of a batch, one cooperative launch: the paths still queued run to their ends, and once all have
// finished the pixels' means take the batch's samples.  This form, a warp on each path over the BVH32 (the
// warp engine's path loop), counts and serves scenes without the 8-wide tree or of differing albedos.
template <bool kAcc, bool kMeasure>
__global__ void __launch_bounds__(256, kTailBlocks) k_wf_tail(SceneView S, EnvView E, ParamsView P, WfBuffers b, const uint32_t* q,
                                                 const uint32_t* count, unsigned int* work, Counters* ctr,
                                                 uint32_t batch, uint32_t n_pix, float4* __restrict__ mean,
                                                 float4* __restrict__ m2, uint32_t* __restrict__ pix_count) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  WarpSmem W = carve(vp_dyn_smem + kRootStageBytes + warp * warp_smem_bytes(S.argmin_cap, kExtendHitCap), S.argmin_cap,
                     kExtendHitCap);
  if constexpr (VP_STAGE_ROOT) {
    stage_root(S.wide, S.wide_root);
    W.root_staged = true;
  }
  if constexpr (!kMeasure) P.measure = 0;
  const uint32_t n = *count;
  uint32_t status = 0;
  WarpStats ws;
  PathStats ps;
  const bool measure = kMeasure && P.measure != 0;
  if (measure) ws.hist = &ctr->hits_hist[0][0];
  WarpQueries<kAcc> queries{S, W, status, ws, measure};
  while (n != 0u) {
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(work, 1u);
    item = __shfl_sync(kFull, item, 0);
    if (item >= n) break;
    const uint32_t p = __ldg(q + item);
    uint64_t key;
    uint32_t meta;
    PathState s = load_path(b, p, key, meta);
    run_path(S, E, P, queries, s, key, ps);
    const float3 L = finalize_sample(P, s.rad);
    if (lane == 0) b.L4[p] = make_float4(L.x, L.y, L.z, 0.f);
    if (status) break;
  }
  if (lane == 0) flush_stats(ctr, ps, ws, status, measure);
  cooperative_groups::this_grid().sync();
  for (uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x; pix < n_pix; pix += gridDim.x * blockDim.x)
    welford_pixel(P, b, batch, pix, mean, m2, pix_count);
}

// The same, thread per ray (vp_trace8.cuh): a warp keeps up to `share` of the queued paths and runs its own
// little wavefront over them -- one traversal for the paths' next free flights and the transmittance
// queries of their last vertices together, then a lane per path gathers and shades -- so no bounce waits for
// another warp's.  For scenes of one albedo.
constexpr uint32_t kTailShare = 16;
struct TailWarp {  // in shared memory, after the traversal's
  uint32_t path[32];               // this round's paths: flying ones first, then those that only have queries left
  uint32_t query[3 * kTailShare];  // shadow-query slots to trace
  uint32_t next;
};
template <bool kAcc>
__global__ void __launch_bounds__(kT8Threads, kTailBlocks) k_wf_tail8(SceneView S, EnvView E, ParamsView P, WfBuffers b,
                                                                     const uint32_t* q, const uint32_t* count,
                                                                     unsigned int* work, Counters* ctr, uint32_t batch,
                                                                     uint32_t n_pix, float4* __restrict__ mean,
                                                                     float4* __restrict__ m2,
                                                                     uint32_t* __restrict__ pix_count) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  uint32_t* smem = reinterpret_cast<uint32_t*>(vp_dyn_smem) + warp * trace8_warp_words(S.depth8);
  TailWarp& T = reinterpret_cast<TailWarp*>(vp_dyn_smem + trace8_smem_bytes(S.depth8, kT8Threads))[warp];
  const uint8_t* order = stage_order8();
  const OneScene8 scene{scene8_of(S)};
  const uint32_t n = *count, warps = grid_warps();
  const uint32_t share = min(kTailShare, max(1u, (n + warps - 1u) / warps));
  uint32_t status = 0, flying = 0, ending = 0, queries = 0;  // the warp's paths and queries in T
  bool more = n != 0u;
  unsigned long long opaque = 0;
  while (true) {
    if (more && flying + ending < share) {  // (ending paths leave after this round)
      const uint32_t want = share - flying - ending;
      uint32_t first = 0;
      if (lane == 0) first = atomicAdd(work, want);
      first = __shfl_sync(kFull, first, 0);
      const uint32_t got = first < n ? min(want, n - first) : 0u;
      more = first + want < n;
      // new paths go behind the flying ones, in front of the ending
      uint32_t keep = 0;
      if ((uint32_t)lane < ending) keep = T.path[flying + lane];
      __syncwarp();
      if ((uint32_t)lane < got) {
        const uint32_t p = __ldg(q + first + lane);
        T.path[flying + lane] = p;
        b.st[4u * p].w = __uint_as_float(path_meta(b, p) & ~(3u << 16));  // its last vertex's queries are gathered already
      }
      if ((uint32_t)lane < ending) T.path[flying + got + lane] = keep;
      flying += got;
    }
    if (flying + ending == 0u) break;
    if (lane == 0) T.next = 0u;
    __syncwarp();
    const uint32_t rays = flying + queries;
    trace8<kAcc, kBoth8>(
        scene, S.depth8, smem, order, rays, &T.next, 1u, (int)min(32u, rays), status,
        [&](uint32_t i, Ray8& ray) {
          ray.flight = i < flying;
          if (ray.flight) {
            const uint32_t p = T.path[i];
            path_ray(b, p, ray.o, ray.d, ray.key);
            ray.seed = meta_bounce(path_meta(b, p)) ? path_gauss(b, p) : kNoGauss;
          } else {
            query_ray(b, T.query[i - flying], ray.o, ray.d, ray.seed, ray.seed_tau);
          }
          return true;
        },
        [&](uint32_t i, const Ray8&, const Hit8& h) {
          if (i < flying) {
            set_scatter(b, T.path[i], h.t < kInf ? S.albedo : f3(0.f, 0.f, 0.f), h.t, h.gauss);
          } else {
            set_transmittance(b, T.query[i - flying], (float)h.w);
          }
        });
    __syncwarp();
    if (__any_sync(kFull, status != 0u)) break;
    // gather the last vertices' queries, shade the new ones
    const bool mine = (uint32_t)lane < flying + ending, fly = (uint32_t)lane < flying;
    const uint32_t p = mine ? T.path[lane] : 0u;
    int ns = 0;
    unsigned queued = 0u;
    bool alive = false;
    if (mine) gather_path(P, b, p);
    if (fly) queued = shade_path(S, E, P, b, p, ns, alive, opaque);
    // a path that ends here without a query to trace is finished at once
    if (fly && !alive && queued == 0u) gather_path(P, b, p);
    __syncwarp();
    const unsigned am = __ballot_sync(kFull, fly && alive), em = __ballot_sync(kFull, fly && !alive && queued != 0u);
    if ((am >> lane) & 1u) T.path[__popc(am & lt)] = p;
    if ((em >> lane) & 1u) T.path[__popc(am) + __popc(em & lt)] = p;
    flying = (uint32_t)__popc(am);
    ending = (uint32_t)__popc(em);
    queries = 0u;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const unsigned qm = __ballot_sync(kFull, (queued >> k) & 1u);
      if ((qm >> lane) & 1u) T.query[queries + __popc(qm & lt)] = 3u * p + k;
      queries += (uint32_t)__popc(qm);
    }
    __syncwarp();
  }
  if (status) atomicOr(&ctr->status, status);
  cooperative_groups::this_grid().sync();
  for (uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x; pix < n_pix; pix += gridDim.x * blockDim.x)
    welford_pixel(P, b, batch, pix, mean, m2, pix_count);
}

// Morton key (10 bits per axis) of each queued path's origin over the scene bounds: sorting the
// queue by it makes neighbouring warps traverse the same BVH32 region (L1 reuse).
__device__ __forceinline__ uint32_t expand10(uint32_t v) {
  v = (v * 0x00010001u) & 0xFF0000FFu;
  v = (v * 0x00000101u) & 0x0F00F00Fu;
  v = (v * 0x00000011u) & 0xC30C30C3u;
  v = (v * 0x00000005u) & 0x49249249u;
  return v;
}

__global__ void k_wf_sort_keys(uint32_t n, const uint32_t* __restrict__ q, const float4* __restrict__ ray,
                               float3 lo, float3 inv_ext, uint32_t* __restrict__ keys) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 o = ray[2u * q[i]];
  auto quant = [](float x) { return (uint32_t)fminf(fmaxf(x, 0.0f), 1023.0f); };
  const uint32_t x = quant((o.x - lo.x) * inv_ext.x), y = quant((o.y - lo.y) * inv_ext.y),
                 z = quant((o.z - lo.z) * inv_ext.z);
  keys[i] = (expand10(z) << 2) | (expand10(y) << 1) | expand10(x);
}

template <class K>
int resident_blocks(K kernel, int threads, size_t smem) {
  int b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, threads, smem) != cudaSuccess) b = 1;
  return b < 1 ? 1 : b;
}

template <class T>
void carve_buf(char*& cur, T*& out, size_t count) {
  out = reinterpret_cast<T*>(cur);
  cur += (count * sizeof(T) + 255) & ~size_t(255);
}

vp_status ensure_workspace(vp_context* ctx, size_t paths) {
  WfWorkspace& w = ctx->wf;
  if (w.cap >= paths && w.base) return VP_OK;
  free_wavefront(ctx);
  const size_t per_path = 2 * 16 + 4 * 16 + 3 * 48 + 16 + 4 * 3 + 3 * 4;
  const size_t bytes = paths * per_path + 64 * 256 + 4096;
  cudaError_t e = cudaMalloc(&w.base, bytes);
  if (e == cudaErrorMemoryAllocation) {  // give back what the context's pool keeps, and try again
    (void)cudaGetLastError();
    VP_CUDA(cudaStreamSynchronize(ctx->stream));
    VP_CUDA(cudaMemPoolTrimTo(ctx->pool, 0));
    e = cudaMalloc(&w.base, bytes);
  }
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    w.base = nullptr;
    return fail(VP_ERROR_OUT_OF_MEMORY, "wavefront workspace of " + std::to_string(bytes) + " bytes");
  }
  if (!w.host_count) {
    e = cudaMallocHost(&w.host_count, sizeof(uint32_t));
    if (e != cudaSuccess) return cuda_fail(e, "cudaMallocHost");
  }
  char* cur = static_cast<char*>(w.base);
  WfBuffers& b = w.b;
  carve_buf(cur, b.ray, 2 * paths);
  carve_buf(cur, b.st, 4 * paths);
  carve_buf(cur, b.sq, 6 * paths);
  carve_buf(cur, b.sw, 3 * paths);
  carve_buf(cur, b.L4, paths);
  carve_buf(cur, b.qa, paths);
  carve_buf(cur, b.qb, paths);
  carve_buf(cur, b.qs, 3 * paths);
  carve_buf(cur, b.sk_a, paths);
  carve_buf(cur, b.ctr, 64);
  w.cap = paths;
  const size_t tmp = radix_sort_tmp_bytes_u32(paths);
  e = cudaMalloc(&w.sort_tmp, tmp);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    free_wavefront(ctx);
    return fail(VP_ERROR_OUT_OF_MEMORY, "wavefront sort scratch");
  }
  w.sort_tmp_bytes = tmp;
  return VP_OK;
}

}  // namespace

void free_wavefront(vp_context* ctx) {
  WfWorkspace& w = ctx->wf;
  if (w.base) cudaFree(w.base);
  if (w.sort_tmp) cudaFree(w.sort_tmp);
  w.base = nullptr;
  w.sort_tmp = nullptr;
  w.sort_tmp_bytes = 0;
  w.cap = 0;
}

vp_status launch_wavefront(vp_scene* s, vp_env* e, const CameraView& cam, const ParamsView& P, vp_image* img,
                           uint32_t spp_offset, uint32_t spp_count) {
  vp_context* ctx = s->ctx;
  cudaStream_t st = ctx->stream;
  const uint32_t n_pix = P.width * P.height;
  const uint64_t paths64 = (uint64_t)n_pix * spp_count;
  if (paths64 == 0) return VP_OK;
  if (paths64 >= (1ull << 31) / 3) return fail(VP_ERROR_LIMIT, "batch too large for the wavefront engine");
  const uint32_t paths = (uint32_t)paths64;
  vp_status r;
  if ((r = ensure_workspace(ctx, paths))) return r;
  WfBuffers b = ctx->wf.b;
  const int threads = 256;
  const size_t smem = kRootStageBytes + (size_t)(threads / 32) * warp_smem_bytes(s->view.argmin_cap, kExtendHitCap);
  const size_t smem_sh = kRootStageBytes + (size_t)(threads / 32) * warp_smem_bytes(s->view.stack_cap, 32);
  if (smem > 200 * 1024) return fail(VP_ERROR_LIMIT, "BVH too deep for the shared-memory stack");
  auto ext = P.accurate ? (P.measure ? k_wf_extend<true, true> : k_wf_extend<true, false>)
                        : (P.measure ? k_wf_extend<false, true> : k_wf_extend<false, false>);
  auto shd = P.accurate ? (P.measure ? k_wf_shadow<true, true> : k_wf_shadow<true, false>)
                        : (P.measure ? k_wf_shadow<false, true> : k_wf_shadow<false, false>);
  if (smem > 48 * 1024) VP_CUDA(cudaFuncSetAttribute(ext, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  if (smem_sh > 48 * 1024)
    VP_CUDA(cudaFuncSetAttribute(shd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_sh));
  const int ext_blocks = ctx->sm_count * resident_blocks(ext, threads, smem);
  const int shd_blocks = ctx->sm_count * resident_blocks(shd, threads, smem_sh);
  const int thr_blocks = ctx->sm_count * 8;
  // The thread-per-ray stages, but for a scene without the 8-wide BVH and for the counting variants.
  const bool use8 = s->view.depth8 != 0u && !P.measure;
  const size_t smem8 = trace8_smem_bytes(s->view.depth8, kT8Threads);
  const bool mixed = s->view.one_albedo == 0;
  auto ext8 = P.accurate ? (mixed ? k_wf_extend8<true, true> : k_wf_extend8<true, false>)
                         : (mixed ? k_wf_extend8<false, true> : k_wf_extend8<false, false>);
  auto shd8 = P.accurate ? k_wf_shadow8<true> : k_wf_shadow8<false>;
  int ext8_blocks = 0, shd8_blocks = 0;
  if (use8) {
    if (smem8 > kSmem8Default)
      for (auto k : {(const void*)ext8, (const void*)shd8})
        VP_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem8));
    ext8_blocks = ctx->sm_count * resident_blocks(ext8, kT8Threads, smem8);
    shd8_blocks = ctx->sm_count * resident_blocks(shd8, kT8Threads, smem8);
  }
  // VP_MEASURE_STAGES: events around the extend and shadow launches of each iteration (a ring of 4 iterations,
  // read back at every poll, when the stream has drained)
  cudaEvent_t* ev = ctx->stage_ev;
  const bool timed = ctx->time_stages;
  if (timed && !ev[0])
    for (int i = 0; i < vp_context::kStageEvents; ++i) VP_CUDA(cudaEventCreate(&ev[i]));
  uint32_t pending = 0;  // iterations whose events are recorded but not yet read
  auto harvest = [&]() -> cudaError_t {
    for (uint32_t j = 0; j < pending; ++j) {
      float a = 0.f, c = 0.f;
      cudaError_t er = cudaEventElapsedTime(&a, ev[4 * j + 0], ev[4 * j + 1]);
      if (er == cudaSuccess) er = cudaEventElapsedTime(&c, ev[4 * j + 2], ev[4 * j + 3]);
      if (er != cudaSuccess) return er;
      ctx->stage_ms[0] += a;
      ctx->stage_ms[1] += c;
    }
    pending = 0;
    return cudaSuccess;
  };
  if (P.adaptive_threshold > 0.0f) VP_CUDA(cudaMemsetAsync(b.ctr, 0, 5 * sizeof(uint32_t), st));
  k_wf_generate<<<(paths + 255) / 256, 256, 0, st>>>(cam, P, spp_offset, spp_count, paths, b, img->mean, img->m2,
                                                     img->count, ctx->counters);
  VP_CUDA(cudaGetLastError());
  ctx->launches += 1;
  uint32_t* qcur = b.qa;
  uint32_t* qnext = b.qb;
  // Path origins' Morton order: the queue is re-sorted after every poll (the count is known on
  // the host then); compaction keeps most of the order in between.
  const vp_scene_info& si = s->info;
  const float3 blo = make_float3((float)si.bounds_min[0], (float)si.bounds_min[1], (float)si.bounds_min[2]);
  auto inv_ext1 = [](double a, double b) { return (float)(1024.0 / std::max(b - a, 1e-30)); };
  const float3 binv = make_float3(inv_ext1(si.bounds_min[0], si.bounds_max[0]),
                                  inv_ext1(si.bounds_min[1], si.bounds_max[1]),
                                  inv_ext1(si.bounds_min[2], si.bounds_max[2]));
  auto tail = P.accurate ? (P.measure ? k_wf_tail<true, true> : k_wf_tail<true, false>)
                         : (P.measure ? k_wf_tail<false, true> : k_wf_tail<false, false>);
  size_t smem_tail = smem;
  const bool tail8 = use8 && !mixed;
  const bool deep = P.max_bounces > kTailDeep;
  const uint32_t resident = (uint32_t)(ctx->sm_count * kTailBlocks * (threads / 32));
  uint32_t tail_max = deep ? 2u * resident : resident;
  if (tail8) {
    tail_max = s->overlap > kTailOverlap ? 2u * resident
               : !(P.accurate && s->overlap > kTailOverlapAccurate) ? kTailMax
               : deep ? kTailMaxAccurate : 2u * resident;
    tail = P.accurate ? k_wf_tail8<true> : k_wf_tail8<false>;
    smem_tail = smem8 + (kT8Threads / 32) * sizeof(TailWarp);
  }
  if (smem_tail > kSmem8Default)
    VP_CUDA(cudaFuncSetAttribute(tail, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_tail));
  uint32_t polled = paths;
  for (uint32_t it = 0; it < P.max_bounces; ++it) {
    // Few paths left (the count last read), or none that can be (a scatter in an albedo-0 scene ends its
    // path): the tail takes over.  The first bounce always runs as stages.
    if (it != 0u && (polled <= tail_max || s->view.albedo_all_zero)) break;
    if (it != 0u && (it & 3u) == 0u && polled >= kSortMinPaths) {  // (camera rays share one origin)
      k_wf_sort_keys<<<(polled + 255) / 256, 256, 0, st>>>(polled, qcur, b.ray, blo, binv, b.sk_a);
      vp_status r = radix_sort_pairs(b.sk_a, qcur, polled, 30, ctx->wf.sort_tmp, ctx->wf.sort_tmp_bytes, st,
                                     &ctx->launches);
      if (r) return r;
    }
    cudaEvent_t* e4 = ev + 4 * (it & 3u);
    if (timed) VP_CUDA(cudaEventRecord(e4[0], st));
    if (use8 && (!mixed || polled > kMixedExtendMin)) {
      ext8<<<ext8_blocks, kT8Threads, smem8, st>>>(s->view, b, qcur, b.ctr + 0, b.ctr + 3, ctx->counters);
    } else {
      ext<<<ext_blocks, threads, smem, st>>>(s->view, P, b, qcur, b.ctr + 0, b.ctr + 3, ctx->counters);
    }
    if (timed) VP_CUDA(cudaEventRecord(e4[1], st));
    k_wf_shade<<<thr_blocks, threads, 0, st>>>(s->view, e->view, P, b, qcur, b.ctr + 0, qnext, b.ctr + 1,
                                               ctx->counters);
    if (timed) VP_CUDA(cudaEventRecord(e4[2], st));
    if (use8 && (!mixed || polled > kMixedShadowMin))
      shd8<<<shd8_blocks, kT8Threads, smem8, st>>>(s->view, b, b.ctr + 2, b.ctr + 4, ctx->counters);
    else
      shd<<<shd_blocks, threads, smem_sh, st>>>(s->view, b, b.ctr + 2, b.ctr + 4, ctx->counters, P.measure);
    if (timed) VP_CUDA(cudaEventRecord(e4[3], st));
    k_wf_gather<<<thr_blocks, threads, 0, st>>>(P, b, qcur, b.ctr + 0);
    k_wf_advance<<<1, 1, 0, st>>>(b.ctr);
    VP_CUDA(cudaGetLastError());
    ctx->launches += 5;
    ctx->stage_launches[0] += 1;
    ctx->stage_launches[1] += 1;
    if (timed) ++pending;
    std::swap(qcur, qnext);
    if ((it & 3u) == 3u) {  // stop once no path is alive
      VP_CUDA(cudaMemcpyAsync(ctx->wf.host_count, b.ctr, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
      VP_CUDA(cudaStreamSynchronize(st));
      VP_CUDA(harvest());
      polled = *ctx->wf.host_count;
      if (polled == 0u) break;
    }
  }
  {
    const uint32_t* tcount = b.ctr + 0;
    unsigned int* twork = b.ctr + 3;
    Counters* tctr = ctx->counters;
    SceneView tS = s->view;
    EnvView tE = e->view;
    ParamsView tP = P;
    uint32_t tbatch = spp_count, tpix = n_pix;
    void* args[] = {&tS, &tE, &tP, &b, &qcur, &tcount, &twork, &tctr, &tbatch, &tpix, &img->mean, &img->m2, &img->count};
    VP_CUDA(cudaLaunchCooperativeKernel((const void*)tail, dim3(ctx->sm_count * resident_blocks(tail, threads, smem_tail)),
                                        dim3(threads), args, smem_tail, st));
  }
  ctx->launches += 1;
  if (timed && pending) {
    VP_CUDA(cudaStreamSynchronize(st));
    VP_CUDA(harvest());
  }
  return VP_OK;
}

}  // namespace vp
