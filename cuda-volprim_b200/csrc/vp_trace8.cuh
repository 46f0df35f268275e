// Thread-per-ray queries over the compressed 8-wide BVH, with the per-Gaussian work of a warp's 32
// rays pooled: the queries of the wavefront and serving engines and of vp_transmittance.
//
// What bounds it, and why this split.  The warp-cooperative query (vp_traverse.cuh) spends 32 lanes
// on one ray; its chord set-up runs with about two lanes busy.  Here a lane walks its own ray through
// the inner nodes, and what it finds is shared out over the whole warp:
//   node step   every lane with nodes left tests the 8 quantised child boxes of one node (64 B + one
//               child reference); hit inner children stay with the lane (one stack entry a level),
//               hit Gaussians go to the warp's queue 1 as (lane, node, slot);
//   chord step  when queue 1 holds 32 entries, lane e loads the e-th Gaussian's record and sets up
//               its chord against the owner's ray (shuffled over); the few that cross go to queue 2;
//   value step  when queue 2 holds 32 chords, lane e evaluates the e-th (optical depth, free flight
//               or albedo weight) and each owner collects its own by shuffles.
// So box tests, chord set-ups and erf / erfinv evaluations each run with nearly full warps, whatever
// the 32 rays do.  A warp refills its finished lanes together, after draining both queues; once there is
// nothing left to fetch, its idle lanes take over subtrees of the rays still walking.  Without that, a batch
// ended with its longest rays, whose lanes walked alone, and below some 115k rays a whole warp on each ray
// was sooner done; with it this form is the faster one at every batch in scenes of many small Gaussians (transmittance
// of 1k / 65k / 250k rays through a 100k-Gaussian cloud: 0.08 / 0.14 / 0.26 ms, 0.10 / 0.29 / 0.39 without, 0.10 /
// 0.24 / 0.63 with a warp on each ray; the 2M-Gaussian stress image 64 / 77 / 180 ms).  A warp on each ray stays
// better for short batches through small scenes (launch_transmittance, vp_render.cu), where the Gaussians are as large
// as the scene (kMaxOverlap8, vp_build.cu) and for few paths through differing albedos (vp_wavefront.cu).
//
// Results do not depend on which rays share a warp or in which order chords are met: the argmin is a
// minimum, and the sums (optical depth, albedo weights) are carried in FP64 and rounded once.
#pragma once

#include "vp_traverse.cuh"

namespace vp {

// ---- node layout: 96 B = 24 words ------------------------------------------------------------
//   words 0..2   box origin p (FP32)
//   word  3      bytes: 15 + exponent of the x / y / z quantum (biased as a float's), inner mask
//   words 4..15  child planes, a byte each: lo.x[8] lo.y[8] lo.z[8] hi.x[8] hi.y[8] hi.z[8]
//   words 16..23 child references: an inner node's index or kLeafBit | Gaussian (scene order)
// Child slot s holds the child that lies furthest towards (s&1 ? +x : -x, s&2 ? +y : -y, s&4 ? +z : -z),
// so visiting slots in ascending (s ^ sign bits of the direction) is roughly front to back.
// An unused slot has lo = 255, hi = 0 and no reference (a hit of it is dropped).  Node 0 only points to the root (slot 0).
constexpr uint32_t kNode8Words = 24;
constexpr uint32_t kMaxNodes8 = 1u << 24;   // stack entries hold (node << 8 | child mask)
constexpr uint32_t kMaxDepth8 = 40;         // deeper trees take the warp-cooperative query
// A value step runs once queue 2 holds this many chords.  Fuller steps cost fewer instructions a chord,
// earlier ones tighten the free-flight bound (and reach MAX_OPTICAL_DEPTH) sooner: 8 measured fastest or
// level with 16 on every scene tried (showcase 66.6 / 67.2 / 69.8 ms at 8 / 16 / 32; a 100k-Gaussian image
// of 361k paths 6.3 / 6.7 / 7.6 ms).
constexpr int kValueStep = 8;
constexpr int kQ1Cap = 32 + 256, kQ2Cap = 64, kQ2Words = 7;

// Words of shared memory per warp: stack, queue 1, queue 2, owner masks, a work counter of its own.
__host__ __device__ __forceinline__ uint32_t trace8_warp_words(uint32_t depth) {
  return depth * 32u + kQ1Cap + kQ2Cap * kQ2Words + 33u;
}
__host__ __device__ __forceinline__ size_t trace8_smem_bytes(uint32_t depth, int threads) {
  return (size_t)trace8_warp_words(depth) * 4u * (size_t)(threads / 32);
}

enum Query8 { kFlight8 = 0, kTau8 = 1, kScatter8 = 2, kBoth8 = 3 /* flights and transmittances by Ray8::flight */ };

// What a query reads of a scene.
struct Scene8 {
  const uint32_t* nodes;
  const float4* prims;
  const uint32_t* perm;
};
__device__ __forceinline__ Scene8 scene8_of(const SceneView& S) { return Scene8{S.nodes8, S.prims, S.perm}; }
// The scene of every ray of a launch, or (the serving engine) each ray's own, from a table in shared memory.
struct OneScene8 {
  Scene8 s;
  __device__ __forceinline__ Scene8 of(uint32_t) const { return s; }
};
struct ManyScenes8 {
  const Scene8* table;
  __device__ __forceinline__ Scene8 of(uint32_t k) const { return table[k]; }
};

struct Ray8 {
  float3 o, d;
  uint64_t key;    // kFlight8: free-flight key
  float t;         // kScatter8: scatter distance
  uint32_t scene;  // ManyScenes8: index into the table
  bool flight;     // kBoth8: a free flight, else a transmittance
  uint32_t seed;   // kTau8: the Gaussian already accounted for; kFlight8: one to start with (kNoGauss: none)
  float seed_tau;  // its optical depth (0 without one)
};
struct Hit8 {
  float t;          // kFlight8: free-flight minimum (kInf: escape)
  uint32_t gauss;   // kFlight8: its Gaussian
  double w, r, g, b;  // kTau8: w = optical depth; kScatter8: sums of weight, weight x albedo
};

__device__ __forceinline__ float byte_plane(uint32_t word, uint32_t sel) {  // 1 + q / 32768
  return __uint_as_float(__byte_perm(word, 0x3F800000u, sel));
}

// order[sign bits << 8 | child mask]: the mask's first slot in the direction's visiting order.
struct Order8 {
  alignas(16) uint8_t slot[2048];
};
constexpr Order8 make_order8() {
  Order8 t{};
  for (uint32_t k = 0; k < 2048u; ++k) {
    const uint32_t neg = k >> 8;
    uint32_t s = 0u;
    for (uint32_t b = 8u; b-- > 0u;)
      if ((k >> (b ^ neg)) & 1u) s = b ^ neg;
    t.slot[k] = (uint8_t)s;
  }
  return t;
}
static __device__ const Order8 g_order8 = make_order8();

// The table in shared memory.  All threads of the block call it, before any of its trace8 calls.
__device__ __forceinline__ const uint8_t* stage_order8() {
  __shared__ Order8 order;
  for (uint32_t k = threadIdx.x; k < sizeof(Order8) / 16u; k += blockDim.x)
    reinterpret_cast<uint4*>(order.slot)[k] = reinterpret_cast<const uint4*>(g_order8.slot)[k];
  __syncthreads();
  return order.slot;
}

// A child is met where far x kFar8 >= near.  A plane's distance t is off by at most 4 u t, u = 2^-24, beyond what the
// 1/64 quantum of its rounding outward covers: p - o, the reciprocal of the direction, their product and the final
// FMA, u each.  So 8 u between a far and a near plane; 16 u is allowed.  Without it Gaussians of some ulps of their
// distance were lost.  (An FMA in the place of the subtraction: no instruction more.)
constexpr float kFar8 = 1.0f + 16.0f / 16777216.0f;

// Two FMAs in one instruction (sm_100).
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{.reg .b64 ra, rb, rc, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}

// One warp's share of n rays, handed out through *work to `warps` warps.  source(item, ray) fills the ray of an item and returns false when the
// item needs no query (its sink is not called); sink(item, ray, hit) takes the result.  `rpw` rays are
// in flight per warp: fewer than 32 when the batch is too small to give every resident warp 32, since
// the chord and value steps use all lanes anyway.
template <bool kAcc, int kKind, class Scenes, class Source, class Sink>
__device__ __forceinline__ void trace8(const Scenes& scenes, uint32_t depth, uint32_t* smem, const uint8_t* order,
                                       uint32_t n, unsigned int* work, uint32_t warps, int rpw, uint32_t& status,
                                       Source&& source, Sink&& sink) {
  constexpr bool kMany = std::is_same_v<Scenes, ManyScenes8>;
  constexpr bool kFlights = kKind == kFlight8 || kKind == kBoth8, kTaus = kKind == kTau8 || kKind == kBoth8;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  uint32_t* stack = smem + lane;  // entry k at stack[32 k]: conflict-free whatever the lanes' depths
  uint32_t* q1 = smem + depth * 32u;
  uint32_t* q2 = q1 + kQ1Cap;
  uint32_t* own = q2 + kQ2Cap * kQ2Words;
  int q1n = 0, q2n = 0;
  Ray8 ray;
  ray.o = ray.d = f3(0.f, 0.f, 0.f);
  ray.key = 0ull;
  ray.seed = kNoGauss;
  ray.t = 0.f;
  ray.scene = 0u;
  ray.flight = kKind == kFlight8;
  // the scene of another lane's ray
  auto scene_of = [&](int ow) { return scenes.of(kMany ? __shfl_sync(kFull, ray.scene, ow) : 0u); };
  // what this lane walks: its own ray or, late in a batch, part of another lane's (owner)
  float3 no = f3(0.f, 0.f, 0.f), inv = f3(0.f, 0.f, 0.f);
  uint32_t item = 0, node = 0, mask = 0, neg = 0, walk_scene = 0;
  int sp = 0, sb = 0, owner = lane;  // its stack entries are [sb, sp)
  bool active = false, more = true;
  float t_hi = kInf;
  uint32_t arg = kNoGauss;
  double acc = 0.0, ar = 0.0, ag = 0.0, ab = 0.0;
  const unsigned used = rpw >= 32 ? kFull : ((1u << rpw) - 1u);
  const int refill = max(1, rpw / 4);

  // value step over the top k chords of queue 2
  auto values = [&](int k) {
    const int e = q2n - k + lane;
    q2n -= k;
    uint32_t id = 0;
    float v = kInf, wa = 0.f, wb = 0.f, wc = 0.f;
    const bool on = lane < k;
    if (on) id = q2[e];
    const int ow = (int)(id >> 27) & 31;
    const uint32_t gi = id & 0x07FFFFFFu;
    const Scene8 sc = scene_of(ow);
    uint64_t key = 0ull;
    float ts = 0.f;
    bool flight = kKind == kFlight8;
    if constexpr (kKind == kBoth8) flight = __shfl_sync(kFull, (int)ray.flight, ow) != 0;
    if constexpr (kFlights)
      key = ((uint64_t)__shfl_sync(kFull, (uint32_t)(ray.key >> 32), ow) << 32) |
            __shfl_sync(kFull, (uint32_t)ray.key, ow);
    if constexpr (kKind == kScatter8) ts = __shfl_sync(kFull, ray.t, ow);
    if (on) {
      Chord ch;
      ch.tc = __uint_as_float(q2[kQ2Cap + e]);
      ch.rw = __uint_as_float(q2[2 * kQ2Cap + e]);
      ch.d2 = __uint_as_float(q2[3 * kQ2Cap + e]);
      ch.h = __uint_as_float(q2[4 * kQ2Cap + e]);
      const float icf = __uint_as_float(q2[5 * kQ2Cap + e]);
      ch.d2lo = kAcc ? __uint_as_float(q2[6 * kQ2Cap + e]) : 0.0f;
      ch.t_in = fmaf(-ch.h, ch.rw, ch.tc);
      ch.t_out = fmaf(ch.h, ch.rw, ch.tc);
      if (kTaus && !flight) {
        v = chord_tau<kAcc>(ch.tc, ch.rw, ch.d2, ch.h, chord_u0(ch, 0.0f), fmaxf(ch.t_in, 0.0f), ch.t_out, icf, ch.d2lo);
      } else if (kFlights) {
        v = chord_free_flight<kAcc>(ch.tc, ch.rw, ch.d2, ch.h, chord_u0(ch, 0.0f), ch.t_in, ch.t_out, icf,
                                    free_flight_tau<kAcc>(key, __ldg(sc.perm + gi)), ch.d2lo);
      } else {
        const float u = (ts - ch.tc) / ch.rw;
        v = icf * vexp<kAcc>(-0.5f * fmaf(u, u, ch.d2));
        const float3 al = load_albedo(sc.prims, gi);
        wa = al.x, wb = al.y, wc = al.z;
      }
    }
    // each owner finds its chords: the mask of lanes holding them, left in own[] by their lowest lane
    const unsigned peers = __match_any_sync(kFull, on ? ow : 32 + lane);
    own[lane] = 0u;
    __syncwarp();
    if (on && (peers & lt) == 0u) own[ow] = peers;
    __syncwarp();
    unsigned m = own[lane];
    while (__any_sync(kFull, m != 0u)) {
      const int j = m ? __ffs(m) - 1 : lane;
      const float vj = __shfl_sync(kFull, v, j);
      if constexpr (kKind != kScatter8) {
        if (kTaus && m && !ray.flight) acc += (double)vj;
        if constexpr (kFlights) {
          const uint32_t gj = __shfl_sync(kFull, gi, j);
          if (m && ray.flight && vj < t_hi) {
            t_hi = vj;
            arg = gj;
          }
        }
      } else {
        const float x = __shfl_sync(kFull, wa, j), y = __shfl_sync(kFull, wb, j), z = __shfl_sync(kFull, wc, j);
        if (m) {
          acc += (double)vj;
          ar += (double)vj * (double)x;
          ag += (double)vj * (double)y;
          ab += (double)vj * (double)z;
        }
      }
      m &= m - 1u;
    }
    __syncwarp();
  };

  // chord step over the top k entries of queue 1
  auto chords = [&](int k) {
    const int e = q1n - k + lane;
    q1n -= k;
    const uint32_t w = lane < k ? q1[e] : 0u;
    __syncwarp();
    const int ow = (int)(w >> 27);
    const uint32_t at = w & 0x07FFFFFFu;  // node * 8 + slot
    const Scene8 sc = scene_of(ow);
    uint32_t gi = kEmptyRef;
    if (lane < k) gi = __ldg(sc.nodes + (size_t)(at >> 3) * kNode8Words + 16u + (at & 7u));
    // an unused slot's planes (lo 255, hi 0) coincide when the ray's distance rounds the whole node away
    bool hit = gi != kEmptyRef;
    gi &= ~kLeafBit;
    const float3 o = f3(__shfl_sync(kFull, ray.o.x, ow), __shfl_sync(kFull, ray.o.y, ow), __shfl_sync(kFull, ray.o.z, ow));
    const float3 d = f3(__shfl_sync(kFull, ray.d.x, ow), __shfl_sync(kFull, ray.d.y, ow), __shfl_sync(kFull, ray.d.z, ow));
    float bound = kInf;
    if constexpr (kTaus) {
      const uint32_t seed = __shfl_sync(kFull, ray.seed, ow);
      hit = hit && gi != seed;
    }
    if constexpr (kKind != kTau8) bound = __shfl_sync(kFull, kKind == kScatter8 ? ray.t : t_hi, ow);
    Chord ch;
    if (hit) {
      PrimGeo g;
      ldg256(sc.prims + 4u * gi, g.a, g.b);
      g.c = __ldg(sc.prims + 4u * gi + 2u);
      hit = chord_setup<kAcc>(g, o, d, ch);
      if constexpr (kKind == kScatter8) hit = hit && ch.t_in <= bound && bound <= ch.t_out;
      else hit = hit && ch.t_out > 0.0f && ch.t_in <= bound;
    }
    const unsigned hm = __ballot_sync(kFull, hit);
    if (hm == 0u) return;
    if (hit) {
      const int p = q2n + __popc(hm & lt);
      q2[p] = ((uint32_t)ow << 27) | gi;
      q2[kQ2Cap + p] = __float_as_uint(ch.tc);
      q2[2 * kQ2Cap + p] = __float_as_uint(ch.rw);
      q2[3 * kQ2Cap + p] = __float_as_uint(ch.d2);
      q2[4 * kQ2Cap + p] = __float_as_uint(ch.h);
      q2[5 * kQ2Cap + p] = __ldg(reinterpret_cast<const uint32_t*>(sc.prims + 4u * gi + 3u));
      if (kAcc) q2[6 * kQ2Cap + p] = __float_as_uint(ch.d2lo);
    }
    q2n += __popc(hm);
    __syncwarp();
    if (q2n >= kValueStep) values(min(q2n, 32));
  };

  while (true) {
    if (status) mask = 0u, sp = sb;  // (raised below: the lane gives its ray up)
    if constexpr (kTaus) {  // opaque: the rest of the ray's nodes cannot matter
      const bool opaque = acc >= (double)kMaxOpticalDepth;
      if (__any_sync(kFull, opaque)) {
        if (__shfl_sync(kFull, (int)opaque, owner)) mask = 0u, sp = sb;
      }
    }
    unsigned busy = __ballot_sync(kFull, mask != 0u || sp != sb);
    const int free_lanes = __popc(used & ~busy);
    if (busy == 0u || (more && free_lanes >= refill)) {
      while (q1n > 0) chords(min(q1n, 32));
      if (q2n > 0) values(q2n);
      if (active && mask == 0u && sp == sb) {
        Hit8 h;
        h.t = t_hi, h.gauss = arg, h.w = acc, h.r = ar, h.g = ag, h.b = ab;
        sink(item, ray, h);
        active = false;
      }
      if (more) {
        const unsigned want = used & __ballot_sync(kFull, !active);
        uint32_t first = 0;
        if (lane == 0) first = atomicAdd(work, (unsigned)__popc(want));
        first = __shfl_sync(kFull, first, 0);
        // (where every warp's first share covers the batch, there is nothing more to fetch)
        more = first + (uint32_t)__popc(want) < n && n > (uint32_t)rpw * warps;
        if ((want >> lane) & 1u) {
          item = first + (uint32_t)__popc(want & lt);
          if (item < n && source(item, ray)) {
            active = true;
            inv = safe_inv(ray.d);
            neg = (inv.x < 0.f ? 0x100u : 0u) | (inv.y < 0.f ? 0x200u : 0u) | (inv.z < 0.f ? 0x400u : 0u);
            no = ray.o;
            walk_scene = ray.scene;
            owner = lane;
            node = 0u;
            mask = 1u;  // slot 0 of node 0: the root
            sp = sb = 0;
            t_hi = kKind == kScatter8 ? ray.t : kInf;
            arg = kNoGauss;
            acc = ar = ag = ab = 0.0;
            if constexpr (kTaus) {
              if (!ray.flight && ray.seed != kNoGauss) acc = (double)ray.seed_tau;
            }
            if constexpr (kFlights) {
              // a path that scattered starts inside the Gaussian that scattered it: its free flight
              // bounds the traversal from the start (showcase: 63 -> 33 nodes a ray with it)
              if (ray.flight && ray.seed != kNoGauss) {
                const Scene8 sc = scenes.of(ray.scene);
                const PrimGeo g = load_geo(sc.prims, ray.seed);
                Chord ch;
                if (chord_setup<kAcc>(g, ray.o, ray.d, ch) && ch.t_out > 0.0f) {
                  const float v = chord_free_flight<kAcc>(ch.tc, ch.rw, ch.d2, ch.h, chord_u0(ch, 0.0f), ch.t_in, ch.t_out,
                                                          g.icf, free_flight_tau<kAcc>(ray.key, __ldg(sc.perm + ray.seed)),
                                                          ch.d2lo);
                  if (v < t_hi) t_hi = v, arg = ray.seed;
                }
                ray.seed = kNoGauss;  // (the traversal meets it again)
              }
            }
          }
        }
      }
      if (!__any_sync(kFull, active) && !more) break;
      continue;
    }
    if (!more && busy != kFull) {
      // No rays left to fetch: lanes without nodes take the oldest stack entry -- the largest subtree -- of
      // lanes that have more than one thing to do, and walk it for its owner.  Queue entries carry the owner,
      // so nothing else changes; the warp's last rays no longer walk alone.
      const unsigned donors = __ballot_sync(kFull, sp - sb + (mask != 0u ? 1 : 0) >= 2 && sp != sb);
      if (donors != 0u) {
        const bool give = (donors >> lane) & 1u, idle = !((busy >> lane) & 1u);
        const int rank = __popc((give ? donors : ~busy) & lt), pairs = min(__popc(donors), __popc(~busy));
        if (give && rank < pairs) own[rank] = (uint32_t)lane;
        __syncwarp();
        const bool take = idle && rank < pairs;
        const int from = take ? (int)own[rank] : lane;
        const int at = __shfl_sync(kFull, sb, from);
        const float ox = __shfl_sync(kFull, no.x, from), oy = __shfl_sync(kFull, no.y, from), oz = __shfl_sync(kFull, no.z, from);
        const float ix = __shfl_sync(kFull, inv.x, from), iy = __shfl_sync(kFull, inv.y, from), iz = __shfl_sync(kFull, inv.z, from);
        const uint32_t ng = __shfl_sync(kFull, neg, from);
        const int ow = __shfl_sync(kFull, owner, from);
        const uint32_t ws = kMany ? __shfl_sync(kFull, walk_scene, from) : 0u;
        if (take) {
          const uint32_t e = smem[32 * at + from];
          node = e >> 8;
          mask = e & 0xFFu;
          no = f3(ox, oy, oz);
          inv = f3(ix, iy, iz);
          neg = ng;
          owner = ow;
          walk_scene = ws;
          sp = sb = 0;
        }
        if (give && rank < pairs) ++sb;
        __syncwarp();
      }
    }
    // node step
    uint32_t leaf = 0u;
    const uint32_t* nodes = scenes.of(walk_scene).nodes;
    const float far_t = kFlights ? __shfl_sync(kFull, t_hi, owner) : 0.f;
    const float at_t = kKind == kScatter8 ? __shfl_sync(kFull, ray.t, owner) : 0.f;
    if (mask != 0u || sp != sb) {
      if (mask == 0u) {
        const uint32_t e = stack[32 * --sp];
        node = e >> 8;
        mask = e & 0xFFu;
      }
      const uint32_t slot = order[neg | mask];
      mask &= ~(1u << slot);
      const uint32_t cur = __ldg(nodes + (size_t)node * kNode8Words + 16u + slot);
      if (mask != 0u) {
        if ((uint32_t)sp >= depth) {  // cannot happen for a tree of the recorded depth
          status |= kStatusStackOverflow;
        } else {
          stack[32 * sp++] = (node << 8) | mask;
        }
      }
      const float4* p4 = reinterpret_cast<const float4*>(nodes + (size_t)cur * kNode8Words);
      float4 h, wa, wb, wc;
      ldg256(p4, h, wa);
      ldg256(p4 + 2, wb, wc);
      auto bits = [](float4 v) {
        return make_uint4(__float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w));
      };
      const uint4 a = bits(wa), bq = bits(wb), c = bits(wc);
      const uint32_t ew = __float_as_uint(h.w);
      const float ax = __uint_as_float((ew & 0xFFu) << 23) * inv.x;
      const float ay = __uint_as_float((ew & 0xFF00u) << 15) * inv.y;
      const float az = __uint_as_float((ew & 0xFF0000u) << 7) * inv.z;
      const float bx = fmaf(h.x - no.x, inv.x, -ax), by = fmaf(h.y - no.y, inv.y, -ay),
                  bz = fmaf(h.z - no.z, inv.z, -az);
      const bool nx = inv.x < 0.f, ny = inv.y < 0.f, nz = inv.z < 0.f;
      // near / far planes by the direction's signs: (lo.x, hi.x) = (a.xy, bq.zw), (lo.y, hi.y) = (a.zw, c.xy),
      // (lo.z, hi.z) = (bq.xy, c.zw)
      const uint32_t nxw[2] = {nx ? bq.z : a.x, nx ? bq.w : a.y}, fxw[2] = {nx ? a.x : bq.z, nx ? a.y : bq.w};
      const uint32_t nyw[2] = {ny ? c.x : a.z, ny ? c.y : a.w}, fyw[2] = {ny ? a.z : c.x, ny ? a.w : c.y};
      const uint32_t nzw[2] = {nz ? c.z : bq.x, nz ? c.w : bq.y}, fzw[2] = {nz ? bq.x : c.z, nz ? bq.y : c.w};
      // child j is missed when far - near is negative: the signs are shifted into a mask, child 0's last
      uint32_t miss = 0u;
      const float2 a2x = make_float2(ax, ax), a2y = make_float2(ay, ay), a2z = make_float2(az, az);
      const float2 b2x = make_float2(bx, bx), b2y = make_float2(by, by), b2z = make_float2(bz, bz);
#pragma unroll
      for (int j = 6; j >= 0; j -= 2) {  // two children at a time: packed FMAs
        const uint32_t s0 = 0x7604u | ((uint32_t)(j & 3) << 4), s1 = 0x7604u | ((uint32_t)((j + 1) & 3) << 4);
        const int w = j >> 2;
        auto plane2 = [&](uint32_t word, float2 A, float2 B) {
          return fma2(make_float2(byte_plane(word, s0), byte_plane(word, s1)), A, B);
        };
        const float2 nx2 = plane2(nxw[w], a2x, b2x), ny2 = plane2(nyw[w], a2y, b2y), nz2 = plane2(nzw[w], a2z, b2z);
        const float2 fx2 = plane2(fxw[w], a2x, b2x), fy2 = plane2(fyw[w], a2y, b2y);
        float2 fz2 = plane2(fzw[w], a2z, b2z);
        const float t0 = at_t;  // 0 but for kScatter8
        if constexpr (kKind != kTau8) {
          const float t1 = kKind == kScatter8 ? at_t : far_t;
          fz2 = make_float2(fminf(fz2.x, t1), fminf(fz2.y, t1));
        }  // a transmittance query has no far end
        const float d1 = fmaf(fmin3f(fx2.y, fy2.y, fz2.y), kFar8, -fmax3f(nx2.y, ny2.y, fmaxf(nz2.y, t0)));
        const float d0 = fmaf(fmin3f(fx2.x, fy2.x, fz2.x), kFar8, -fmax3f(nx2.x, ny2.x, fmaxf(nz2.x, t0)));
        miss = __funnelshift_l(__float_as_uint(d1), miss, 1);
        miss = __funnelshift_l(__float_as_uint(d0), miss, 1);
      }
      const uint32_t hits = ~miss & 0xFFu, inner = ew >> 24;
      node = cur;
      mask = hits & inner;
      leaf = hits & ~inner;
    }
    // hit Gaussians to queue 1: a vote per round, or (faster for transmittance, whose rays meet more of them;
    // 33.3 / 34.9 ms of the showcase, but 19.9 / 19.2 for the argmin) one shared-memory atomic per lane
    if constexpr (kTaus) {
      if (lane == 0) own[0] = (uint32_t)q1n;
      __syncwarp();
      if (leaf != 0u) {
        uint32_t at = atomicAdd(own, (uint32_t)__popc(leaf));
        do {
          q1[at++] = ((uint32_t)owner << 27) | (node << 3) | ((uint32_t)__ffs(leaf) - 1u);
          leaf &= leaf - 1u;
        } while (leaf != 0u);
      }
      __syncwarp();
      q1n = (int)own[0];
    } else {
      unsigned bal;
      while ((bal = __ballot_sync(kFull, leaf != 0u)) != 0u) {
        if (leaf != 0u) {
          const uint32_t b = (uint32_t)__ffs(leaf) - 1u;
          leaf &= leaf - 1u;
          q1[q1n + __popc(bal & lt)] = ((uint32_t)owner << 27) | (node << 3) | b;
        }
        q1n += __popc(bal);
      }
    }
    __syncwarp();
    while (q1n >= 32) chords(32);
  }
}

// Dynamic shared memory above which a kernel has to ask for it: 48 KB less its static part (the order table).
constexpr size_t kSmem8Default = 48 * 1024 - sizeof(Order8) - 1024;

// Threads of a block of the stages, and the resident blocks per SM of their register budget: 3 (80 registers).
// 4 (64 registers) spills and leaves less of the SM's memory to L1, 2 hides less latency: the showcase batch
// took 93 ms at 4 against 86 at 3, and 83 ms at 2 against 70 at 3.
constexpr int kT8Blocks = 3;
constexpr int kT8Threads = 256;

__device__ __forceinline__ uint32_t grid_warps() { return gridDim.x * (blockDim.x / 32u); }
// Rays in flight per warp: 32, or an even share of a batch too small for that.
__device__ __forceinline__ int rays_per_warp(uint32_t n, uint32_t warps) {
  return (int)min(32u, max(1u, (n + warps - 1u) / warps));
}

// The extend stage of one path queue: free flights and then, where a scene's Gaussians differ in albedo
// (kMixed), the albedo at the scatter points -- the sigma_t * pdf-weighted mean over the chords containing the
// scatter distance (evaluate_albedo over the rebuilt active set, sampling.cuh:257-283, 422-458).  With kMixed
// a warp takes a share of the queue at a time through both.  load(item, ray) and store(item, ray, hit) are
// the flights' source and sink; at(item, ray) fills a scattered path's ray and distance (false: nothing to
// look up) and albedo(item, ray, rgb) takes the result.
constexpr uint32_t kMixedShare = 256;
template <bool kAcc, bool kMixed, class Scenes, class Load, class Store, class At, class Albedo>
__device__ __forceinline__ void extend8(const Scenes& scenes, uint32_t depth, uint32_t* smem, uint32_t n,
                                        unsigned int* work, uint32_t& status, Load&& load, Store&& store, At&& at,
                                        Albedo&& albedo) {
  const uint8_t* order = stage_order8();
  const uint32_t warps = grid_warps();
  if constexpr (!kMixed) {
    trace8<kAcc, kFlight8>(scenes, depth, smem, order, n, work, warps, rays_per_warp(n, warps), status, load, store);
  } else {
    const int lane = threadIdx.x & 31;
    unsigned int* next = smem + trace8_warp_words(depth) - 1u;
    const uint32_t share = min(kMixedShare, max(1u, (n + warps - 1u) / warps));
    while (!__any_sync(kFull, status != 0u)) {
      uint32_t first = 0;
      if (lane == 0) first = atomicAdd(work, share);
      first = __shfl_sync(kFull, first, 0);
      if (first >= n) break;
      const uint32_t m = min(share, n - first);
      const int rpw = (int)min(32u, m);
      if (lane == 0) *next = 0u;
      __syncwarp();
      trace8<kAcc, kFlight8>(
          scenes, depth, smem, order, m, next, 1u, rpw, status,
          [&](uint32_t i, Ray8& ray) { return load(first + i, ray); },
          [&](uint32_t i, const Ray8& ray, const Hit8& h) { store(first + i, ray, h); });
      __syncwarp();
      if (lane == 0) *next = 0u;
      __syncwarp();
      trace8<kAcc, kScatter8>(
          scenes, depth, smem, order, m, next, 1u, rpw, status,
          [&](uint32_t i, Ray8& ray) { return at(first + i, ray); },
          [&](uint32_t i, const Ray8& ray, const Hit8& h) { albedo(first + i, ray, mean_albedo(h.w, h.r, h.g, h.b)); });
      __syncwarp();
    }
  }
}

}  // namespace vp
