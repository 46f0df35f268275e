// Absorption-plus-emission image and its hand-written adjoint (the differentiation form; the
// reference renderer has no emission and no gradients).
//
// Image model.  Along a camera ray x(t) = o + t d, Gaussian i contributes the closed-form optical
// depth tau_i of its 3-sigma chord over [0, inf) -- the same truncated-chord sum as the
// transmittance query (Primitive::optical_depth, primitive.h:249-318) -- and emits RGB e_i per
// unit optical depth.  With S = sum_i tau_i, C = sum_i tau_i e_i and T = exp(-S):
//
//     L = (1 - T) C / S + T env(d)        (L = env(d) when S = 0)
//
// which is the exact emission-absorption integral int T(t) sigma(t) c(t) dt + T env when the
// emission-to-extinction ratio c(t) along the ray equals its tau-weighted mean C / S (exact for a
// single Gaussian, for disjoint chords of equal colour, and in the optically thin limit, where
// L -> sum_i tau_i e_i).  It depends on the Gaussians only through the order-independent sums S
// and C, so a ray's Gaussians are visited in any order and no hit list is sorted or stored.
// Limitation: no occlusion between Gaussians -- a Gaussian behind an opaque one still colours the
// pixel with its tau-weighted share; only the background term is attenuated.
//
// Adjoint.  For one ray with upstream gradient G = dLoss/dL (RGB):
//     dL/dS = C (T - a) / S - T env,  a = (1 - T) / S,      dL/dC = a
//     g_tau_i = G . (dL/dS + a e_i),   dLoss/de_i = G a tau_i
// and tau_i is differentiated in closed form through the whitening p = W (o - mu), w = W d,
// W = diag(1/s) R(q)^T (see tau_grad below).  The backward kernel meets each ray's Gaussians twice --
// once for S and C, once to scatter per-Gaussian gradients -- and stores no per-ray hits: its first
// traversal lists the Gaussians of a packet of rays (below), which the second pass goes through.
// Per Gaussian it accumulates 16 floats (float4 atomics, internal order): dLoss/dW (9),
// sum g_tau dtau/dp (3, for the mean), sum g_tau tau (1, for density and the scale
// normaliser), dLoss/de (3); a finishing kernel maps them to mean / scale / quaternion /
// density / emission gradients in the caller's order.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "vp_internal.h"
#include "vp_traverse.cuh"

namespace vp {
namespace {

// Packets.  A warp takes the samples of a small tile of pixels -- up to 32 camera rays that cross nearly the
// same Gaussians -- and walks the BVH32 once for all of them: at an inner node lane c tests child c's box
// against the packet's frustum, at a leaf lane j tests the j-th Gaussian's, and each candidate is then met
// by all 32 rays at once (its record one broadcast load, every lane setting up its own ray's chord).  One
// ray a warp instead leaves about two lanes busy in the chord work, and the adjoint issues its 64 bytes of
// atomics per (ray, Gaussian) where a packet reduces its rays' gradients first; that form stays for images of
// few rays (few_rays).
//
// Tile of the packet: k = min(spp, 32) samples of 2^floor(log2(32 / k)) pixels, near square.
struct Tiling {
  uint32_t k, tw, th, tiles_x, tiles;
};

// A block of kGroup warps shares a packet: the critical path is the tile whose rays cross the densest part
// (some thousand Gaussians one after the other), so the tree's first levels are expanded into a list of
// subtrees that the block's warps take one at a time, each with all 32 rays.
constexpr uint32_t kFrontier = 96;  // list capacity; expansion stops when another node's 32 children may not fit
constexpr uint32_t kShares = 48;    // subtrees that are enough to share

// The packet's bounds, in shared memory (read by every lane at every step): the four side planes of its
// frustum (n, w): inside where n . x + w >= 0, with w already widened by the tolerance; its middle ray and
// how far the others are from it: |o - oc| <= r0, |d - dc| <= r1.
struct PacketBounds {
  float4 plane[4];
  float4 oc;  // origin, r0
  float4 dc;  // direction, r1
};

__device__ __forceinline__ float3 cross3(float3 a, float3 b) {
  return f3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, o));
  return v;
}

// extent: the largest |coordinate| of the scene's boxes.  The side planes go through the pixel coordinates
// of the outermost samples, moved out by 0.02 pixels; w also holds what FP32 rounding may move a ray out of its plane.
// With u = 2^-24 and D the distance to the scene's far side: the corner's and the rays' directions are off by 3 u
// each and n by 3 u (divided by the sine of the angle between its factors), all of which tilt about the eye and so weigh
// D, and n . x + w is off by 4 u (extent + |eye|) before it cancels; 2e-6 is 33 u.  From far away through a
// narrow lens that is more than the 0.02 pixels: with a term in the extent alone, views from 1e5 times a Gaussian's
// size lost some at the tiles' edges.
__device__ __forceinline__ void packet_bounds(const CameraView& C, float extent, bool active, float x, float y, float3 o,
                                              float3 d, PacketBounds* B) {
  const int lane = threadIdx.x & 31;
  const float x0 = -warp_max(active ? -x : -kInf) - 0.02f, x1 = warp_max(active ? x : -kInf) + 0.02f;
  const float y0 = -warp_max(active ? -y : -kInf) - 0.02f, y1 = warp_max(active ? y : -kInf) + 0.02f;
  float3 oc, dc;
  camera_ray_at(C, 0.5f * (x0 + x1), 0.5f * (y0 + y1), oc, dc);
  const float3 eo = sub(o, oc), ed = sub(d, dc);
  const float r0 = warp_max(active ? sqrtf(dot3(eo, eo)) : 0.f), r1 = warp_max(active ? sqrtf(dot3(ed, ed)) : 0.f);
  if (lane < 4) {
    const bool vertical = lane < 2;                     // planes of constant x, else of constant y
    const float px = (lane == 1) ? x1 : x0, py = (lane == 3) ? y1 : y0;
    const float3 corner = camera_offset(C, px, py);
    const float3 along = vertical ? C.dv : C.du;
    float3 inward = vertical ? C.du : C.dv;
    if (lane & 1) inward = mul(inward, -1.0f);
    const float3 axis = C.ortho ? C.view_dir : corner;
    float3 n = cross3(axis, along);
    const float inv = rsqrtf(fmaxf(dot3(n, n), 1e-37f));
    const float skew = sqrtf(dot3(axis, axis)) * sqrtf(dot3(along, along)) * inv;  // 1 / sin
    n = mul(n, inv);
    if (dot3(n, inward) < 0.f) n = mul(n, -1.0f);
    const float3 at = C.ortho ? add(C.eye, corner) : C.eye;
    const float w = -dot3(n, at);
    const float reach = sqrtf(dot3(at, at)) + 1.7321f * extent;
    const float tol = 2e-6f * reach * fmaxf(skew, 1.0f);
    B->plane[lane] = make_float4(n.x, n.y, n.z, w + tol);
  }
  if (lane == 4) B->oc = make_float4(oc.x, oc.y, oc.z, r0 * 1.001f + 1e-6f * extent);
  if (lane == 5) B->dc = make_float4(dc.x, dc.y, dc.z, r1 * 1.001f + 1e-6f);
  __syncwarp();
}

__device__ __forceinline__ bool in_frustum(const PacketBounds* B, float4 lo, float4 hi) {
  bool in = true;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float4 n = B->plane[k];
    const float s = fmaxf(n.x * lo.x, n.x * hi.x) + fmaxf(n.y * lo.y, n.y * hi.y) + fmaxf(n.z * lo.z, n.z * hi.z) + n.w;
    in = in && !(s < 0.f);
  }
  return in;
}

// Whether some ray of the packet can meet the Gaussian's 3-sigma ellipsoid.  At such a ray's point x(t), t at
// most the distance to the far side of the Gaussian's box, the middle ray is within r0 + t r1, so its
// whitened distance from the centre is at most 3 + |W| (r0 + t r1); |W| is bounded by the Frobenius norm.
__device__ __forceinline__ bool near_packet(const PacketBounds* B, const PrimGeo& g, float4 lo, float4 hi) {
  const float4 oc = B->oc, dc = B->dc;
  const float3 d = f3(dc.x, dc.y, dc.z), v = sub(f3(oc.x, oc.y, oc.z), f3(g.a.x, g.a.y, g.a.z));
  const float ex = hi.x - lo.x, ey = hi.y - lo.y, ez = hi.z - lo.z;
  const float t = sqrtf(dot3(v, v)) + oc.w + 0.5f * sqrtf(fmaf(ex, ex, fmaf(ey, ey, ez * ez)));
  const float3 w = whiten(g, d);
  const float a2 = dot3(w, w);
  const float tc = -dot3(whiten(g, v), w) * __frcp_rn(a2);
  const float3 p = whiten(g, fma3(tc, d, v));
  const float w2 = g.a.w * g.a.w + g.b.x * g.b.x + g.b.y * g.b.y + g.b.z * g.b.z + g.b.w * g.b.w + g.c.x * g.c.x +
                   g.c.y * g.c.y + g.c.z * g.c.z + g.c.w * g.c.w;
  const float wn = sqrtf(w2);
  // 1e-6 |W| t covers the FP32 rounding of the middle ray's own closest approach
  const float reach = 3.001f + wn * (oc.w + t * dc.w + 2e-6f * t);
  return !(dot3(p, p) > reach * reach);
}

// f(pi, g, ch, hit) for every Gaussian under the sp references on the stack that some active ray's chord
// crosses over [0, inf); `hit` and `ch` are the lane's own, all lanes call it.
template <bool kAcc, class F>
__device__ __forceinline__ void packet_visit(const SceneView& S, uint32_t* stack, const PacketBounds* B, float3 o, float3 d,
                                             bool active, uint32_t& status, int sp, F&& f) {
  const int lane = threadIdx.x & 31;
  const unsigned lt_mask = (1u << lane) - 1u;
  uint32_t ref = 0u;
  bool have = false;
  while (true) {
    if (!have) {
      if (sp == 0) break;
      ref = stack[--sp];
      __syncwarp();
    }
    have = false;
    if (ref_is_leaf(ref)) {
      // leaves next on the stack join this step while their Gaussians fit in the 32 lanes
      int total = (int)wide_leaf_count(ref);
      uint32_t pi = wide_leaf_first(ref) + (uint32_t)lane;
      while (VP_LEAF_PACK && sp > 0) {
        const uint32_t r2 = stack[sp - 1];
        if (!ref_is_leaf(r2)) break;
        const int c2 = (int)wide_leaf_count(r2);
        if (total + c2 > 32) break;
        --sp;
        if (lane >= total && lane < total + c2) pi = wide_leaf_first(r2) + (uint32_t)(lane - total);
        total += c2;
      }
      __syncwarp();
      bool candidate = false;
      if (lane < total) {
        const float4 lo = __ldg(S.pbox + 2u * pi), hi = __ldg(S.pbox + 2u * pi + 1u);
        if (in_frustum(B, lo, hi)) candidate = near_packet(B, load_geo(S.prims, pi), lo, hi);
      }
      unsigned cm = __ballot_sync(kFull, candidate);
      while (cm != 0u) {
        const int j = __ffs(cm) - 1;
        cm &= cm - 1u;
        const uint32_t gi = __shfl_sync(kFull, pi, j);
        const PrimGeo g = load_geo(S.prims, gi);
        Chord ch;
        const bool hit = active && chord_setup<kAcc>(g, o, d, ch) && ch.t_out > 0.0f;
        if (__any_sync(kFull, hit)) f(gi, g, ch, hit);
      }
    } else {
      const float4* node = S.wide + (size_t)ref * 64u;
      const float4 lo = __ldg(node + lane);
      const float4 hi = __ldg(node + 32 + lane);
      const uint32_t cref = __float_as_uint(lo.w);
      const bool hit = (cref != kEmptyRef) && in_frustum(B, lo, hi);
      const unsigned m = __ballot_sync(kFull, hit);
      const int nh = __popc(m);
      if (nh > 0) {
        if ((uint32_t)(sp + nh) > S.stack_cap + 1u) {  // cannot happen for a BVH of the recorded depth
          status |= kStatusStackOverflow;
          break;
        }
        const int first = __ffs(m) - 1;
        if (hit && lane != first) stack[sp + __popc(m & lt_mask) - 1] = cref;
        sp += nh - 1;
        ref = __shfl_sync(kFull, cref, first);
        have = true;
      }
    }
    __syncwarp();
  }
  __syncwarp();
}

// tau of one chord over [max(t_in, 0), t_out] (0 for a segment below RAY_SEGMENT_MIN_LENGTH).
template <bool kAcc>
__device__ __forceinline__ float chord_tau0(const Chord& ch, float icf) {
  return chord_tau<kAcc>(ch.tc, ch.rw, ch.d2, ch.h, chord_u0(ch, 0.0f), fmaxf(ch.t_in, 0.0f), ch.t_out, icf,
                         ch.d2lo);
}

// This lane's ray of a packet: sample s of its pixel (the renderer's jittered camera ray,
// raygen.cuh:82-99).  A lane without one takes part with any ray.
struct PacketRay {
  float x, y;
  float3 o, d;
};
__device__ __forceinline__ PacketRay packet_ray(const CameraView& C, const ParamsView& P, uint32_t px, uint32_t py,
                                                uint32_t s) {
  PacketRay r;
  Pcg32 rng = pcg_init(P.seed, seq_hash(((uint64_t)py * P.width + px) * (uint64_t)P.spp_total + s));
  camera_jitter(P, px, py, rng, r.x, r.y);
  camera_ray_at(C, r.x, r.y, r.o, r.d);
  return r;
}
struct PacketLane {
  uint32_t px, py, s;  // pixel, sample of the first pass
  bool on;             // has a pixel of the image
};
__device__ __forceinline__ PacketLane packet_lane(const Tiling& T, const ParamsView& P, uint32_t tile) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t p = lane / T.k;
  PacketLane l;
  l.s = lane - p * T.k;
  const uint32_t ty = tile / T.tiles_x, tx = tile - ty * T.tiles_x;
  l.px = tx * T.tw + p % T.tw;
  l.py = ty * T.th + p / T.tw;
  l.on = p < T.tw * T.th && l.px < P.width && l.py < P.height;
  return l;
}

struct RaySums {
  float S, r, g, b;  // sum tau, sum tau * e (RGB)
};

// Gaussians a warp met in the packet's first traversal, for the adjoint's second pass (n beyond the
// capacity: not all, and it traverses its subtrees again).
constexpr uint32_t kListCap = 512;

// Shared memory of a block: the packet, its frontier and the warps' partial sums.
template <int kGroup>
struct PacketShared {
  PacketBounds bounds;
  uint32_t tile, n_front, next, pad;
  uint32_t front[kFrontier];
  uint8_t owner[kFrontier];  // the warp that took each
  double sums[kGroup][4][32];
};
// Words after PacketShared, per warp: stack, Gaussian list (adjoint).
__host__ __device__ __forceinline__ uint32_t packet_words(uint32_t stack_cap, bool list) {
  return ((stack_cap + 4u) & ~3u) + (list ? kListCap : 0u);
}
template <int kGroup>
constexpr size_t packet_smem(uint32_t stack_cap, bool list) {
  return sizeof(PacketShared<kGroup>) + 4u * (size_t)kGroup * packet_words(stack_cap, list);
}

// The block's first warp lists the subtrees below the tree's first levels that the packet meets.
template <int kGroup>
__device__ __forceinline__ void expand_frontier(const SceneView& S, PacketShared<kGroup>& sh) {
  const int lane = threadIdx.x & 31;
  if (lane == 0) sh.front[0] = S.wide_root;
  __syncwarp();
  uint32_t n = 1, at = 0;
  while (at < n && n + 31u <= kFrontier) {
    const uint32_t ref = sh.front[at];
    __syncwarp();
    if (ref_is_leaf(ref)) {
      ++at;
      continue;
    }
    const float4* node = S.wide + (size_t)ref * 64u;
    const float4 lo = __ldg(node + lane);
    const float4 hi = __ldg(node + 32 + lane);
    const uint32_t cref = __float_as_uint(lo.w);
    const bool hit = cref != kEmptyRef && in_frustum(&sh.bounds, lo, hi);
    const unsigned m = __ballot_sync(kFull, hit);
    // its children take its place and the list's end
    if (m == 0u) {
      if (lane == 0) sh.front[at] = sh.front[n - 1u];
      --n;
    } else {
      const int rank = __popc(m & ((1u << lane) - 1u));
      if (hit) sh.front[rank == 0 ? at : n + (uint32_t)rank - 1u] = cref;
      if (n > 1u) ++at;  // on to its siblings
      n += (uint32_t)__popc(m) - 1u;
    }
    __syncwarp();
    if (n >= kShares) break;
  }
  if (lane == 0) {
    sh.n_front = n;
    sh.next = 0u;
  }
  for (uint32_t i = lane; i < n; i += 32u) sh.owner[i] = 0xFFu;
}

// Sums of this lane's ray over the packet's Gaussians, by the whole block: on every warp.  They run over up
// to thousands of Gaussians one after the other, so they are carried in FP64, eight FP32 terms at a time.  The eight
// never span two subtrees: which warp takes which is a matter of timing, and an image is to be the same each time.
template <bool kAcc, bool kList, int kGroup>
__device__ __forceinline__ RaySums packet_sums(const SceneView& S, const float4* __restrict__ emis, uint32_t* stack,
                                               PacketShared<kGroup>& sh, float3 o, float3 d, bool active, uint32_t& status,
                                               unsigned long long& crossings, uint32_t* list, uint32_t& n) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double s = 0.0, r = 0.0, g = 0.0, b = 0.0;
  float fs = 0.f, fr = 0.f, fg = 0.f, fb = 0.f;  // the last few terms
  unsigned int nc = 0, met = 0;
  auto flush = [&]() {
    s += (double)fs, r += (double)fr, g += (double)fg, b += (double)fb;
    fs = fr = fg = fb = 0.f;
  };
  n = 0;
  if (warp == 0) expand_frontier(S, sh);
  __syncthreads();
  const uint32_t n_front = sh.n_front;
  while (true) {
    uint32_t i = 0;
    if (lane == 0) i = atomicAdd(&sh.next, 1u);
    i = __shfl_sync(kFull, i, 0);
    if (i >= n_front) break;
    flush();
    met = 0u;
    if (lane == 0) {
      stack[0] = sh.front[i];
      if (kList) sh.owner[i] = (uint8_t)warp;
    }
    __syncwarp();
    packet_visit<kAcc>(S, stack, &sh.bounds, o, d, active, status, 1,
                       [&](uint32_t gi, const PrimGeo& geo, const Chord& ch, bool hit) {
      if (kList) {
        if (n < kListCap && lane == 0) list[n] = gi;
        ++n;
      }
      if (hit) {
        const float tau = chord_tau0<kAcc>(ch, geo.icf);
        const float4 e = __ldg(emis + gi);
        fs += tau;
        fr = fmaf(tau, e.x, fr);
        fg = fmaf(tau, e.y, fg);
        fb = fmaf(tau, e.z, fb);
        ++nc;
      }
      if ((++met & 7u) == 0u) flush();
    });
  }
  flush();
  crossings += nc;
  sh.sums[warp][0][lane] = s, sh.sums[warp][1][lane] = r, sh.sums[warp][2][lane] = g, sh.sums[warp][3][lane] = b;
  __syncthreads();
  s = r = g = b = 0.0;
#pragma unroll
  for (int w = 0; w < kGroup; ++w)
    s += sh.sums[w][0][lane], r += sh.sums[w][1][lane], g += sh.sums[w][2][lane], b += sh.sums[w][3][lane];
  return RaySums{(float)s, (float)r, (float)g, (float)b};
}

// (1 - T) / S and (T - (1 - T) / S) / S for S >= 0, with their series below 1e-3.
__device__ __forceinline__ void opacity_terms(float S, float& T, float& a, float& q) {
  T = expf(-S);
  if (S < 1e-3f) {
    a = 1.0f - S * (0.5f - S * (1.0f / 6.0f));
    q = -0.5f + S * (1.0f / 3.0f - S * 0.125f);
  } else {
    a = -expm1f(-S) / S;
    q = (T - a) / S;
  }
}

__device__ __forceinline__ float3 ray_radiance(const RaySums& rs, float3 env) {
  float T, a, q;
  opacity_terms(rs.S, T, a, q);
  return f3(fmaf(a, rs.r, T * env.x), fmaf(a, rs.g, T * env.y), fmaf(a, rs.b, T * env.z));
}

// Resident warps per SM the FP32 kernels' register budgets are sized for (16 for the ACCURATE ones).  On the
// 100k-Gaussian cloud: forward 256x256 4.1 / 3.5 ms at 24 / 32; adjoint of two 160x120 views 8.4 / 8.1 ms at
// 20 / 24.
constexpr int kFwdWarps = 32, kBwdWarps = 24;

template <bool kAcc, int kGroup>
__global__ void __launch_bounds__(32 * kGroup, (kAcc ? 16 : kFwdWarps) / kGroup) k_emis_forward(SceneView S, EnvView E, CameraView C, ParamsView P,
                                                      Tiling T, float extent, const float4* __restrict__ emis,
                                                      float4* __restrict__ out, unsigned int* work, Counters* ctr) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto& sh = *reinterpret_cast<PacketShared<kGroup>*>(vp_dyn_smem);
  uint32_t* stack = reinterpret_cast<uint32_t*>(vp_dyn_smem + sizeof(sh)) + warp * packet_words(S.stack_cap, false);
  uint32_t status = 0, n_list;
  unsigned long long crossings = 0;
  while (true) {
    if (threadIdx.x == 0) sh.tile = atomicAdd(work, 1u);
    __syncthreads();
    const uint32_t tile = sh.tile;
    if (tile >= T.tiles) break;
    const PacketLane l = packet_lane(T, P, tile);
    float3 sum = f3(0.f, 0.f, 0.f);
    for (uint32_t s0 = 0; s0 < P.spp_total; s0 += T.k) {
      const uint32_t k = min(T.k, P.spp_total - s0);  // samples of this pass
      const bool active = l.on && l.s < k;
      const PacketRay r = packet_ray(C, P, l.px, l.py, s0 + l.s);
      if (warp == 0) packet_bounds(C, extent, active, r.x, r.y, r.o, r.d, &sh.bounds);
      const RaySums rs = packet_sums<kAcc, false, kGroup>(S, emis, stack, sh, r.o, r.d, active, status, crossings, nullptr, n_list);
      const float3 L = ray_radiance(rs, env_lookup(E, r.d));
      // the pixel's samples in order
      const int base = lane - (int)l.s;
      for (uint32_t j = 0; j < k; ++j)
        sum = add(sum, f3(__shfl_sync(kFull, L.x, (base + (int)j) & 31), __shfl_sync(kFull, L.y, (base + (int)j) & 31),
                          __shfl_sync(kFull, L.z, (base + (int)j) & 31)));
    }
    const float inv = 1.0f / (float)P.spp_total;
    if (warp == 0 && l.on && l.s == 0u)
      out[(size_t)l.py * P.width + l.px] = make_float4(sum.x * inv, sum.y * inv, sum.z * inv, 1.0f);
    if (__syncthreads_or(status != 0u)) break;
  }
  if (status) atomicOr(&ctr->status, status);
  if (P.measure) atomicAdd(&ctr->crossings, crossings);
}

// ---- a warp on each ray (images of few rays) ----
// The Gaussians of one ray by the warp: f(index, record, chord) on the lane that set the chord up.
template <bool kAcc, class F>
__device__ void warp_visit(const SceneView& S, uint32_t* stack, float3 o, float3 d, uint32_t& status, F&& f) {
  const int lane = threadIdx.x & 31;
  const unsigned lt_mask = (1u << lane) - 1u;
  const RayBox rb = ray_box(o, d);
  int sp = 0;
  uint32_t ref = S.wide_root;
  bool have = true;
  while (true) {
    if (!have) {
      if (sp == 0) break;
      ref = stack[--sp];
      __syncwarp();
    }
    have = false;
    if (ref_is_leaf(ref)) {
      // leaves next on the stack join this step while their Gaussians fit in the 32 lanes
      int total = (int)wide_leaf_count(ref);
      uint32_t pi = wide_leaf_first(ref) + (uint32_t)lane;
      while (sp > 0) {
        const uint32_t r2 = stack[sp - 1];
        if (!ref_is_leaf(r2)) break;
        const int c2 = (int)wide_leaf_count(r2);
        if (total + c2 > 32) break;
        --sp;
        if (lane >= total && lane < total + c2) pi = wide_leaf_first(r2) + (uint32_t)(lane - total);
        total += c2;
      }
      __syncwarp();
      if (lane < total) {
        float tb;
        if (slab(rb, __ldg(S.pbox + 2u * pi), __ldg(S.pbox + 2u * pi + 1u), 0.0f, kInf, tb)) {
          const PrimGeo g = load_geo(S.prims, pi);
          Chord ch;
          if (chord_setup<kAcc>(g, o, d, ch) && ch.t_out > 0.0f) f(pi, g, ch);
        }
      }
    } else {
      const float4* node = S.wide + (size_t)ref * 64u;
      const float4 lo = __ldg(node + lane);
      const float4 hi = __ldg(node + 32 + lane);
      const uint32_t cref = __float_as_uint(lo.w);
      float tnear = 0.f;
      const bool hit = (cref != kEmptyRef) && slab(rb, lo, hi, 0.0f, kInf, tnear);
      const unsigned m = __ballot_sync(kFull, hit);
      const int nh = __popc(m);
      if (nh > 0) {
        if ((uint32_t)(sp + nh) > S.stack_cap) {  // cannot happen for a BVH of the recorded depth
          status |= kStatusStackOverflow;
          break;
        }
        const int first = __ffs(m) - 1;
        if (hit && lane != first) stack[sp + __popc(m & lt_mask) - 1] = cref;
        sp += nh - 1;
        ref = __shfl_sync(kFull, cref, first);
        have = true;
      }
    }
    __syncwarp();
  }
  __syncwarp();
}

template <bool kAcc>
__device__ RaySums ray_sums(const SceneView& S, const float4* __restrict__ emis, uint32_t* stack, float3 o, float3 d,
                            uint32_t& status, unsigned long long& crossings) {
  double s = 0.0, r = 0.0, g = 0.0, b = 0.0;
  warp_visit<kAcc>(S, stack, o, d, status, [&](uint32_t pi, const PrimGeo& geo, const Chord& ch) {
    const float tau = chord_tau0<kAcc>(ch, geo.icf);
    const float4 e = __ldg(emis + pi);
    s += (double)tau;
    r += (double)tau * (double)e.x;
    g += (double)tau * (double)e.y;
    b += (double)tau * (double)e.z;
    ++crossings;
  });
  return RaySums{(float)warp_sum(s), (float)warp_sum(r), (float)warp_sum(g), (float)warp_sum(b)};
}

// A block of up to 8 warps takes a pixel, a warp each of its samples.
template <bool kAcc>
__global__ void __launch_bounds__(256, kAcc ? 2 : 4) k_emis_forward_ray(SceneView S, EnvView E, CameraView C, ParamsView P,
                                                                       const float4* __restrict__ emis,
                                                                       float4* __restrict__ out, unsigned int* work,
                                                                       Counters* ctr) {
  __shared__ float radiance[8][3];
  __shared__ uint32_t taken;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  uint32_t* stack = reinterpret_cast<uint32_t*>(vp_dyn_smem) + warp * S.stack_cap;
  uint32_t status = 0;
  unsigned long long crossings = 0;
  while (true) {
    if (threadIdx.x == 0) taken = atomicAdd(work, 1u);
    __syncthreads();
    const uint32_t pix = taken;
    if (pix >= P.width * P.height) break;
    float3 sum = f3(0.f, 0.f, 0.f);
    for (uint32_t s0 = 0; s0 < P.spp_total; s0 += warps) {
      if (s0 + warp < P.spp_total) {
        const PacketRay r = packet_ray(C, P, pix % P.width, pix / P.width, s0 + warp);
        const RaySums rs = ray_sums<kAcc>(S, emis, stack, r.o, r.d, status, crossings);
        const float3 L = ray_radiance(rs, env_lookup(E, r.d));
        if (lane == 0) radiance[warp][0] = L.x, radiance[warp][1] = L.y, radiance[warp][2] = L.z;
      }
      __syncthreads();
      for (uint32_t j = 0; j < min(warps, P.spp_total - s0); ++j)  // the pixel's samples in order
        sum = add(sum, f3(radiance[j][0], radiance[j][1], radiance[j][2]));
      __syncthreads();
    }
    const float inv = 1.0f / (float)P.spp_total;
    if (threadIdx.x == 0) out[pix] = make_float4(sum.x * inv, sum.y * inv, sum.z * inv, 1.0f);
    if (__syncthreads_or(status != 0u)) break;
  }
  if (status) atomicOr(&ctr->status, status);
  if (P.measure) atomicAdd(&ctr->crossings, crossings);
}

// dtau/dp and dtau/dw of one chord, with tau itself, where p = W (x0 - mu), w = W d and x0 is a
// point of the ray taken as fixed:
//   tau = icf |w|^-1 exp(-d2/2) [erf(h/sqrt2) - erf(u/sqrt2)],  h = sqrt(9 - d2),
//   A = w.w, B = p.w, d2 = p.p - B^2/A, u = B/sqrt(A) when the segment starts at x0 (origin inside
//   the chord, x0 = o), else u = -h.  The boundary terms of the moving 3-sigma limits enter through
//   h: icf |w|^-1 exp(-d2/2) sqrt(2/pi) exp(-h^2/2) = icf |w|^-1 sqrt(2/pi) exp(-9/2).
// For a ray that enters the chord (t_in >= 0) tau depends on the line only, so x0 is the closest
// approach o + t_c d: then |p| <= 3 and no term carries the camera's lever arm |o - mu| / s (which
// would make the accumulated dLoss/dW cancel to a few digits).  For an origin inside the chord,
// x0 = o, already within 3 whitened units.  v returns x0 - mu, formed as the chord set-up forms it
// (o - mu exact as a float pair, plus t_c d).  FP32; under kAcc p and d2 are float pairs, as in
// chord_accurate.  Returns false (no contribution) for a segment below RAY_SEGMENT_MIN_LENGTH.
template <bool kAcc>
__device__ __forceinline__ bool tau_grad(const PrimGeo& g, const Chord& ch, float3 o, float3 d, float& tau,
                                         float3& v, float3& dp, float3& dw) {
  const float t0 = fmaxf(ch.t_in, 0.0f);
  if (ch.t_out - t0 <= kSegmentMin) return false;
  const bool inside = !(ch.t_in >= 0.0f);
  float Dh[3], Dl[3];
  two_sum(o.x, -g.a.x, Dh[0], Dl[0]);
  two_sum(o.y, -g.a.y, Dh[1], Dl[1]);
  two_sum(o.z, -g.a.z, Dh[2], Dl[2]);
  const float t = inside ? 0.0f : ch.tc;
  const float dd[3] = {d.x, d.y, d.z};
  float vh[3], vl[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float pr, pe, sm, se;
    two_prod(t, dd[k], pr, pe);
    two_sum(Dh[k], pr, sm, se);
    fast_two_sum(sm, __fadd_rn(se, __fadd_rn(pe, Dl[k])), vh[k], vl[k]);
  }
  const float W[9] = {g.a.w, g.b.x, g.b.y, g.b.z, g.b.w, g.c.x, g.c.y, g.c.z, g.c.w};
  float px, py, pz, pp, pplo = 0.0f;
  if constexpr (kAcc) {
    FF p3[3];
    mat_vec_ff(W, vh, vl, p3);
    const FF n2 = norm2_ff(p3);
    px = p3[0].hi, py = p3[1].hi, pz = p3[2].hi;
    pp = n2.hi;
    pplo = n2.lo;
  } else {
    const float3 pv = whiten(g, f3(vh[0] + vl[0], vh[1] + vl[1], vh[2] + vl[2]));
    px = pv.x, py = pv.y, pz = pv.z;
    pp = dot3(pv, pv);
  }
  const float3 w3 = whiten(g, d);
  const float wx = w3.x, wy = w3.y, wz = w3.z;
  const float A = dot3(w3, w3), B = fmaf(px, wx, fmaf(py, wy, pz * wz));
  const float rA = __frcp_rn(A), rw = __frsqrt_rn(A);
  // d2 = p.p - B^2 / A; at the closest approach B = 0 up to rounding, so the pair's low part
  // carries the bits that matter on grazing chords
  const float d2 = __fadd_rn(fmaf(-B * B, rA, pp), pplo);
  if (!(d2 < 9.0f)) return false;
  const float h = sqrtf(9.0f - d2);
  const float u = inside ? B * rw : -h;
  const float E = expf(-0.5f * d2);
  const float base = g.icf * rw;
  const float k2pi = 0.79788456080286535588f, kis2 = 0.70710678118654752440f;
  const float D = inside ? erff(h * kis2) - erff(u * kis2) : 2.0f * erff(h * kis2);
  const float tt = base * E * D;
  const float dtau_dh = (inside ? 1.0f : 2.0f) * base * k2pi * 0.011108996538242306f;
  const float dtau_dd2 = -0.5f * tt - dtau_dh * 0.5f / h;
  const float dtau_du = inside ? -base * E * k2pi * expf(-0.5f * u * u) : 0.0f;
  const float gP = dtau_dd2;
  const float gB = dtau_dd2 * (-2.0f * B * rA) + dtau_du * rw;
  const float gA = -0.5f * tt * rA + dtau_dd2 * B * B * rA * rA - dtau_du * 0.5f * B * rA * rw;
  tau = tt;
  v = f3(vh[0] + vl[0], vh[1] + vl[1], vh[2] + vl[2]);
  dp = f3(2.0f * gP * px + gB * wx, 2.0f * gP * py + gB * wy, 2.0f * gP * pz + gB * wz);
  dw = f3(2.0f * gA * wx + gB * px, 2.0f * gA * wy + gB * py, 2.0f * gA * wz + gB * pz);
  return true;
}

// Sums of 16 values over the warp, two lanes a value: lane l returns the sum of v[(l >> 1)], bits of the index
// from the top (15 shuffles halve the values a lane carries, one adds the last pair).
__device__ __forceinline__ float warp_sum16(float (&v)[16]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int half = 8, bit = 16; half > 0; half >>= 1, bit >>= 1) {
    const bool up = (lane & bit) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float send = up ? v[i] : v[half + i];
      const float keep = up ? v[half + i] : v[i];
      v[i] = keep + __shfl_xor_sync(kFull, send, bit);
    }
  }
  return v[0] + __shfl_xor_sync(kFull, v[0], 1);
}

template <bool kAcc, int kGroup>
__global__ void __launch_bounds__(32 * kGroup, (kAcc ? 16 : kBwdWarps) / kGroup) k_emis_backward(SceneView S, EnvView E, CameraView C, ParamsView P,
                                                       Tiling T, float extent, const float4* __restrict__ emis,
                                                       const float4* __restrict__ dl_dpix, float4* __restrict__ acc,
                                                       unsigned int* work, Counters* ctr) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto& sh = *reinterpret_cast<PacketShared<kGroup>*>(vp_dyn_smem);
  uint32_t* stack = reinterpret_cast<uint32_t*>(vp_dyn_smem + sizeof(sh)) + warp * packet_words(S.stack_cap, true);
  uint32_t* list = stack + ((S.stack_cap + 4u) & ~3u);
  const float inv_spp = 1.0f / (float)P.spp_total;
  uint32_t status = 0;
  unsigned long long crossings = 0;
  while (true) {
    if (threadIdx.x == 0) sh.tile = atomicAdd(work, 1u);
    __syncthreads();
    const uint32_t tile = sh.tile;
    if (tile >= T.tiles) break;
    const PacketLane l = packet_lane(T, P, tile);
    const float4 gp = l.on ? __ldg(dl_dpix + (size_t)l.py * P.width + l.px) : make_float4(0.f, 0.f, 0.f, 0.f);
    const bool wanted = gp.x != 0.0f || gp.y != 0.0f || gp.z != 0.0f;  // else nothing flows back (e.g. a crop)
    const float3 G = f3(gp.x * inv_spp, gp.y * inv_spp, gp.z * inv_spp);
    for (uint32_t s0 = 0; s0 < P.spp_total; s0 += T.k) {
      const uint32_t k = min(T.k, P.spp_total - s0);
      const bool active = wanted && l.s < k;
      if (!__any_sync(kFull, active)) continue;
      const PacketRay r = packet_ray(C, P, l.px, l.py, s0 + l.s);
      const float3 o = r.o, d = r.d;
      if (warp == 0) packet_bounds(C, extent, active, r.x, r.y, o, d, &sh.bounds);
      uint32_t n = 0;
      const RaySums rs = packet_sums<kAcc, true, kGroup>(S, emis, stack, sh, o, d, active, status, crossings, list, n);
      const float3 env = env_lookup(E, d);
      float Tr, a, q;
      opacity_terms(rs.S, Tr, a, q);
      const float gS = G.x * fmaf(rs.r, q, -Tr * env.x) + G.y * fmaf(rs.g, q, -Tr * env.y) +
                       G.z * fmaf(rs.b, q, -Tr * env.z);
      const float3 gC = mul(G, a);
      auto scatter = [&](uint32_t gi, const PrimGeo& geo, const Chord& ch, bool hit) {
        float v16[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v16[i] = 0.f;
        float tau;
        float3 v, dp, dw;
        if (hit && tau_grad<kAcc>(geo, ch, o, d, tau, v, dp, dw)) {
          const float4 e = __ldg(emis + gi);
          const float gt = gS + gC.x * e.x + gC.y * e.y + gC.z * e.z;
          const float3 gp3 = mul(dp, gt), gw3 = mul(dw, gt);
          // dLoss/dW_kl = gp_k v_l + gw_k d_l
          v16[0] = fmaf(gp3.x, v.x, gw3.x * d.x), v16[1] = fmaf(gp3.x, v.y, gw3.x * d.y);
          v16[2] = fmaf(gp3.x, v.z, gw3.x * d.z), v16[3] = fmaf(gp3.y, v.x, gw3.y * d.x);
          v16[4] = fmaf(gp3.y, v.y, gw3.y * d.y), v16[5] = fmaf(gp3.y, v.z, gw3.y * d.z);
          v16[6] = fmaf(gp3.z, v.x, gw3.z * d.x), v16[7] = fmaf(gp3.z, v.y, gw3.z * d.y);
          v16[8] = fmaf(gp3.z, v.z, gw3.z * d.z);
          v16[9] = gp3.x, v16[10] = gp3.y, v16[11] = gp3.z;
          v16[12] = gt * tau, v16[13] = gC.x * tau, v16[14] = gC.y * tau, v16[15] = gC.z * tau;
        }
        const float sum = warp_sum16(v16);
        if (!(lane & 1)) atomicAdd(reinterpret_cast<float*>(acc + 4u * gi) + (lane >> 1), sum);
      };
      __syncwarp();
      if (n <= kListCap) {
        for (uint32_t i = 0; i < n; ++i) {
          const uint32_t gi = list[i];
          const PrimGeo g = load_geo(S.prims, gi);
          Chord ch;
          const bool hit = active && chord_setup<kAcc>(g, o, d, ch) && ch.t_out > 0.0f;
          scatter(gi, g, ch, hit);
        }
      } else {
        for (uint32_t i = 0; i < sh.n_front; ++i) {
          if (sh.owner[i] != (uint8_t)warp) continue;
          if (lane == 0) stack[0] = sh.front[i];
          __syncwarp();
          packet_visit<kAcc>(S, stack, &sh.bounds, o, d, active, status, 1, scatter);
        }
      }
      __syncthreads();  // the packet's shared state is the next pass's
    }
    if (__syncthreads_or(status != 0u)) break;
  }
  if (status) atomicOr(&ctr->status, status);
  if (P.measure) atomicAdd(&ctr->crossings, crossings);
}

// The adjoint with a warp on each ray: its second traversal adds every (ray, Gaussian) pair's terms by itself.
template <bool kAcc>
__global__ void __launch_bounds__(256, kAcc ? 2 : 4) k_emis_backward_ray(SceneView S, EnvView E, CameraView C, ParamsView P,
                                                                        const float4* __restrict__ emis,
                                                                        const float4* __restrict__ dl_dpix,
                                                                        float4* __restrict__ acc, unsigned int* work,
                                                                        Counters* ctr) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t* stack = reinterpret_cast<uint32_t*>(vp_dyn_smem) + warp * S.stack_cap;
  const uint32_t n_rays = P.width * P.height * P.spp_total;
  const float inv_spp = 1.0f / (float)P.spp_total;
  uint32_t status = 0;
  unsigned long long crossings = 0;
  while (true) {
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(work, 1u);
    item = __shfl_sync(kFull, item, 0);
    if (item >= n_rays) break;
    const uint32_t pix = item / P.spp_total;
    const float4 gp = __ldg(dl_dpix + pix);
    if (gp.x == 0.0f && gp.y == 0.0f && gp.z == 0.0f) continue;  // nothing flows back (e.g. a crop)
    const float3 G = f3(gp.x * inv_spp, gp.y * inv_spp, gp.z * inv_spp);
    const PacketRay ray = packet_ray(C, P, pix % P.width, pix / P.width, item % P.spp_total);
    const float3 o = ray.o, d = ray.d;
    const RaySums rs = ray_sums<kAcc>(S, emis, stack, o, d, status, crossings);
    const float3 env = env_lookup(E, d);
    float T, a, q;
    opacity_terms(rs.S, T, a, q);
    const float gS = G.x * fmaf(rs.r, q, -T * env.x) + G.y * fmaf(rs.g, q, -T * env.y) + G.z * fmaf(rs.b, q, -T * env.z);
    const float3 gC = mul(G, a);
    warp_visit<kAcc>(S, stack, o, d, status, [&](uint32_t pi, const PrimGeo& geo, const Chord& ch) {
      float tau;
      float3 v, dp, dw;
      if (!tau_grad<kAcc>(geo, ch, o, d, tau, v, dp, dw)) return;
      const float4 e = __ldg(emis + pi);
      const float gt = gS + gC.x * e.x + gC.y * e.y + gC.z * e.z;
      const float3 gp3 = mul(dp, gt), gw3 = mul(dw, gt);
      // dLoss/dW_kl = gp_k v_l + gw_k d_l
      float4* a4 = acc + 4u * pi;
      atomicAdd(a4 + 0, make_float4(fmaf(gp3.x, v.x, gw3.x * d.x), fmaf(gp3.x, v.y, gw3.x * d.y),
                                    fmaf(gp3.x, v.z, gw3.x * d.z), fmaf(gp3.y, v.x, gw3.y * d.x)));
      atomicAdd(a4 + 1, make_float4(fmaf(gp3.y, v.y, gw3.y * d.y), fmaf(gp3.y, v.z, gw3.y * d.z),
                                    fmaf(gp3.z, v.x, gw3.z * d.x), fmaf(gp3.z, v.y, gw3.z * d.y)));
      atomicAdd(a4 + 2, make_float4(fmaf(gp3.z, v.z, gw3.z * d.z), gp3.x, gp3.y, gp3.z));
      atomicAdd(a4 + 3, make_float4(gt * tau, gC.x * tau, gC.y * tau, gC.z * tau));
    });
    if (status) break;
  }
  if (status) atomicOr(&ctr->status, status);
  if (P.measure) atomicAdd(&ctr->crossings, crossings);
}

// Per-Gaussian accumulators (internal order) -> gradients of the caller's parameters (caller
// order), added to out[].  W_kl = R_lk / s_k with R = R(q / |q|) (the build's rotation matrix) and
// icf proportional to density / (s_x s_y s_z):
//   dL/dmu = -W^T sum(g dtau/dp);  dL/ds_k = -(sum_l gW_kl W_kl + gK) / s_k;
//   dL/dR_lk = gW_kl / s_k -> dL/dq_hat -> dL/dq = (g - q_hat (q_hat . g)) / |q|;
//   dL/ddensity = gK / density.
__global__ void k_emis_finish(uint32_t n, const uint32_t* __restrict__ perm, const float4* __restrict__ prims,
                              const float4* __restrict__ raw, const float4* __restrict__ acc, int scale_is_log,
                              float* __restrict__ g_mean, float* __restrict__ g_scale, float* __restrict__ g_quat,
                              float* __restrict__ g_dens, float* __restrict__ g_emis) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t c = perm[i];
  const float4 a0 = acc[4 * i], a1 = acc[4 * i + 1], a2 = acc[4 * i + 2], a3 = acc[4 * i + 3];
  const float gW[3][3] = {{a0.x, a0.y, a0.z}, {a0.w, a1.x, a1.y}, {a1.z, a1.w, a2.x}};
  const float gP[3] = {a2.y, a2.z, a2.w};
  const float gK = a3.x;
  const float4 r0 = prims[4 * i], r1 = prims[4 * i + 1], r2 = prims[4 * i + 2];
  const float W[3][3] = {{r0.w, r1.x, r1.y}, {r1.z, r1.w, r2.x}, {r2.y, r2.z, r2.w}};
  const float4 q4 = raw[2 * i], sd = raw[2 * i + 1];
  for (int l = 0; l < 3; ++l) g_mean[3 * c + l] += -(W[0][l] * gP[0] + W[1][l] * gP[1] + W[2][l] * gP[2]);
  float s[3] = {sd.x, sd.y, sd.z};
  if (scale_is_log)
    for (int k = 0; k < 3; ++k) s[k] = expf(s[k]);
  for (int k = 0; k < 3; ++k) {
    const float gs = -(gW[k][0] * W[k][0] + gW[k][1] * W[k][1] + gW[k][2] * W[k][2] + gK) / s[k];
    g_scale[3 * c + k] += scale_is_log ? gs * s[k] : gs;
  }
  // dL/dR_lk = gW_kl / s_k
  float gR[3][3];
  for (int l = 0; l < 3; ++l)
    for (int k = 0; k < 3; ++k) gR[l][k] = gW[k][l] / s[k];
  const float qn = sqrtf(q4.x * q4.x + q4.y * q4.y + q4.z * q4.z + q4.w * q4.w);
  const float w = q4.x / qn, x = q4.y / qn, y = q4.z / qn, z = q4.w / qn;
  // R(q) = [[1-2(y2+z2), 2(xy-wz), 2(xz+wy)], [2(xy+wz), 1-2(x2+z2), 2(yz-wx)], [2(xz-wy), 2(yz+wx), 1-2(x2+y2)]]
  const float gw = 2.0f * (-z * gR[0][1] + y * gR[0][2] + z * gR[1][0] - x * gR[1][2] - y * gR[2][0] + x * gR[2][1]);
  const float gx = 2.0f * (y * gR[0][1] + z * gR[0][2] + y * gR[1][0] - 2.0f * x * gR[1][1] - w * gR[1][2] +
                           z * gR[2][0] + w * gR[2][1] - 2.0f * x * gR[2][2]);
  const float gy = 2.0f * (-2.0f * y * gR[0][0] + x * gR[0][1] + w * gR[0][2] + x * gR[1][0] + z * gR[1][2] -
                           w * gR[2][0] + z * gR[2][1] - 2.0f * y * gR[2][2]);
  const float gz = 2.0f * (-2.0f * z * gR[0][0] - w * gR[0][1] + x * gR[0][2] + w * gR[1][0] - 2.0f * z * gR[1][1] +
                           y * gR[1][2] + x * gR[2][0] + y * gR[2][1]);
  const float dotq = w * gw + x * gx + y * gy + z * gz;
  g_quat[4 * c + 0] += (gw - w * dotq) / qn;
  g_quat[4 * c + 1] += (gx - x * dotq) / qn;
  g_quat[4 * c + 2] += (gy - y * dotq) / qn;
  g_quat[4 * c + 3] += (gz - z * dotq) / qn;
  g_dens[c] += gK / sd.w;
  if (g_emis) {
    g_emis[3 * c + 0] += a3.y;
    g_emis[3 * c + 1] += a3.z;
    g_emis[3 * c + 2] += a3.w;
  }
}

__global__ void k_set_emission(uint32_t n, const uint32_t* __restrict__ perm, const float* __restrict__ rgb,
                               float4* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t c = perm[i];
  out[i] = make_float4(rgb[3 * c], rgb[3 * c + 1], rgb[3 * c + 2], 0.0f);
}

template <class K>
int blocks_per_sm(K kernel, int threads, size_t smem) {
  int b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, threads, smem) != cudaSuccess) b = 1;
  return b < 1 ? 1 : b;
}

vp_status ensure_emission(vp_scene* s) {
  if (s->emis) return VP_OK;
  vp_status r;
  if ((r = dev_alloc(&s->emis, s->info.count, s->ctx->stream))) return r;
  VP_CUDA(cudaMemsetAsync(s->emis, 0, 16ull * s->info.count, s->ctx->stream));
  s->info.device_bytes += 16ull * s->info.count;
  return VP_OK;
}

struct Common {
  CameraView cv;
  ParamsView P;
  Tiling tiles;
  float extent;
};

// Warps a packet's block has: more where there are few tiles to fill the chip and hide the dense ones, fewer
// where they only wait for one another at the block's barriers.  Forward, 100k-Gaussian cloud: 16,384 tiles
// 3.0 / 3.3 ms with 2 / 4 warps; 4,800 tiles 2.0 / 1.6 ms.
// A tree so deep that the warps' stacks do not fit a block takes fewer.
template <class F>
vp_status with_group(uint32_t tiles, uint32_t stack_cap, F&& f) {
  constexpr size_t kMost = 200 * 1024;
  if (tiles >= 10240u || packet_smem<4>(stack_cap, true) > kMost) return f(std::integral_constant<int, 2>{});
  if (tiles >= 1024u || packet_smem<8>(stack_cap, true) > kMost) return f(std::integral_constant<int, 4>{});
  return f(std::integral_constant<int, 8>{});
}

// Images of few rays take a warp on each ray: their packets are few, and wide at one or two samples a pixel, so
// the chip waits for the densest.  Both sides at 12,800 / 40,000 / 65,536 / 180,000 rays (8, 1, 1 and 8 samples a pixel),
// packets and then rays:
// forward, 100k Gaussians 2.18 / 1.78 / 1.67 / 1.84 and 0.57 / 1.04 / 1.63 / 3.96 ms, 20k Gaussians 0.59 / 0.47 /
// 0.45 / 0.49 and 0.17 / 0.30 / 0.44 / 1.06, 5k Gaussians 0.18 / 0.16 / 0.155 / 0.17 and 0.10 / 0.145 / 0.20 / 0.45;
// ACCURATE crosses over at four fifths of that.  A gradient step at 38k / 154k rays (two views the latter; build
// and forward in it): 100k Gaussians 9.4 / 15.0 and 5.7 / 20.5 ms, 5k 2.32 / 2.75 and 2.19 / 3.77: the adjoint's
// packets, which it meets twice, pay later.  Sample counts that fill a packet badly do not move the line: 70,000 rays through
// 100k Gaussians take 1.68 ms in packets at 1 and at 17 samples a pixel, 2.37 at 33, which is a second pass for one ray.
bool few_rays(const ParamsView& P, uint32_t count, bool adjoint) {
  uint64_t limit = count >= 16384u ? 65536u : 45056u;
  if (P.accurate) limit = limit * 4u / 5u;
  if (adjoint) limit = limit * 3u / 2u;
  return (uint64_t)P.width * P.height * P.spp_total <= limit;
}

Tiling tiling(uint32_t width, uint32_t height, uint32_t spp) {
  Tiling t{};
  t.k = std::min(spp, 32u);
  uint32_t log = 0;
  while ((2u << log) * t.k <= 32u) ++log;  // 2^log pixels
  t.tw = 1u << ((log + 1u) / 2u);
  t.th = 1u << (log / 2u);
  t.tiles_x = (width + t.tw - 1u) / t.tw;
  t.tiles = t.tiles_x * ((height + t.th - 1u) / t.th);
  return t;
}

vp_status prepare(vp_scene* s, vp_env* e, const vp_camera* cam, const vp_render_params* p, Common& c) {
  if (!s || !e || !cam || !p) return fail(VP_ERROR_INVALID_ARGUMENT, "NULL argument");
  if (s->ctx != e->ctx) return fail(VP_ERROR_INVALID_ARGUMENT, "objects belong to different contexts");
  if (s->info.count == 0) return fail(VP_ERROR_INVALID_ARGUMENT, "the emission model needs a scene with Gaussians");
  if (p->width == 0 || p->height == 0 || p->spp == 0)
    return fail(VP_ERROR_INVALID_ARGUMENT, "width, height and spp must be positive");
  if ((uint64_t)p->width * p->height >= (1ull << 32)) return fail(VP_ERROR_LIMIT, "image too large");
  VP_CUDA(cudaSetDevice(s->ctx->device));
  build_camera(*cam, p->width, p->height, c.cv);
  c.P = make_params(*p, s);
  if (packet_smem<2>(s->view.stack_cap, true) > 200 * 1024 || (size_t)8 * s->view.stack_cap * 4u > 200 * 1024)
    return fail(VP_ERROR_LIMIT, "BVH too deep for the shared-memory stack");
  c.tiles = tiling(p->width, p->height, p->spp);
  c.extent = 0.0f;
  for (int k = 0; k < 3; ++k)
    c.extent = std::max({c.extent, (float)std::fabs(s->info.bounds_min[k]), (float)std::fabs(s->info.bounds_max[k])});
  vp_status r;
  if ((r = ensure_emission(s))) return r;
  return VP_OK;
}

vp_status finish_stats(vp_context* ctx, const vp_render_params* p, uint32_t launches, vp_render_stats* stats) {
  VP_CUDA(cudaEventRecord(ctx->ev1, ctx->stream));
  vp_status r;
  if ((r = fetch_counters(ctx))) return r;
  VP_CUDA(cudaStreamSynchronize(ctx->stream));
  const Counters& c = *ctx->host_counters;
  if (stats) {
    float ms = 0.f;
    VP_CUDA(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
    std::memset(stats, 0, sizeof(*stats));
    stats->ms_kernels = ms;
    stats->paths = (uint64_t)p->width * p->height * p->spp;
    stats->crossings = c.crossings;
    stats->device_status = c.status;
    stats->launches = launches;
  }
  if (c.status) return fail(VP_ERROR_DEVICE_STATUS, "an emission kernel raised device status " + std::to_string(c.status));
  return VP_OK;
}

}  // namespace
}  // namespace vp

using namespace vp;

extern "C" {

vp_status vp_scene_set_emission(vp_scene* s, const float* rgb, int32_t memory) {
  if (!s) return fail(VP_ERROR_INVALID_ARGUMENT, "NULL argument");
  if (s->info.count == 0) return fail(VP_ERROR_INVALID_ARGUMENT, "the emission model needs a scene with Gaussians");
  if (!rgb) return fail(VP_ERROR_INVALID_ARGUMENT, "NULL argument");
  if (memory != VP_MEMORY_HOST && memory != VP_MEMORY_DEVICE) return fail(VP_ERROR_INVALID_ARGUMENT, "bad memory kind");
  VP_CUDA(cudaSetDevice(s->ctx->device));
  cudaStream_t st = s->ctx->stream;
  const uint32_t n = s->info.count;
  vp_status r;
  if ((r = ensure_emission(s))) return r;
  const float* src = rgb;
  float* tmp = nullptr;
  if (memory == VP_MEMORY_HOST) {
    if ((r = dev_alloc(&tmp, 3ull * n, st))) return r;
    VP_CUDA(cudaMemcpyAsync(tmp, rgb, 12ull * n, cudaMemcpyHostToDevice, st));
    src = tmp;
  }
  k_set_emission<<<(n + 255) / 256, 256, 0, st>>>(n, s->perm, src, s->emis);
  const cudaError_t e = cudaGetLastError();
  if (tmp) dev_free(tmp, st);
  if (e != cudaSuccess) return cuda_fail(e, "k_set_emission");
  VP_CUDA(cudaStreamSynchronize(st));
  return VP_OK;
}

vp_status vp_render_emission(vp_scene* s, vp_env* e, const vp_camera* cam, const vp_render_params* p,
                             float* out_rgba, int32_t memory, vp_render_stats* stats) {
  if (!out_rgba) return fail(VP_ERROR_INVALID_ARGUMENT, "NULL argument");
  if (memory != VP_MEMORY_HOST && memory != VP_MEMORY_DEVICE) return fail(VP_ERROR_INVALID_ARGUMENT, "bad memory kind");
  Common c;
  vp_status r;
  if ((r = prepare(s, e, cam, p, c))) return r;
  vp_context* ctx = s->ctx;
  cudaStream_t st = ctx->stream;
  const size_t n_pix = (size_t)p->width * p->height;
  float4* out = reinterpret_cast<float4*>(out_rgba);
  float4* tmp = nullptr;
  if (memory == VP_MEMORY_HOST) {
    if ((r = dev_alloc(&tmp, n_pix, st))) return r;
    out = tmp;
  }
  if ((r = clear_counters(ctx))) return r;
  VP_CUDA(cudaEventRecord(ctx->ev0, st));
  auto per_ray = [&]() -> vp_status {
    auto kern = c.P.accurate ? k_emis_forward_ray<true> : k_emis_forward_ray<false>;
    const int warps = (int)std::min(std::max(c.P.spp_total, 1u), 8u);
    const size_t smem = (size_t)warps * s->view.stack_cap * 4u;
    if (smem > 47 * 1024) VP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int blocks = ctx->sm_count * blocks_per_sm(kern, 32 * warps, smem);
    kern<<<blocks, 32 * warps, smem, st>>>(s->view, e->view, c.cv, c.P, s->emis, out, ctx->work_counter, ctx->counters);
    return VP_OK;
  };
  auto packets = [&](auto group) -> vp_status {
    constexpr int G = decltype(group)::value;
    auto kern = c.P.accurate ? k_emis_forward<true, G> : k_emis_forward<false, G>;
    const size_t smem = packet_smem<G>(s->view.stack_cap, false);
    if (smem > 48 * 1024) VP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int blocks = ctx->sm_count * blocks_per_sm(kern, 32 * G, smem);
    kern<<<blocks, 32 * G, smem, st>>>(s->view, e->view, c.cv, c.P, c.tiles, c.extent, s->emis, out, ctx->work_counter,
                                       ctx->counters);
    return VP_OK;
  };
  const vp_status lr = few_rays(c.P, s->info.count, false) ? per_ray() : with_group(c.tiles.tiles, s->view.stack_cap, packets);
  if (lr) {
    dev_free(tmp, st);
    return lr;
  }
  VP_CUDA(cudaGetLastError());
  r = finish_stats(ctx, p, 1, stats);
  if (tmp) {
    if (r == VP_OK) {
      const cudaError_t ce = cudaMemcpy(out_rgba, tmp, 16ull * n_pix, cudaMemcpyDeviceToHost);
      if (ce != cudaSuccess) r = cuda_fail(ce, "vp_render_emission read-back");
    }
    dev_free(tmp, st);
    cudaStreamSynchronize(st);
  }
  return r;
}

vp_status vp_render_emission_backward(vp_scene* s, vp_env* e, const vp_camera* cam, const vp_render_params* p,
                                      const float* dloss_drgba, int32_t memory, vp_gaussian_grads* grads,
                                      vp_render_stats* stats) {
  if (!dloss_drgba || !grads || !grads->mean || !grads->scale || !grads->quat_wxyz || !grads->density)
    return fail(VP_ERROR_INVALID_ARGUMENT, "NULL argument");
  if (memory != VP_MEMORY_HOST && memory != VP_MEMORY_DEVICE) return fail(VP_ERROR_INVALID_ARGUMENT, "bad memory kind");
  if (grads->memory != VP_MEMORY_HOST && grads->memory != VP_MEMORY_DEVICE)
    return fail(VP_ERROR_INVALID_ARGUMENT, "bad memory kind of the gradient arrays");
  Common c;
  vp_status r;
  if ((r = prepare(s, e, cam, p, c))) return r;
  vp_context* ctx = s->ctx;
  cudaStream_t st = ctx->stream;
  const uint32_t n = s->info.count;
  const size_t n_pix = (size_t)p->width * p->height;
  // scratch: per-Gaussian accumulators, the staged upstream gradient, staged outputs
  float4* acc = nullptr;
  float4* dl = nullptr;
  float* gout = nullptr;  // 14 n floats: mean 3n, scale 3n, quat 4n, density n, emission 3n
  const float4* dsrc = reinterpret_cast<const float4*>(dloss_drgba);
  auto cleanup = [&]() {
    dev_free(acc, st);
    dev_free(dl, st);
    dev_free(gout, st);
    cudaStreamSynchronize(st);
  };
  if ((r = dev_alloc(&acc, 4ull * n, st))) return r;
  if (memory == VP_MEMORY_HOST) {
    if ((r = dev_alloc(&dl, n_pix, st))) return cleanup(), r;
    VP_CUDA(cudaMemcpyAsync(dl, dloss_drgba, 16ull * n_pix, cudaMemcpyHostToDevice, st));
    dsrc = dl;
  }
  const bool host_out = grads->memory == VP_MEMORY_HOST;
  float *gm = grads->mean, *gs = grads->scale, *gq = grads->quat_wxyz, *gd = grads->density, *ge = grads->emission;
  if (host_out) {
    if ((r = dev_alloc(&gout, 14ull * n, st))) return cleanup(), r;
    VP_CUDA(cudaMemsetAsync(gout, 0, 56ull * n, st));
    gm = gout;
    gs = gout + 3ull * n;
    gq = gout + 6ull * n;
    gd = gout + 10ull * n;
    ge = grads->emission ? gout + 11ull * n : nullptr;
  }
  VP_CUDA(cudaMemsetAsync(acc, 0, 64ull * n, st));
  if ((r = clear_counters(ctx))) return cleanup(), r;
  VP_CUDA(cudaEventRecord(ctx->ev0, st));
  auto per_ray = [&]() -> vp_status {
    auto kern = c.P.accurate ? k_emis_backward_ray<true> : k_emis_backward_ray<false>;
    const size_t smem = 8u * (size_t)s->view.stack_cap * 4u;
    if (smem > 48 * 1024) VP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int blocks = ctx->sm_count * blocks_per_sm(kern, 256, smem);
    kern<<<blocks, 256, smem, st>>>(s->view, e->view, c.cv, c.P, s->emis, dsrc, acc, ctx->work_counter, ctx->counters);
    return VP_OK;
  };
  auto packets = [&](auto group) -> vp_status {
    constexpr int G = decltype(group)::value;
    auto kern = c.P.accurate ? k_emis_backward<true, G> : k_emis_backward<false, G>;
    const size_t smem = packet_smem<G>(s->view.stack_cap, true);
    if (smem > 48 * 1024) VP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int blocks = ctx->sm_count * blocks_per_sm(kern, 32 * G, smem);
    kern<<<blocks, 32 * G, smem, st>>>(s->view, e->view, c.cv, c.P, c.tiles, c.extent, s->emis, dsrc, acc, ctx->work_counter,
                                       ctx->counters);
    return VP_OK;
  };
  const vp_status lr = few_rays(c.P, s->info.count, true) ? per_ray() : with_group(c.tiles.tiles, s->view.stack_cap, packets);
  if (lr) return cleanup(), lr;
  VP_CUDA(cudaGetLastError());
  k_emis_finish<<<(n + 255) / 256, 256, 0, st>>>(n, s->perm, s->prims, s->raw, acc, s->scale_is_log, gm, gs, gq, gd, ge);
  VP_CUDA(cudaGetLastError());
  r = finish_stats(ctx, p, 2, stats);
  if (r == VP_OK && host_out) {
    std::vector<float> h(14ull * n);
    const cudaError_t ce = cudaMemcpy(h.data(), gout, 56ull * n, cudaMemcpyDeviceToHost);
    if (ce != cudaSuccess) {
      r = cuda_fail(ce, "vp_render_emission_backward read-back");
    } else {
      for (size_t k = 0; k < 3ull * n; ++k) grads->mean[k] += h[k];
      for (size_t k = 0; k < 3ull * n; ++k) grads->scale[k] += h[3ull * n + k];
      for (size_t k = 0; k < 4ull * n; ++k) grads->quat_wxyz[k] += h[6ull * n + k];
      for (size_t k = 0; k < 1ull * n; ++k) grads->density[k] += h[10ull * n + k];
      if (grads->emission)
        for (size_t k = 0; k < 3ull * n; ++k) grads->emission[k] += h[11ull * n + k];
    }
  }
  cleanup();
  return r;
}

}  // extern "C"
