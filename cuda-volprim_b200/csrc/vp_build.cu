// Scene build on the device: per-Gaussian precompute, 3-sigma ellipsoid bounds, 63-bit Morton
// codes, radix sort, then two binary trees over the sorted boxes -- a Karras radix tree with a
// bottom-up refit (the thread-per-ray megakernel's tree) and a PLOC agglomerative clustering
// (the other engines' tree) -- and two collapses of the latter: a 32-wide BVH (the warp-per-ray queries'), whose
// depth-first leaf order becomes the scene order of the Gaussians, and a compressed 8-wide one (the thread-per-ray
// queries', vp_trace8.cuh).
//
// Replaces the reference's host Morton sort + OptiX unit-sphere GAS / instance IAS build
// (src/thesis/host/app/renderer.cpp:85-173, include/thesis/host/utils/math.h:103-131,
// include/thesis/host/optix/acceleration_structure.h:23-87) and the Primitive precompute
// (include/thesis/device/params/primitive.h:70-87) plus PLY-load validation
// (src/thesis/host/utils/io/ply.cpp:124-172).

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "vp_internal.h"
#include "vp_trace8.cuh"

namespace vp {
namespace {

struct ErrorWords {
  int bad_scale, bad_density, bad_center;  // lowest failing index (INT_MAX = none)
  unsigned int any_albedo;                 // 1 if some albedo component > 0
  unsigned int opaque_cores;               // Gaussians opaque at their core (vp_tau_order AUTO)
  unsigned int mixed_albedo;               // 1 if some albedo differs from the first Gaussian's
  float albedo0[3];                        // the first Gaussian's
  float overlap;                           // the share of the scene a Gaussian fills (k_overlap)
};

// A Gaussian is "opaque at its core" when the optical depth through its centre along its thinnest
// direction, M / (2 pi s_mid s_max), is at least this (4 x MAX_OPTICAL_DEPTH).
constexpr float kOpaqueCoreTau = 4.0f * kMaxOpticalDepth;

__device__ __forceinline__ float clamp_albedo(float v) {
  if (!isfinite(v)) return 0.0f;
  if (v < 0.0f) return 0.0f;
  if (v > 1.0f) return 1.0f;
  return v;
}

// One thread per Gaussian: the reference's Primitive constructor arithmetic in FP32 (host
// order; IEEE division/sqrt), the whitening matrix W = diag(1/s) R(q)^T and the 3-sigma
// ellipsoid's axis-aligned bound (from renderer.cpp:142-157's local-to-world TRS with 3x scale).
__global__ void k_precompute(uint32_t n, const float* __restrict__ mean,
                             const float* __restrict__ scale, const float* __restrict__ quat,
                             const float* __restrict__ density, const float* __restrict__ albedo,
                             int scale_is_log, float sigma_multiplier, float4* __restrict__ rec,
                             float4* __restrict__ lo, float4* __restrict__ hi,
                             ErrorWords* __restrict__ err) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float cx = mean[3 * i], cy = mean[3 * i + 1], cz = mean[3 * i + 2];
  float sx = scale[3 * i], sy = scale[3 * i + 1], sz = scale[3 * i + 2];
  if (scale_is_log) {
    sx = expf(sx);
    sy = expf(sy);
    sz = expf(sz);
  }
  const float qw = quat[4 * i], qx = quat[4 * i + 1], qy = quat[4 * i + 2], qz = quat[4 * i + 3];
  // UnitQuaternion::from: rlength(float4(w,x,y,z)) = 1 / sqrt(fma(w,w,fma(x,x,fma(y,y,z*z))))
  const float qr = __fdiv_rn(1.0f, __fsqrt_rn(fmaf(qw, qw, fmaf(qx, qx, fmaf(qy, qy, __fmul_rn(qz, qz))))));
  const float w = __fmul_rn(qw, qr), x = __fmul_rn(qx, qr), y = __fmul_rn(qy, qr), z = __fmul_rn(qz, qr);
  const float M = __fmul_rn(density[i], sigma_multiplier);  // ply.cpp:116
  float ar = 0.f, ag = 0.f, ab = 0.f;
  if (albedo) {
    ar = clamp_albedo(albedo[3 * i]);
    ag = clamp_albedo(albedo[3 * i + 1]);
    ab = clamp_albedo(albedo[3 * i + 2]);
  }
  if (ar > 0.f || ag > 0.f || ab > 0.f) atomicOr(&err->any_albedo, 1u);
  if (albedo && (ar != clamp_albedo(albedo[0]) || ag != clamp_albedo(albedo[1]) || ab != clamp_albedo(albedo[2])))
    atomicOr(&err->mixed_albedo, 1u);
  if (i == 0u) err->albedo0[0] = ar, err->albedo0[1] = ag, err->albedo0[2] = ab;
  const bool scale_ok = sx > 0.f && sy > 0.f && sz > 0.f && isfinite(sx) && isfinite(sy) && isfinite(sz);
  if (!scale_ok) atomicMin(&err->bad_scale, (int)i);
  if (!(M > 0.f) || !isfinite(M)) atomicMin(&err->bad_density, (int)i);
  if (!isfinite(cx) || !isfinite(cy) || !isfinite(cz) || !isfinite(w) || !isfinite(x) ||
      !isfinite(y) || !isfinite(z))
    atomicMin(&err->bad_center, (int)i);
  {
    const float smax = fmaxf(sx, fmaxf(sy, sz)), smin = fminf(sx, fminf(sy, sz));
    const float smid = sx + sy + sz - smax - smin;
    const bool core = scale_ok && M >= kOpaqueCoreTau * 6.28318531f * smid * smax;
    const unsigned am = __activemask();
    const unsigned cm = __ballot_sync(am, core);
    if (cm && (int)(threadIdx.x & 31) == __ffs(am) - 1) atomicAdd(&err->opaque_cores, (unsigned)__popc(cm));
  }
  // Primitive ctor (primitive.h:80-87): rcp_scale, density_norm_factor, inv_cdf_factor.
  const float rx = __fdiv_rn(1.0f, sx), ry = __fdiv_rn(1.0f, sy), rz = __fdiv_rn(1.0f, sz);
  const float dnf = __fmul_rn(0.0634936359f, __fmul_rn(__fmul_rn(rx, ry), rz));
  const float icf = __fmul_rn(__fmul_rn(M, dnf), 1.2533141373f);
  // Forward rotation matrix R(q) (include/thesis/host/utils/math.h:52-97 without scale) as float
  // pairs: each product of two quaternion components is exact as a TwoProduct pair, so every
  // entry carries ~44 bits, and W = diag(rcp_scale) R^T is rounded to FP32 once.
  auto sq2 = [](float a, float b, float c, float d, float sgn) {  // a*b + sgn*c*d as a float pair
    float p, pe, q, qe, s, se;
    two_prod(a, b, p, pe);
    two_prod(c, d, q, qe);
    if (sgn < 0.f) q = -q, qe = -qe;
    two_sum(p, q, s, se);
    FF r;
    fast_two_sum(s, __fadd_rn(se, __fadd_rn(pe, qe)), r.hi, r.lo);
    return r;
  };
  auto one_minus_2 = [](FF v) {  // 1 - 2 v
    float s, se;
    two_sum(1.0f, -2.0f * v.hi, s, se);
    FF r;
    fast_two_sum(s, __fsub_rn(se, 2.0f * v.lo), r.hi, r.lo);
    return r;
  };
  auto twice = [](FF v) { return FF{2.0f * v.hi, 2.0f * v.lo}; };
  FF R[3][3];
  R[0][0] = one_minus_2(sq2(y, y, z, z, 1.f));
  R[0][1] = twice(sq2(x, y, w, z, -1.f));
  R[0][2] = twice(sq2(x, z, w, y, 1.f));
  R[1][0] = twice(sq2(x, y, w, z, 1.f));
  R[1][1] = one_minus_2(sq2(x, x, z, z, 1.f));
  R[1][2] = twice(sq2(y, z, w, x, -1.f));
  R[2][0] = twice(sq2(x, z, w, y, -1.f));
  R[2][1] = twice(sq2(y, z, w, x, 1.f));
  R[2][2] = one_minus_2(sq2(x, x, y, y, 1.f));
  const float rs[3] = {rx, ry, rz};
  const float ss[3] = {sx, sy, sz};
  float W[3][3];
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) {
      float p, pe;
      two_prod(rs[r], R[c][r].hi, p, pe);
      W[r][c] = __fadd_rn(p, __fmaf_rn(rs[r], R[c][r].lo, pe));
    }
  rec[4 * i + 0] = make_float4(cx, cy, cz, W[0][0]);
  rec[4 * i + 1] = make_float4(W[0][1], W[0][2], W[1][0], W[1][1]);
  rec[4 * i + 2] = make_float4(W[1][2], W[2][0], W[2][1], W[2][2]);
  rec[4 * i + 3] = make_float4(icf, ar, ag, ab);
  float e[3];
  const float cen[3] = {cx, cy, cz};
  for (int k = 0; k < 3; ++k) {
    const float a0 = R[k][0].hi * ss[0], a1 = R[k][1].hi * ss[1], a2 = R[k][2].hi * ss[2];
    // 3-sigma half extent along world axis k, padded (1e-5 relative, far above the few-ulp error
    // of this FP32 evaluation) so FP32 chord tests never escape it; the box is rounded outward.
    e[k] = __fadd_ru(__fmul_ru(3.0f * sqrtf(fmaf(a0, a0, fmaf(a1, a1, a2 * a2))), 1.0f + 1e-5f),
                     1e-7f * (1.0f + fabsf(cen[k])));
  }
  lo[i] = make_float4(__fsub_rd(cx, e[0]), __fsub_rd(cy, e[1]), __fsub_rd(cz, e[2]), 0.f);
  hi[i] = make_float4(__fadd_ru(cx, e[0]), __fadd_ru(cy, e[1]), __fadd_ru(cz, e[2]), 0.f);
}

__device__ __forceinline__ unsigned int f2ord(float f) {
  const unsigned int u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(unsigned int u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// Bounds of the Gaussian centres (Morton frame, as computeBounds in math.h:135-160) and of
// the 3-sigma boxes (scene bounds).
__global__ void k_bounds(uint32_t n, const float* __restrict__ mean, const float4* __restrict__ lo,
                         const float4* __restrict__ hi, unsigned int* __restrict__ out12) {
  float cmn[3] = {INFINITY, INFINITY, INFINITY}, cmx[3] = {-INFINITY, -INFINITY, -INFINITY};
  float bmn[3] = {INFINITY, INFINITY, INFINITY}, bmx[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    for (int k = 0; k < 3; ++k) {
      const float c = mean[3 * i + k];
      cmn[k] = fminf(cmn[k], c);
      cmx[k] = fmaxf(cmx[k], c);
    }
    const float4 l = lo[i], h = hi[i];
    bmn[0] = fminf(bmn[0], l.x); bmn[1] = fminf(bmn[1], l.y); bmn[2] = fminf(bmn[2], l.z);
    bmx[0] = fmaxf(bmx[0], h.x); bmx[1] = fmaxf(bmx[1], h.y); bmx[2] = fmaxf(bmx[2], h.z);
  }
  for (int k = 0; k < 3; ++k) {
    for (int o = 16; o > 0; o >>= 1) {
      cmn[k] = fminf(cmn[k], __shfl_xor_sync(0xFFFFFFFFu, cmn[k], o));
      cmx[k] = fmaxf(cmx[k], __shfl_xor_sync(0xFFFFFFFFu, cmx[k], o));
      bmn[k] = fminf(bmn[k], __shfl_xor_sync(0xFFFFFFFFu, bmn[k], o));
      bmx[k] = fmaxf(bmx[k], __shfl_xor_sync(0xFFFFFFFFu, bmx[k], o));
    }
  }
  if ((threadIdx.x & 31) == 0) {
    for (int k = 0; k < 3; ++k) {
      atomicMin(&out12[k], f2ord(cmn[k]));
      atomicMax(&out12[3 + k], f2ord(cmx[k]));
      atomicMin(&out12[6 + k], f2ord(bmn[k]));
      atomicMax(&out12[9 + k], f2ord(bmx[k]));
    }
  }
}

__device__ __forceinline__ uint64_t expand21(uint64_t v) {  // 21 bits -> every third of 63
  v &= 0x1FFFFFull;
  v = (v | (v << 32)) & 0x1F00000000FFFFull;
  v = (v | (v << 16)) & 0x1F0000FF0000FFull;
  v = (v | (v << 8)) & 0x100F00F00F00F00Full;
  v = (v | (v << 4)) & 0x10C30C30C30C30C3ull;
  v = (v | (v << 2)) & 0x1249249249249249ull;
  return v;
}

// 63-bit Morton code of each centre (21 bits per axis; the reference uses 10 bits per axis on
// the host, math.h:117-131 -- more bits keep 2M-Gaussian scenes from collapsing into shared
// codes).
__global__ void k_morton(uint32_t n, const float* __restrict__ mean, const unsigned int* __restrict__ b,
                         uint64_t* __restrict__ codes, uint32_t* __restrict__ idx) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint64_t code = 0;
  for (int k = 0; k < 3; ++k) {
    const float mn = ord2f(b[k]), mx = ord2f(b[3 + k]);
    const float inv = 1.0f / fmaxf(mx - mn, 1e-30f);
    const float t = fminf(fmaxf((mean[3 * i + k] - mn) * inv, 0.0f), 1.0f);
    const uint64_t q = (uint64_t)(t * 2097151.0f);
    code |= expand21(q) << k;  // x lowest bit, then y, then z (math.h:128)
  }
  codes[i] = code;
  idx[i] = i;
}

// Records and 3-sigma boxes in scene order (order[i] = caller index of scene position i).
__global__ void k_gather(uint32_t n, const uint32_t* __restrict__ order, const float4* __restrict__ rec_in,
                         const float4* __restrict__ lo_in, const float4* __restrict__ hi_in,
                         float4* __restrict__ rec_out, float4* __restrict__ pbox) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t s = order[i];
  for (int k = 0; k < 4; ++k) rec_out[4 * i + k] = rec_in[4 * s + k];
  pbox[2 * i] = lo_in[s];
  pbox[2 * i + 1] = hi_in[s];
}

// 3-sigma boxes in Morton order: the input of both tree builders.
__global__ void k_gather_boxes(uint32_t n, const uint32_t* __restrict__ order, const float4* __restrict__ lo_in,
                               const float4* __restrict__ hi_in, float4* __restrict__ lo_out,
                               float4* __restrict__ hi_out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t s = order[i];
  lo_out[i] = make_float4(lo_in[s].x, lo_in[s].y, lo_in[s].z, 0.f);
  hi_out[i] = make_float4(hi_in[s].x, hi_in[s].y, hi_in[s].z, 0.f);
}

__global__ void k_gather_raw(uint32_t n, const uint32_t* __restrict__ order, const float* __restrict__ scale,
                             const float* __restrict__ quat, const float* __restrict__ density,
                             float4* __restrict__ raw) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t s = order[i];
  raw[2 * i] = make_float4(quat[4 * s], quat[4 * s + 1], quat[4 * s + 2], quat[4 * s + 3]);
  raw[2 * i + 1] = make_float4(scale[3 * s], scale[3 * s + 1], scale[3 * s + 2], density[s]);
}

__device__ __forceinline__ int karras_delta(const uint64_t* __restrict__ codes, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  const uint64_t a = codes[i], b = codes[j];
  if (a == b) return 64 + __clz(i ^ j);
  return __clzll(a ^ b);
}

// Karras 2012 ("Maximizing parallelism in the construction of BVHs, octrees, and k-d trees"):
// one thread per internal node of the binary radix tree over the sorted codes.
__global__ void k_karras(int n, const uint64_t* __restrict__ codes, uint32_t* __restrict__ left,
                         uint32_t* __restrict__ right, uint32_t* __restrict__ first,
                         uint32_t* __restrict__ last, uint32_t* __restrict__ parent_int,
                         uint32_t* __restrict__ parent_leaf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  const int d = (karras_delta(codes, n, i, i + 1) - karras_delta(codes, n, i, i - 1)) >= 0 ? 1 : -1;
  const int dmin = karras_delta(codes, n, i, i - d);
  int lmax = 2;
  while (karras_delta(codes, n, i, i + lmax * d) > dmin) lmax <<= 1;
  int l = 0;
  for (int t = lmax >> 1; t >= 1; t >>= 1)
    if (karras_delta(codes, n, i, i + (l + t) * d) > dmin) l += t;
  const int j = i + l * d;
  const int dnode = karras_delta(codes, n, i, j);
  int s = 0, t = l;
  do {
    t = (t + 1) >> 1;
    if (karras_delta(codes, n, i, i + (s + t) * d) > dnode) s += t;
  } while (t > 1);
  const int gamma = i + s * d + min(d, 0);
  const int lo_i = min(i, j), hi_i = max(i, j);
  uint32_t lref, rref;
  if (lo_i == gamma) {
    lref = kLeafBit | (uint32_t)gamma;
    parent_leaf[gamma] = i;
  } else {
    lref = (uint32_t)gamma;
    parent_int[gamma] = i;
  }
  if (hi_i == gamma + 1) {
    rref = kLeafBit | (uint32_t)(gamma + 1);
    parent_leaf[gamma + 1] = i;
  } else {
    rref = (uint32_t)(gamma + 1);
    parent_int[gamma + 1] = i;
  }
  left[i] = lref;
  right[i] = rref;
  first[i] = lo_i;
  last[i] = hi_i;
}

// Box of a binary-tree child and the number of Gaussians under it (internal nodes keep the count
// in hi.w).
__device__ __forceinline__ uint32_t child_box(uint32_t ref, const float4* plo, const float4* phi,
                                              const float4* nlo, const float4* nhi, float4& l, float4& h) {
  if (ref_is_leaf(ref)) {
    const uint32_t p = ref & ~kLeafBit;
    l = plo[p];
    h = phi[p];
    return 1u;
  }
  l = __ldcg(nlo + ref);
  h = __ldcg(nhi + ref);
  return __float_as_uint(h.w);
}

// Bottom-up refit: the second thread to reach an internal node unions its children.
__global__ void k_refit(int n, const uint32_t* __restrict__ left, const uint32_t* __restrict__ right,
                        const uint32_t* __restrict__ parent_int, const uint32_t* __restrict__ parent_leaf,
                        const float4* __restrict__ plo, const float4* __restrict__ phi,
                        float4* nlo, float4* nhi, unsigned int* flags) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n || n < 2) return;
  uint32_t node = parent_leaf[k];
  while (true) {
    __threadfence();
    if (atomicAdd(&flags[node], 1u) == 0u) return;
    __threadfence();
    float4 al, ah, bl, bh;
    const uint32_t ca = child_box(left[node], plo, phi, nlo, nhi, al, ah);
    const uint32_t cb = child_box(right[node], plo, phi, nlo, nhi, bl, bh);
    __stcg(nlo + node, make_float4(fminf(al.x, bl.x), fminf(al.y, bl.y), fminf(al.z, bl.z), 0.f));
    __stcg(nhi + node, make_float4(fmaxf(ah.x, bh.x), fmaxf(ah.y, bh.y), fmaxf(ah.z, bh.z), __uint_as_float(ca + cb)));
    if (node == 0u) return;
    node = parent_int[node];
  }
}

// Binary-LBVH node records for the thread-per-ray megakernel: (l_lo, l_hi, r_lo, r_hi), child
// refs in l_lo.w / r_lo.w (leaf bit | scene-order Gaussian index: pos maps Morton order to it).
__global__ void k_binary_nodes(int n, const uint32_t* __restrict__ left, const uint32_t* __restrict__ right,
                               const float4* __restrict__ plo, const float4* __restrict__ phi,
                               const float4* __restrict__ nlo, const float4* __restrict__ nhi,
                               const uint32_t* __restrict__ pos, float4* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  auto scene_ref = [&](uint32_t r) { return ref_is_leaf(r) ? (kLeafBit | pos[r & ~kLeafBit]) : r; };
  float4 al, ah, bl, bh;
  child_box(left[i], plo, phi, nlo, nhi, al, ah);
  child_box(right[i], plo, phi, nlo, nhi, bl, bh);
  al.w = __uint_as_float(scene_ref(left[i]));
  bl.w = __uint_as_float(scene_ref(right[i]));
  ah.w = 0.f;
  bh.w = 0.f;
  out[4 * i + 0] = al;
  out[4 * i + 1] = ah;
  out[4 * i + 2] = bl;
  out[4 * i + 3] = bh;
}

// ------------------------------------------------------------------------------------------
// PLOC: Meister & Bittner, "Parallel Locally-Ordered Clustering for Bounding Volume Hierarchy
// Construction" (IEEE TVCG 2018).  Clusters start as the Morton-sorted Gaussian boxes; every pass,
// each cluster finds the neighbour within kPlocRadius positions whose union box has the smallest
// surface area, mutual nearest neighbours merge into a new binary node (at the lower position),
// and the cluster array is compacted in order.  Node ids are handed out in merge order, so the
// root is node n - 2.
// ------------------------------------------------------------------------------------------
constexpr int kPlocRadius = 32;
constexpr int kPlocBlock = 256;

// A cluster is (lo.xyz, ref bits in lo.w) and (hi.xyz, Gaussian count bits in hi.w); refs are
// binary node ids or kLeafBit | Morton position.
__global__ void k_ploc_init(uint32_t n, const float4* __restrict__ plo, const float4* __restrict__ phi,
                            float4* __restrict__ cl, float4* __restrict__ ch) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 l = plo[i], h = phi[i];
  l.w = __uint_as_float(kLeafBit | i);
  h.w = __uint_as_float(1u);
  cl[i] = l;
  ch[i] = h;
}

// Surface area of the union of two boxes; the same value whichever box comes first, and NaN
// (from non-finite extents) ordered as +inf, so the pair order below is a total order and the
// globally smallest pair is always mutual (every pass merges at least once).
__device__ __forceinline__ float union_area(float4 al, float4 ah, float4 bl, float4 bh) {
  const float dx = fmaxf(ah.x, bh.x) - fminf(al.x, bl.x);
  const float dy = fmaxf(ah.y, bh.y) - fminf(al.y, bl.y);
  const float dz = fmaxf(ah.z, bh.z) - fminf(al.z, bl.z);
  const float a = 2.f * (dx * dy + dy * dz + dz * dx);
  return a == a ? a : INFINITY;
}

// The nearest neighbour of the cluster at tile position c (array position i of m): the pair order is area,
// then buddy pairs (2k, 2k + 1) first -- so equal boxes pair up in halves instead of chaining -- then the
// pair's lower position, then its upper position.
__device__ __forceinline__ int ploc_nearest(const float4* sl, const float4* sh, int c, int i, int m) {
  const float4 al = sl[c], ah = sh[c];
  float best = INFINITY;
  int bj = -1;
  for (int k = -kPlocRadius; k <= kPlocRadius; ++k) {
    const int j = i + k;
    if (k == 0 || j < 0 || j >= m) continue;
    const float a = union_area(al, ah, sl[c + k], sh[c + k]);
    bool take = bj < 0 || a < best;
    if (!take && a == best) {
      const int lo_new = min(i, j), lo_old = min(i, bj);
      const bool bud_new = !(lo_new & 1) && max(i, j) == lo_new + 1;
      const bool bud_old = !(lo_old & 1) && max(i, bj) == lo_old + 1;
      take = (bud_new != bud_old) ? bud_new
                                  : (lo_new < lo_old || (lo_new == lo_old && max(i, j) < max(i, bj)));
    }
    if (take) {
      best = a;
      bj = j;
    }
  }
  return bj;
}

// A merge of clusters (l, h) and (bl, bh) as binary node `node` (Gaussian count in nhi.w, height in nlo.w);
// l, h become the new cluster.
__device__ __forceinline__ void ploc_make_node(uint32_t node, float4& l, float4& h, float4 bl, float4 bh,
                                               uint32_t* left, uint32_t* right, float4* nlo, float4* nhi) {
  const uint32_t lref = __float_as_uint(l.w), rref = __float_as_uint(bl.w);
  left[node] = lref;
  right[node] = rref;
  // the children were made in earlier passes; heights of leaf references are 0
  const uint32_t hl = ref_is_leaf(lref) ? 0u : __float_as_uint(nlo[lref].w);
  const uint32_t hr = ref_is_leaf(rref) ? 0u : __float_as_uint(nlo[rref].w);
  l = make_float4(fminf(l.x, bl.x), fminf(l.y, bl.y), fminf(l.z, bl.z), __uint_as_float(node));
  h = make_float4(fmaxf(h.x, bh.x), fmaxf(h.y, bh.y), fmaxf(h.z, bh.z),
                  __uint_as_float(__float_as_uint(h.w) + __float_as_uint(bh.w)));
  nlo[node] = make_float4(l.x, l.y, l.z, __uint_as_float(1u + max(hl, hr)));
  nhi[node] = h;
}

// A pass is two launches, which take the live state from ctr_in = (clusters, nodes made so far, passes), so a
// run of passes needs no host round trip (grids cover an upper bound):
//   k_ploc_pair   nearest neighbours of a tile and of the kPlocRadius clusters on either side of it, so that
//                 mutual pairs are known in the block; counts of the tile's merges and kept clusters
//   k_ploc_merge  every tile's output position from the counts before it, the merged nodes, the compacted
//                 clusters
// (one launch each for neighbours, flags, three of a scan, and the write took 6 a pass, 8 ms of a 500k build's
// 13).  Once at most kPlocTail clusters are left, passes only carry them over and k_ploc_tail finishes.
constexpr uint32_t kPlocTail = 1024;
constexpr uint32_t kPlocSuper = 64;  // tiles a second-level count covers

// Counts are merges << 32 | kept.  The lower cluster of a mutual pair makes the node and keeps its position;
// the upper one is absorbed.
__global__ void __launch_bounds__(kPlocBlock + 2 * kPlocRadius) k_ploc_pair(
    const uint32_t* __restrict__ ctr_in, const float4* __restrict__ cl, const float4* __restrict__ ch,
    uint32_t* __restrict__ nn, unsigned long long* __restrict__ tile_count, unsigned long long* super_count) {
  constexpr int kHalo = 2 * kPlocRadius, kSpan = kPlocBlock + 2 * kHalo;
  __shared__ float4 sl[kSpan], sh[kSpan];
  __shared__ int snn[kPlocBlock + kHalo];
  __shared__ unsigned long long total;
  const uint32_t m = ctr_in[0];
  if (m <= kPlocTail) return;
  const int b0 = (int)(blockIdx.x * kPlocBlock);
  if (b0 >= (int)m) return;
  for (int k = threadIdx.x; k < kSpan; k += blockDim.x) {
    const int g = b0 - kHalo + k;
    if (g >= 0 && g < (int)m) {
      sl[k] = cl[g];
      sh[k] = ch[g];
    }
  }
  if (threadIdx.x == 0) total = 0ull;
  __syncthreads();
  const int t = (int)threadIdx.x, i = b0 - kPlocRadius + t;
  const bool in = i >= 0 && i < (int)m;
  const int j = in ? ploc_nearest(sl, sh, t + kPlocRadius, i, (int)m) : -1;
  snn[t] = j;
  __syncthreads();
  unsigned long long f = 0ull;
  if (in && t >= kPlocRadius && t < kPlocRadius + kPlocBlock) {
    nn[i] = (uint32_t)j;
    const bool mutual = snn[j - (b0 - kPlocRadius)] == i;
    f = ((mutual && i < j) ? 1ull << 32 : 0ull) | ((mutual && i > j) ? 0ull : 1ull);
  }
  for (int o = 16; o > 0; o >>= 1) f += __shfl_xor_sync(0xFFFFFFFFu, f, o);
  if ((threadIdx.x & 31) == 0 && f) atomicAdd(&total, f);
  __syncthreads();
  if (threadIdx.x == 0) {
    tile_count[blockIdx.x] = total;
    atomicAdd(super_count + blockIdx.x / kPlocSuper, total);
  }
}

// Exclusive block-wide prefix sum over kPlocBlock threads of counts; warp_tot: 32 entries.
__device__ __forceinline__ unsigned long long ploc_scan(unsigned long long v, unsigned long long* warp_tot) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  unsigned long long incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long x = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) warp_tot[w] = incl;
  __syncthreads();
  if (w == 0) {
    unsigned long long x = lane < nw ? warp_tot[lane] : 0ull;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (lane >= o) x += y;
    }
    warp_tot[lane] = x;
  }
  __syncthreads();
  return incl - v + (w ? warp_tot[w - 1] : 0ull);
}

__global__ void __launch_bounds__(kPlocBlock) k_ploc_merge(
    const uint32_t* __restrict__ ctr_in, uint32_t* __restrict__ ctr_out, const uint32_t* __restrict__ nn,
    const unsigned long long* __restrict__ tile_count, const unsigned long long* __restrict__ super_count,
    unsigned long long* __restrict__ super_next, uint32_t n_super, const float4* __restrict__ cl,
    const float4* __restrict__ ch, float4* __restrict__ ol, float4* __restrict__ oh, uint32_t* __restrict__ left,
    uint32_t* __restrict__ right, float4* __restrict__ nlo, float4* __restrict__ nhi) {
  __shared__ unsigned long long warp_tot[32];
  __shared__ unsigned long long before;
  const uint32_t m = ctr_in[0], node_base = ctr_in[1];
  const uint32_t i = blockIdx.x * kPlocBlock + threadIdx.x;
  for (uint32_t k = i; k < n_super; k += gridDim.x * kPlocBlock) super_next[k] = 0ull;
  if (m <= kPlocTail) {  // carried over for k_ploc_tail
    if (i < m) {
      ol[i] = cl[i];
      oh[i] = ch[i];
    }
    if (i < 3u) ctr_out[i] = ctr_in[i];
    return;
  }
  if (blockIdx.x * kPlocBlock >= m) return;
  if (threadIdx.x == 0) before = 0ull;
  __syncthreads();
  {
    const uint32_t s = blockIdx.x / kPlocSuper;
    unsigned long long v = 0ull;
    for (uint32_t k = threadIdx.x; k < s; k += kPlocBlock) v += super_count[k];
    const uint32_t t = s * kPlocSuper + threadIdx.x;
    if (threadIdx.x < kPlocSuper && t < blockIdx.x) v += tile_count[t];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&before, v);
  }
  __syncthreads();
  uint32_t j = 0;
  unsigned long long f = 0ull;
  if (i < m) {
    j = nn[i];
    const bool mutual = nn[j] == i;
    f = ((mutual && i < j) ? 1ull << 32 : 0ull) | ((mutual && i > j) ? 0ull : 1ull);
  }
  const unsigned long long x = before + ploc_scan(f, warp_tot);
  if (i >= m) return;
  if (i == m - 1u) {
    ctr_out[0] = (uint32_t)(x + f);
    ctr_out[1] = node_base + (uint32_t)((x + f) >> 32);
    ctr_out[2] = ctr_in[2] + 1u;
  }
  if (!(f & 1ull)) return;
  float4 l = cl[i], h = ch[i];
  if (f >> 32) ploc_make_node(node_base + (uint32_t)(x >> 32), l, h, cl[j], ch[j], left, right, nlo, nhi);
  const uint32_t p = (uint32_t)x;
  ol[p] = l;
  oh[p] = h;
}

// All remaining passes over at most kPlocTail clusters, in one block: about half of a build's passes, which
// as launches cost more than their work.  ctr = (clusters, nodes, passes), at most max_passes in all; ctr[3]
// receives the finished tree's height.
__global__ void __launch_bounds__(kPlocTail) k_ploc_tail(uint32_t* __restrict__ ctr, uint32_t max_passes,
                                                         const float4* __restrict__ cl, const float4* __restrict__ ch,
                                                         uint32_t* left, uint32_t* right, float4* nlo, float4* nhi) {
  __shared__ float4 sl[kPlocTail], sh[kPlocTail];
  __shared__ int snn[kPlocTail];
  __shared__ unsigned long long warp_tot[32];
  uint32_t m = ctr[0], nodes = ctr[1], passes = ctr[2];
  if (m > kPlocTail || m < 2u) return;
  const int i = (int)threadIdx.x;
  if (i < (int)m) {
    sl[i] = cl[i];
    sh[i] = ch[i];
  }
  __syncthreads();
  while (m > 1u && passes < max_passes) {
    const bool in = i < (int)m;
    const int j = in ? ploc_nearest(sl, sh, i, i, (int)m) : -1;
    snn[i] = j;
    __syncthreads();
    unsigned long long f = 0ull;
    float4 l, h, bl, bh;
    if (in) {
      const bool mutual = snn[j] == i;
      f = ((mutual && i < j) ? 1ull << 32 : 0ull) | ((mutual && i > j) ? 0ull : 1ull);
      l = sl[i], h = sh[i], bl = sl[j], bh = sh[j];
    }
    const unsigned long long x = ploc_scan(f, warp_tot);  // (two barriers: the reads above are done)
    const unsigned long long total = warp_tot[31];
    if (f & 1ull) {
      if (f >> 32) ploc_make_node(nodes + (uint32_t)(x >> 32), l, h, bl, bh, left, right, nlo, nhi);
      sl[(uint32_t)x] = l;
      sh[(uint32_t)x] = h;
    }
    m = (uint32_t)total;
    nodes += (uint32_t)(total >> 32);
    ++passes;
    __syncthreads();
  }
  if (i == 0) {
    ctr[0] = m;
    ctr[1] = nodes;
    ctr[2] = passes;
    ctr[3] = m == 1u ? __float_as_uint(nlo[nodes - 1u].w) : 0u;
  }
}

// How much of the scene its Gaussians fill: with w the sides of a Gaussian's 3-sigma box and s those of the evenly
// filled box that has the centres' spread, the mean over the Gaussians and the three faces of the product of
// w / (w + s) along two axes -- about the share of them that a ray through the middle meets.  1: all in one place; 0.06:
// scales of 0.1 in a box of side 2; 0.01 and 0.03 in the value-noise cloud and the dense clusters.  From at most
// kOverlapSamples of them, evenly spaced in the caller's order, by one block.
constexpr uint32_t kOverlapSamples = 4096;
__global__ void __launch_bounds__(1024) k_overlap(uint32_t n, const float* __restrict__ mean, const float4* __restrict__ lo,
                                                  const float4* __restrict__ hi, ErrorWords* __restrict__ err) {
  __shared__ double part[32][6];
  __shared__ double total[6];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  auto block_sums = [&](double (&v)[6]) {  // on every thread
    for (int q = 0; q < 6; ++q) {
      v[q] = warp_sum(v[q]);
      if (lane == 0u) part[warp][q] = v[q];
    }
    __syncthreads();
    if (warp == 0u)
      for (int q = 0; q < 6; ++q) {
        const double t = warp_sum(part[lane][q]);
        if (lane == 0u) total[q] = t;
      }
    __syncthreads();
    for (int q = 0; q < 6; ++q) v[q] = total[q];
  };
  const uint32_t m = min(n, kOverlapSamples);
  auto sample = [&](uint32_t k) { return (uint32_t)((uint64_t)k * n / m); };
  const float3 at = f3(mean[0], mean[1], mean[2]);  // (relative to the first centre: the spread of a far scene)
  double c[6] = {};
  for (uint32_t k = threadIdx.x; k < m; k += 1024u) {
    const uint32_t i = sample(k);
    const double x = mean[3 * i] - at.x, y = mean[3 * i + 1] - at.y, z = mean[3 * i + 2] - at.z;
    c[0] += x, c[1] += y, c[2] += z, c[3] += x * x, c[4] += y * y, c[5] += z * z;
  }
  block_sums(c);
  float s[3];
  for (int a = 0; a < 3; ++a) s[a] = (float)sqrt(12.0 * fmax(c[3 + a] / m - (c[a] / m) * (c[a] / m), 0.0));
  double f[6] = {};
  for (uint32_t k = threadIdx.x; k < m; k += 1024u) {
    const uint32_t i = sample(k);
    const float4 l = lo[i], h = hi[i];
    const float x = (h.x - l.x) / (h.x - l.x + s[0]), y = (h.y - l.y) / (h.y - l.y + s[1]),
                z = (h.z - l.z) / (h.z - l.z + s[2]);
    f[0] += x * y + y * z + z * x;
  }
  block_sums(f);
  if (threadIdx.x == 0u) err->overlap = (float)(f[0] / (3.0 * m));
}

struct CollapseItem {
  uint32_t bin;     // binary internal node to expand
  uint32_t slot;    // BVH32 node slot it becomes
  uint32_t offset;  // scene position of its first Gaussian (depth-first leaf order)
  uint32_t pad;
};

__device__ __forceinline__ float box_area(float4 l, float4 h) {
  const float dx = fmaxf(h.x - l.x, 0.f), dy = fmaxf(h.y - l.y, 0.f), dz = fmaxf(h.z - l.z, 0.f);
  return 2.f * (dx * dy + dy * dz + dz * dx);
}

__device__ __forceinline__ uint32_t ref_count(uint32_t r, const float4* __restrict__ nhi) {
  return ref_is_leaf(r) ? 1u : __float_as_uint(nhi[r].w);
}

// ------------------------------------------------------------------------------------------
// SAH-optimal collapse (the dynamic programme of Ylitie, Karras & Laine, "Efficient Incoherent Ray
// Traversal on GPUs Through Compressed Wide BVHs", HPG 2017, with 32 slots per node).  For each
// binary node v and slot budget i, C(v, i) is the least expected traversal cost of representing
// v's subtree with at most i child slots of the enclosing BVH32 node:
//   C(v, 1) = min(leaf: A(v) (c_leaf + c_box n(v)) if n(v) <= leaf_max,  node: A(v) c_node + D(v, 32))
//   D(v, i) = min over 2 <= k <= i, 1 <= j < k of C(left, j) + C(right, k - j)
//   C(v, i) = min(C(v, 1), D(v, i))
// with A the surface area.  A Gaussian is a leaf of cost A (c_leaf + c_box).  The costs weigh an
// inner-node step against a leaf range (leaf packing shares warp steps between ranges) and a box
// test: c_node = 1, c_leaf = 0.5, c_box = 0.05 (measured on the showcase: c_leaf 0.3 or 1.0 and
// c_box 0.02 are within 0.3 %).
// ------------------------------------------------------------------------------------------
constexpr float kDpNode = 1.0f, kDpLeaf = 0.5f, kDpBox = 0.05f;

struct DpTables {
  float* cost;       // [ni * 32]: C(v, i) at v * 32 + i - 1
  uint8_t* split;    // [ni * 32]: j of the best split into exactly i slots
  uint8_t* best;     // [ni * 32]: the k <= i of D(v, i)
  uint32_t* single;  // [ni]: bit i - 1 set when C(v, i) uses one slot
  uint8_t* leaf;     // [ni]: the one slot of C(v, 1) is a leaf
};

// Parent links of a binary tree (internal children in parent[], Gaussians in parent_leaf[]).
__global__ void k_parents(uint32_t ni, const uint32_t* __restrict__ left, const uint32_t* __restrict__ right,
                          uint32_t* __restrict__ parent, uint32_t* __restrict__ parent_leaf) {
  const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= ni) return;
  const uint32_t c[2] = {left[v], right[v]};
  for (int k = 0; k < 2; ++k) {
    if (ref_is_leaf(c[k])) parent_leaf[c[k] & ~kLeafBit] = v;
    else parent[c[k]] = v;
  }
}

// Bottom-up.  A warp starts at 32 Gaussians, each lane climbing from its own; the second arrival at a node
// owns it, and the warp computes the nodes its lanes own one after another with lane i holding the costs for
// i + 1 slots: the 496 sums of D(v, .) are 31 shuffled steps.  (A thread per node keeps three 32-entry arrays
// in local memory: 1.44 ms for 250k Gaussians against 0.16.)
__global__ void __launch_bounds__(256) k_dp_cost(uint32_t n, uint32_t root, const uint32_t* __restrict__ left,
                          const uint32_t* __restrict__ right, const float4* __restrict__ plo,
                          const float4* __restrict__ phi, const float4* __restrict__ nlo,
                          const float4* __restrict__ nhi, const uint32_t* __restrict__ parent,
                          const uint32_t* __restrict__ parent_leaf, unsigned int* flags, DpTables T,
                          uint32_t leaf_max) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  constexpr uint32_t kDone = 0xFFFFFFFFu;
  constexpr unsigned kAll = 0xFFFFFFFFu;
  uint32_t v = k < n ? parent_leaf[k] : kDone;
  auto child_cost = [&](uint32_t ref) -> float {
    if (ref_is_leaf(ref)) {
      const uint32_t p = ref & ~kLeafBit;
      return box_area(plo[p], phi[p]) * (kDpLeaf + kDpBox);
    }
    return __ldcg(T.cost + (size_t)ref * 32u + lane);
  };
  while (true) {
    __threadfence();
    const bool mine = v != kDone && atomicAdd(&flags[v], 1u) != 0u;
    __threadfence();
    unsigned todo = __ballot_sync(kAll, mine);
    if (todo == 0u) return;
    for (unsigned r = todo; r != 0u; r &= r - 1u) {
      const uint32_t u = __shfl_sync(kAll, v, __ffs(r) - 1);
      const float Cl = child_cost(left[u]), Cr = child_cost(right[u]);
      float b = INFINITY;
      uint32_t bj = 1;
      for (int j = 1; j < 32; ++j) {  // D(u, lane + 1) over splits j, lane + 1 - j
        const float c = __shfl_sync(kAll, Cl, j - 1) + __shfl_sync(kAll, Cr, (lane - j) & 31);
        if (lane >= j && c < b) {
          b = c;
          bj = (uint32_t)j;
        }
      }
      // least over at most that many slots, the fewest on ties
      uint32_t bk = lane == 0 ? 2u : (uint32_t)lane + 1u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float ob = __shfl_up_sync(kAll, b, o);
        const uint32_t ok = __shfl_up_sync(kAll, bk, o);
        if (lane >= o + 1 && ob <= b) {
          b = ob;
          bk = ok;
        }
      }
      const float D32 = __shfl_sync(kAll, b, 31);
      const float4 l = nlo[u], h = nhi[u];
      const float A = box_area(l, h);
      const uint32_t count = __float_as_uint(h.w);
      const float c_node = fmaf(A, kDpNode, D32);
      const float c_leaf = count <= leaf_max ? A * fmaf(kDpBox, (float)count, kDpLeaf) : INFINITY;
      const float c1 = fminf(c_leaf, c_node);
      const bool one = lane == 0 || c1 <= b;
      const unsigned mask = __ballot_sync(kAll, one);
      __stcg(T.cost + (size_t)u * 32u + lane, one ? c1 : b);
      T.split[(size_t)u * 32u + lane] = (uint8_t)bj;
      T.best[(size_t)u * 32u + lane] = (uint8_t)bk;
      if (lane == 0) {
        T.single[u] = mask;
        T.leaf[u] = count <= leaf_max && c_leaf <= c_node ? 1 : 0;  // a leaf fits in one warp step
      }
    }
    __threadfence();
    __syncwarp();
    v = mine && v != root ? parent[v] : kDone;
  }
}

// Collapse of a binary tree (Gaussian counts in nhi.w) into 32-wide nodes, level by level, a warp per node:
//  - greedy (kDp false): starting from the binary node's two children, repeatedly replace the
//    largest-area child holding more than kLeafMax Gaussians by its two children until 32 slots
//    are used; children with <= kLeafMax Gaussians become leaves, larger ones the next level's
//    nodes;
//  - SAH-optimal (kDp true): replay the choices of k_dp_cost for a budget of 32 slots, all open
//    children of the node at once.
// Then lane c writes child c.  Every child carries the scene position of its first Gaussian in depth-first
// leaf order (left subtree first), so a leaf is one contiguous range of the scene order; pos[Morton position]
// receives each Gaussian's scene position.  The level's item count is read on the device
// (*n_items_dev), so levels run back to back with upper-bound grids.  Nodes beyond max_nodes are
// not written: the build then sees *overflow set and falls back to the greedy collapse.
// (A thread per node walks its up to 32 leaf subtrees one after another: 3.0 ms for 250k Gaussians
// against 0.2.)
template <bool kDp>
__global__ void __launch_bounds__(128) k_collapse(const unsigned int* __restrict__ n_items_dev, const CollapseItem* __restrict__ in,
                           CollapseItem* __restrict__ out, unsigned int* __restrict__ out_count,
                           unsigned int* __restrict__ slot_counter, const uint32_t* __restrict__ left,
                           const uint32_t* __restrict__ right, const float4* __restrict__ plo,
                           const float4* __restrict__ phi, const float4* __restrict__ nlo,
                           const float4* __restrict__ nhi, float4* __restrict__ wide, uint32_t kLeafMax,
                           uint32_t* __restrict__ pos, unsigned int* __restrict__ leaf_counter, DpTables T,
                           uint32_t max_nodes, unsigned int* __restrict__ overflow) {
  __shared__ uint32_t s_ref[4][32], s_off[4][32], s_bud[4][32];
  constexpr unsigned kAll = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const uint32_t n_items = *n_items_dev;
  for (uint32_t t = blockIdx.x * 4u + (uint32_t)w; t < n_items; t += gridDim.x * 4u) {
  const CollapseItem it = in[t];
  // lane c < cnt: the c-th child so far (reference, slot budget, offset), in depth-first order
  uint32_t v = 0, bud = 0, off = 0;
  int cnt = 2;
  {
    const uint32_t l = left[it.bin];
    uint32_t kk = 0, j = 0;
    if constexpr (kDp) {
      kk = T.best[(size_t)it.bin * 32u + 31u];
      j = T.split[(size_t)it.bin * 32u + kk - 1u];
    }
    if (lane == 0) v = l, bud = j, off = it.offset;
    if (lane == 1) v = right[it.bin], bud = kk - j, off = it.offset + ref_count(l, nhi);
  }
  bool leaf = false;
  if constexpr (kDp) {
    while (true) {
      const bool on = lane < cnt;
      const bool open = on && !ref_is_leaf(v) && bud != 1u && !((T.single[v] >> (bud - 1u)) & 1u);
      const unsigned om = __ballot_sync(kAll, open);
      if (om == 0u) break;
      const int p = lane + __popc(om & lt);  // the budgets sum to at most 32, so the children fit the warp
      if (on && !open) {
        s_ref[w][p] = v, s_bud[w][p] = bud, s_off[w][p] = off;
      }
      if (open) {
        const uint32_t kk = T.best[(size_t)v * 32u + bud - 1u], j = T.split[(size_t)v * 32u + kk - 1u];
        const uint32_t l = left[v];
        s_ref[w][p] = l, s_bud[w][p] = j, s_off[w][p] = off;
        s_ref[w][p + 1] = right[v], s_bud[w][p + 1] = kk - j, s_off[w][p + 1] = off + ref_count(l, nhi);
      }
      cnt += __popc(om);
      __syncwarp();
      if (lane < cnt) v = s_ref[w][lane], bud = s_bud[w][lane], off = s_off[w][lane];
      __syncwarp();
    }
    leaf = lane < cnt && !ref_is_leaf(v) && T.leaf[v] != 0;
  } else {
    while (cnt < 32) {
      // the largest-area child above kLeafMax (the first of equals)
      float a = -1.f;
      if (lane < cnt && !ref_is_leaf(v) && ref_count(v, nhi) > kLeafMax) a = box_area(nlo[v], nhi[v]);
      float am = a;
      for (int o = 16; o > 0; o >>= 1) am = fmaxf(am, __shfl_xor_sync(kAll, am, o));
      const unsigned cand = __ballot_sync(kAll, a == am && a > -1.f);
      if (cand == 0u) break;
      const int src = __ffs(cand) - 1;
      const uint32_t r = __shfl_sync(kAll, v, src), o0 = __shfl_sync(kAll, off, src);
      const uint32_t l = left[r];
      if (lane == src) v = l;
      if (lane == cnt) v = right[r], off = o0 + ref_count(l, nhi);
      ++cnt;
    }
    leaf = lane < cnt && !ref_is_leaf(v) && ref_count(v, nhi) <= kLeafMax;
  }
  // lane c writes child c
  const bool on = lane < cnt;
  const bool single = on && ref_is_leaf(v), inner = on && !single && !leaf;
  const unsigned im = __ballot_sync(kAll, inner), lm = __ballot_sync(kAll, single || leaf);
  uint32_t slot0 = 0, q0 = 0;
  if (lane == 0) {
    if (im) slot0 = atomicAdd(slot_counter, (unsigned)__popc(im));
    if (lm) atomicAdd(leaf_counter, (unsigned)__popc(lm));
  }
  slot0 = __shfl_sync(kAll, slot0, 0);
  const bool fits = inner && slot0 + (uint32_t)__popc(im & lt) < max_nodes;
  const unsigned fm = __ballot_sync(kAll, fits);
  if (lane == 0 && fm) q0 = atomicAdd(out_count, (unsigned)__popc(fm));
  q0 = __shfl_sync(kAll, q0, 0);
  float4 l = make_float4(INFINITY, INFINITY, INFINITY, 0.f), h = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
  uint32_t wref = kEmptyRef;
  if (single) {
    const uint32_t p = v & ~kLeafBit;
    l = plo[p];
    h = phi[p];
    pos[p] = off;
    wref = wide_leaf_ref(off, 1u);
  } else if (on) {
    l = nlo[v];
    h = nhi[v];
    if (leaf) {
      wref = wide_leaf_ref(off, ref_count(v, nhi));
      // depth-first walk of the leaf's subtree (<= 32 Gaussians, so <= 32 stacked refs)
      uint32_t st[32];
      int sp = 0;
      uint32_t k = off;
      st[sp++] = v;
      while (sp > 0) {
        const uint32_t x = st[--sp];
        if (ref_is_leaf(x)) {
          pos[x & ~kLeafBit] = k++;
        } else {
          st[sp++] = right[x];
          st[sp++] = left[x];
        }
      }
    } else if (fits) {
      wref = slot0 + (uint32_t)__popc(im & lt);
      out[q0 + (uint32_t)__popc(fm & lt)] = CollapseItem{v, wref, off, 0u};
    } else {  // over the node budget: no write; the build falls back
      atomicOr(overflow, 1u);
    }
  }
  l.w = __uint_as_float(wref);
  h.w = 0.f;
  float4* node = wide + (size_t)it.slot * 64u;
  node[lane] = l;
  node[32 + lane] = h;
  }
}

// ------------------------------------------------------------------------------------------
// Compressed 8-wide BVH (vp_trace8.cuh): the same binary tree cut for 8 slots a node with every
// Gaussian a slot of its own.  The cut minimises the expected cost A (kDp8Node per node, kDp8Prim per
// Gaussian) over the tree by the same dynamic programme as above, with "at most i slots" costs
//   C(v, i) = min(C(v, i - 1), D(v, i)),  D(v, i) = min over 1 <= j < i of C(left, j) + C(right, i - j),
//   C(v, 1) = A(v) kDp8Node + D(v, 8).
// ------------------------------------------------------------------------------------------
constexpr float kDp8Node = 1.0f, kDp8Prim = 0.4f;

// Bottom-up, as k_dp_cost.  cost[8 v + i - 1] = C(v, i); choice[8 v + i - 1] = the j of D(v, i), or 0 for
// C(v, i - 1); choice[8 v] = the j of D(v, 8).
__global__ void k_dp8_cost(uint32_t n, uint32_t root, const uint32_t* __restrict__ left,
                           const uint32_t* __restrict__ right, const float4* __restrict__ plo,
                           const float4* __restrict__ phi, const float4* __restrict__ nlo,
                           const float4* __restrict__ nhi, const uint32_t* __restrict__ parent,
                           const uint32_t* __restrict__ parent_leaf, unsigned int* flags, float* cost,
                           uint8_t* __restrict__ choice) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  uint32_t v = parent_leaf[k];
  while (true) {
    __threadfence();
    if (atomicAdd(&flags[v], 1u) == 0u) return;
    __threadfence();
    float C[2][7];
    const uint32_t ch[2] = {left[v], right[v]};
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (ref_is_leaf(ch[c])) {
        const uint32_t p = ch[c] & ~kLeafBit;
        const float a = box_area(plo[p], phi[p]) * kDp8Prim;
#pragma unroll
        for (int i = 0; i < 7; ++i) C[c][i] = a;
      } else {
        const float4* q = reinterpret_cast<const float4*>(cost + 8ull * ch[c]);
        const float4 x = __ldcg(q), y = __ldcg(q + 1);
        C[c][0] = x.x, C[c][1] = x.y, C[c][2] = x.z, C[c][3] = x.w, C[c][4] = y.x, C[c][5] = y.y, C[c][6] = y.z;
      }
    }
    float out[8];
    uint32_t pick[8];
    float d8 = INFINITY;
#pragma unroll
    for (int i = 2; i <= 8; ++i) {
      float b = INFINITY;
      uint32_t bj = 1;
#pragma unroll
      for (int j = 1; j < i; ++j) {
        const float c = C[0][j - 1] + C[1][i - j - 1];
        if (c < b) {
          b = c;
          bj = (uint32_t)j;
        }
      }
      out[i - 1] = b;
      pick[i - 1] = bj;
      if (i == 8) d8 = b;
    }
    pick[0] = pick[7];
    out[0] = fmaf(box_area(nlo[v], nhi[v]), kDp8Node, d8);
#pragma unroll
    for (int i = 1; i < 8; ++i)
      if (out[i - 1] <= out[i]) {
        out[i] = out[i - 1];
        pick[i] = 0u;
      }
    float4* q = reinterpret_cast<float4*>(cost + 8ull * v);
    __stcg(q, make_float4(out[0], out[1], out[2], out[3]));
    __stcg(q + 1, make_float4(out[4], out[5], out[6], out[7]));
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) lo |= pick[i] << (8 * i), hi |= pick[4 + i] << (8 * i);
    reinterpret_cast<uint2*>(choice)[v] = make_uint2(lo, hi);
    if (v == root) return;
    v = parent[v];
  }
}

// Origin p < lo and power-of-two quantum q of a node's axis with every plane of [lo, hi] at p + k q,
// 0 < k < 254 (the exponent byte holds q with a +15 bias).  q grows where p, one quantum below lo, rounds
// further down than that.
__device__ __forceinline__ void frame8(float lo, float hi, float& p, float& q) {
  const uint32_t u = __float_as_uint((hi - lo) * (1.0f / 253.0f));
  uint32_t e = (u >> 23) + ((u & 0x7FFFFFu) ? 1u : 0u);  // rounded up to a power of two
  for (e = min(max(e, 1u), 239u);; ++e) {
    q = __uint_as_float(e << 23);
    p = __fsub_rd(lo, q);
    if (hi - p <= 254.0f * q || e >= 239u) return;
  }
}
constexpr float kMaxExtent8 = 1e30f;  // larger nodes do not fit the quantisation: no BVH8 then

struct Item8 {
  uint32_t bin, slot;  // binary node (or kLeafBit | Gaussian: a tree of one), BVH8 node it becomes
};

// One level of the cut, eight lanes per node (lane c = its c-th child): each item writes its node and queues
// its inner children, whose nodes are allocated together.
__global__ void __launch_bounds__(128) k_collapse8(const unsigned int* __restrict__ n_items_dev, const Item8* __restrict__ in,
                            Item8* __restrict__ out, unsigned int* __restrict__ out_count,
                            unsigned int* __restrict__ slot_counter, const uint32_t* __restrict__ left,
                            const uint32_t* __restrict__ right, const float4* __restrict__ plo,
                            const float4* __restrict__ phi, const float4* __restrict__ nlo,
                            const float4* __restrict__ nhi, const uint32_t* __restrict__ pos,
                            const uint8_t* __restrict__ choice, uint32_t* __restrict__ nodes, uint32_t max_nodes,
                            unsigned int* __restrict__ overflow) {
  __shared__ uint32_t s_ref[16][8], s_bud[16][8];
  constexpr unsigned kAll = 0xFFFFFFFFu;
  const int c = threadIdx.x & 7, g = threadIdx.x >> 3;          // child, group of the block
  const unsigned shift = threadIdx.x & 24u, below = (1u << c) - 1u;  // the group's lanes in the warp's ballots
  const uint32_t n_items = *n_items_dev;
  for (uint32_t b0 = blockIdx.x * 16u; b0 < n_items; b0 += gridDim.x * 16u) {  // (the same for a whole block)
  const uint32_t t = b0 + (uint32_t)g;
  const bool live = t < n_items;
  const Item8 it = live ? in[t] : Item8{kLeafBit, 0u};
  uint32_t v = it.bin;
  int bud = 1, cnt = live ? 1 : 0;
  if (live && !ref_is_leaf(it.bin)) {
    const int j = choice[8ull * it.bin];
    v = c == 0 ? left[it.bin] : right[it.bin];
    bud = c == 0 ? j : 8 - j;
    cnt = 2;
  }
  while (true) {
    const bool on = c < cnt;
    int j = 0;
    if (on && !ref_is_leaf(v))
      while (bud > 1 && (j = choice[8ull * v + bud - 1]) == 0) --bud;
    const bool open = on && !ref_is_leaf(v) && bud > 1;
    const unsigned all = __ballot_sync(kAll, open);
    if (all == 0u) break;
    const unsigned om = (all >> shift) & 0xFFu;
    const int p = c + __popc(om & below);  // the budgets sum to at most 8
    if (on && !open) s_ref[g][p] = v, s_bud[g][p] = (uint32_t)bud;
    if (open) {
      s_ref[g][p] = left[v], s_bud[g][p] = (uint32_t)j;
      s_ref[g][p + 1] = right[v], s_bud[g][p + 1] = (uint32_t)(bud - j);
    }
    cnt += __popc(om);
    __syncwarp();
    if (c < cnt) v = s_ref[g][c], bud = (int)s_bud[g][c];
    __syncwarp();
  }
  const bool on = c < cnt, leaf = on && ref_is_leaf(v), inner = on && !leaf;
  float4 bl = make_float4(INFINITY, INFINITY, INFINITY, 0.f), bh = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
  if (on) {
    bl = leaf ? plo[v & ~kLeafBit] : nlo[v];
    bh = leaf ? phi[v & ~kLeafBit] : nhi[v];
  }
  float3 lo = f3(bl.x, bl.y, bl.z), hi = f3(bh.x, bh.y, bh.z);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    lo = f3(fminf(lo.x, __shfl_xor_sync(kAll, lo.x, o)), fminf(lo.y, __shfl_xor_sync(kAll, lo.y, o)),
            fminf(lo.z, __shfl_xor_sync(kAll, lo.z, o)));
    hi = f3(fmaxf(hi.x, __shfl_xor_sync(kAll, hi.x, o)), fmaxf(hi.y, __shfl_xor_sync(kAll, hi.y, o)),
            fmaxf(hi.z, __shfl_xor_sync(kAll, hi.z, o)));
  }
  const unsigned im = (__ballot_sync(kAll, inner) >> shift) & 0xFFu;
  const uint32_t n_inner = (uint32_t)__popc(im);
  uint32_t first = 0, q = 0;
  if (live && c == 0 && n_inner) first = atomicAdd(slot_counter, n_inner);
  first = __shfl_sync(kAll, first, 0, 8);
  const bool ok = live && first + n_inner <= max_nodes &&
                  fmaxf(hi.x - lo.x, fmaxf(hi.y - lo.y, hi.z - lo.z)) < kMaxExtent8;
  if (live && !ok && c == 0) atomicOr(overflow, 1u);
  if (ok && c == 0 && n_inner) q = atomicAdd(out_count, n_inner);
  q = __shfl_sync(kAll, q, 0, 8);
  // slots by direction: repeatedly the (child, slot) pair whose child lies furthest towards the slot
  const float3 mid = f3(0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z));
  const float x = 0.5f * (bl.x + bh.x) - mid.x, y = 0.5f * (bl.y + bh.y) - mid.y, z = 0.5f * (bl.z + bh.z) - mid.z;
  uint32_t free_slots = 0xFFu;
  int slot = -1;
  for (int r = 0; r < 8; ++r) {  // lanes without a child take the slots left over, in the last rounds
    float best = -INFINITY;
    int bs = -1, bc = c;
    if (slot < 0) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float d = on ? ((k & 1) ? x : -x) + ((k & 2) ? y : -y) + ((k & 4) ? z : -z) : -INFINITY;
        if (((free_slots >> k) & 1u) && (bs < 0 || d > best)) {
          best = d;
          bs = k;
        }
      }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {  // the best pair of the group: children before none, larger, lower child
      const float ob = __shfl_xor_sync(kAll, best, o);
      const int os = __shfl_xor_sync(kAll, bs, o), oc = __shfl_xor_sync(kAll, bc, o);
      const bool my = bs >= 0, their = os >= 0;
      const bool my_on = my && bc < cnt, their_on = their && oc < cnt;
      bool take;
      if (my_on != their_on) take = their_on;
      else if (my != their) take = their;
      else take = ob > best || (!(best > ob) && oc < bc);
      if (take) best = ob, bs = os, bc = oc;
    }
    if (bc == c) slot = bs;
    free_slots &= ~(1u << bs);
  }
  if (!ok) continue;
  float px, py, pz, qx, qy, qz;
  frame8(lo.x, hi.x, px, qx);
  frame8(lo.y, hi.y, py, qy);
  frame8(lo.z, hi.z, pz, qz);
  uint32_t* wd = nodes + (size_t)it.slot * kNode8Words;
  uint8_t* planes = reinterpret_cast<uint8_t*>(wd + 4) + slot;
  uint32_t ref = kEmptyRef;
  if (on) {
    // outward to whole quanta with 1/64 of one to spare for the FP32 evaluation of the planes
    const float lov[3] = {(bl.x - px) / qx, (bl.y - py) / qy, (bl.z - pz) / qz};
    const float hiv[3] = {(bh.x - px) / qx, (bh.y - py) / qy, (bh.z - pz) / qz};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      planes[8 * a] = (uint8_t)fminf(fmaxf(floorf(lov[a] - 0.015625f), 0.f), 255.f);
      planes[24 + 8 * a] = (uint8_t)fminf(fmaxf(ceilf(hiv[a] + 0.015625f), 0.f), 255.f);
    }
    if (leaf) {
      ref = kLeafBit | pos[v & ~kLeafBit];
    } else {
      const uint32_t k = (uint32_t)__popc(im & below);
      ref = first + k;
      out[q + k] = Item8{v, ref};
    }
  } else {
#pragma unroll
    for (int a = 0; a < 3; ++a) planes[8 * a] = 255u, planes[24 + 8 * a] = 0u;
  }
  wd[16 + slot] = ref;
  // inner slots, gathered over the group
  unsigned is = inner ? 1u << slot : 0u;
  const unsigned gm = 0xFFu << shift;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) is |= __shfl_xor_sync(gm, is, o);
  if (c == 0) {
    auto eb = [](float f) { return (__float_as_uint(f) >> 23) + 15u; };
    wd[0] = __float_as_uint(px);
    wd[1] = __float_as_uint(py);
    wd[2] = __float_as_uint(pz);
    wd[3] = eb(qx) | (eb(qy) << 8) | (eb(qz) << 16) | (is << 24);
  }
  }
}

// Node 0: only a reference to the root, node 1.
__global__ void k_root8(uint32_t* __restrict__ nodes) {
  const uint32_t k = threadIdx.x;
  if (k < kNode8Words) nodes[k] = k == 16u ? 1u : (k >= 17u ? kEmptyRef : 0u);
}

// Scene order from the collapse's positions: order[pos[m]] = Morton order's caller index.
__global__ void k_compose(uint32_t n, const uint32_t* __restrict__ morton_order, const uint32_t* __restrict__ pos,
                          uint32_t* __restrict__ order) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  order[pos[i]] = morton_order[i];
}

__global__ void k_iota(uint32_t n, uint32_t* __restrict__ v) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) v[i] = i;
}

// Root of a scene with <= 32 Gaussians: one node holding one leaf.
__global__ void k_single_leaf_root(uint32_t n, const float4* __restrict__ plo,
                                   const float4* __restrict__ phi, float4* __restrict__ wide) {
  const int c = threadIdx.x;
  if (c >= 32) return;
  if (c == 0) {
    float4 l = make_float4(INFINITY, INFINITY, INFINITY, 0.f), h = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
    for (uint32_t i = 0; i < n; ++i) {
      const float4 a = plo[i], b = phi[i];
      l.x = fminf(l.x, a.x); l.y = fminf(l.y, a.y); l.z = fminf(l.z, a.z);
      h.x = fmaxf(h.x, b.x); h.y = fmaxf(h.y, b.y); h.z = fmaxf(h.z, b.z);
    }
    l.w = __uint_as_float(wide_leaf_ref(0u, n));
    wide[0] = l;
    wide[32] = h;
  } else {
    wide[c] = make_float4(INFINITY, INFINITY, INFINITY, __uint_as_float(kEmptyRef));
    wide[32 + c] = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
  }
}

// One-Gaussian binary "tree": a root whose left child is the Gaussian and right is empty.
__global__ void k_single_binary_root(const float4* __restrict__ plo, const float4* __restrict__ phi,
                                     float4* __restrict__ out) {
  float4 l = plo[0];
  l.w = __uint_as_float(kLeafBit | 0u);
  out[0] = l;
  out[1] = phi[0];
  out[2] = make_float4(INFINITY, INFINITY, INFINITY, __uint_as_float(kEmptyRef));
  out[3] = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
}

template <class T>
struct Scratch {  // stream-ordered temporary, freed on scope exit
  T* p = nullptr;
  cudaStream_t s;
  explicit Scratch(cudaStream_t st) : s(st) {}
  ~Scratch() { dev_free(p, s); }
};

}  // namespace

// A scene without Gaussians (the reference builds an instance AS over zero instances and every
// ray misses; test/scenes/geometric_validation.cpp empty_scene): one BVH32 root and one binary
// root whose children are all empty, and one zeroed element in each per-Gaussian array so that
// no pointer is null.  Every traversal tests the root's children, finds none, and ends.
vp_status build_empty_scene(vp_context* ctx, const vp_gaussians* g, float sigma_multiplier,
                            const vp_scene_options& opt, vp_scene* sc) {
  cudaStream_t st = ctx->stream;
  float ref_empty;
  std::memcpy(&ref_empty, &kEmptyRef, sizeof(ref_empty));
  const float4 lo_empty = make_float4(INFINITY, INFINITY, INFINITY, ref_empty);
  const float4 hi_empty = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
  float4 wide_h[64], bin_h[4];
  for (int c = 0; c < 32; ++c) wide_h[c] = lo_empty, wide_h[32 + c] = hi_empty;
  bin_h[0] = bin_h[2] = lo_empty;
  bin_h[1] = bin_h[3] = hi_empty;
  vp_status s;
  if ((s = dev_alloc(&sc->prims, 4, st)) || (s = dev_alloc(&sc->perm, 1, st)) || (s = dev_alloc(&sc->pbox, 2, st)) ||
      (s = dev_alloc(&sc->raw, 2, st)) || (s = dev_alloc(&sc->wide, 64, st)) || (s = dev_alloc(&sc->bin, 4, st)))
    return s;
  VP_CUDA(cudaMemsetAsync(sc->prims, 0, 4 * sizeof(float4), st));
  VP_CUDA(cudaMemsetAsync(sc->perm, 0, sizeof(uint32_t), st));
  VP_CUDA(cudaMemsetAsync(sc->pbox, 0, 2 * sizeof(float4), st));
  VP_CUDA(cudaMemsetAsync(sc->raw, 0, 2 * sizeof(float4), st));
  VP_CUDA(cudaMemcpyAsync(sc->wide, wide_h, sizeof(wide_h), cudaMemcpyHostToDevice, st));
  VP_CUDA(cudaMemcpyAsync(sc->bin, bin_h, sizeof(bin_h), cudaMemcpyHostToDevice, st));
  VP_CUDA(cudaStreamSynchronize(st));
  sc->ctx = ctx;
  sc->scale_is_log = g->scale_is_log ? 1 : 0;
  sc->sigma_multiplier = sigma_multiplier;
  SceneView& v = sc->view;
  v.prims = sc->prims;
  v.perm = sc->perm;
  v.wide = sc->wide;
  v.bin = sc->bin;
  v.pbox = sc->pbox;
  v.nodes8 = nullptr;
  v.depth8 = 0u;
  v.count = 0u;
  v.wide_root = 0u;
  v.bin_root = 0u;
  v.stack_cap = 31u + 2u;
  v.argmin_cap = v.stack_cap + kArgminBestFirstStack + 64u;
  v.albedo_all_zero = 1;
  v.one_albedo = 1;
  v.albedo = make_float3(0.f, 0.f, 0.f);
  v.tau_nearest = 0;
  vp_scene_info& info = sc->info;
  info = vp_scene_info{};
  info.tau_order = VP_TAU_ORDER_LANE;
  info.wide_nodes = 1;
  info.wide_depth = 1;
  info.binary_nodes = 1;
  info.wide_builder = opt.wide_builder;
  info.binary_builder = opt.binary_builder;
  info.leaf_max = opt.leaf_max;
  info.wide_collapse = opt.wide_collapse;
  info.albedo_all_zero = 1;
  info.device_bytes = 64ull + 4ull + 32ull + 32ull + 1024ull + 64ull;
  return VP_OK;
}

// Above this overlap (k_overlap) a scene of more than one node's Gaussians goes without the 8-wide BVH: a ray meets so
// many of them that there is nothing to cull, and a warp that takes 24 neighbouring records a step does better than
// lanes that gather theirs.  Images of 11k / 60k / 217k paths, thread / warp per ray: 3,000 Gaussians in a
// box of side 2, scales of 0.2 (overlap 0.16) 6.1 / 17.6 / 32.2 and 5.6 / 15.2 / 40.8 ms, of 0.3 (0.25) 17.7 / 52.7 /
// 101.8 and 10.4 / 35.0 / 104.5 ms, of 0.8 (0.53) 48 / 177 / 392 and 23 / 112 / 380 ms; 300 in one place 2.2 / 5.4 / 7.9
// and 1.1 / 2.3 / 5.4 ms.
constexpr float kMaxOverlap8 = 0.2f;

// The compressed 8-wide BVH of a scene (sc->nodes8, depth8 levels counting node 0), cut from the binary
// tree the BVH32 comes from.  depth8 = 0: the tree is too deep or too large for it (kMaxDepth8,
// kMaxNodes8) and the engines use the warp-cooperative queries; the caller takes VP_ERROR_OUT_OF_MEMORY so, too.
static vp_status build_bvh8(vp_context* ctx, uint32_t n, uint32_t root, const uint32_t* wl, const uint32_t* wr,
                            const float4* plo, const float4* phi, const float4* wlo, const float4* whi,
                            const uint32_t* par, const uint32_t* par_leaf, const uint32_t* pos, vp_scene* sc,
                            uint32_t& depth8, uint32_t& nodes8) {
  cudaStream_t st = ctx->stream;
  depth8 = nodes8 = 0;
  const int TB = 256;
  vp_status s;
  Scratch<float> cost(st);
  Scratch<uint8_t> choice(st);
  Scratch<unsigned int> flags(st), ctr(st);
  if (n > 1u) {
    if ((s = dev_alloc(&cost.p, 8ull * (n - 1u), st))) return s;
    if ((s = dev_alloc(&choice.p, 8ull * (n - 1u), st))) return s;
    if ((s = dev_alloc(&flags.p, n - 1u, st))) return s;
    VP_CUDA(cudaMemsetAsync(flags.p, 0, sizeof(unsigned int) * (n - 1u), st));
    k_dp8_cost<<<(n + TB - 1) / TB, TB, 0, st>>>(n, root, wl, wr, plo, phi, wlo, whi, par, par_leaf, flags.p, cost.p,
                                                 choice.p);
    VP_CUDA(cudaGetLastError());
  }
  // every node has at least two children, so there are fewer nodes than Gaussians (+ node 0 and the root
  // of a tree of one)
  const uint32_t max_nodes = std::min(n + 1u, kMaxNodes8);
  Scratch<uint32_t> nodes(st);
  Scratch<Item8> qa(st), qb(st);
  if ((s = dev_alloc(&nodes.p, (size_t)max_nodes * kNode8Words, st))) return s;
  if ((s = dev_alloc(&qa.p, max_nodes, st))) return s;
  if ((s = dev_alloc(&qb.p, max_nodes, st))) return s;
  constexpr uint32_t kLevels = kMaxDepth8;             // levels below node 0 that may hold items
  if ((s = dev_alloc(&ctr.p, kLevels + 3u, st))) return s;  // items per level, then next node, overflow
  unsigned int c0[kLevels + 3u] = {};
  c0[0] = 1u;
  c0[kLevels + 1u] = 2u;
  const Item8 root_item{n > 1u ? root : kLeafBit, 1u};
  VP_CUDA(cudaMemcpyAsync(ctr.p, c0, sizeof(c0), cudaMemcpyHostToDevice, st));
  VP_CUDA(cudaMemcpyAsync(qa.p, &root_item, sizeof(root_item), cudaMemcpyHostToDevice, st));
  k_root8<<<1, 32, 0, st>>>(nodes.p);
  VP_CUDA(cudaGetLastError());
  uint64_t bound = 1;
  uint32_t k = 0;
  unsigned int c[kLevels + 3u];
  while (true) {
    // a 500k-Gaussian tree has some 14 levels, so one read of the counts usually ends the loop
    for (int i = 0; i < 16 && k < kLevels; ++i, ++k) {
      Item8* in = (k & 1u) ? qb.p : qa.p;
      Item8* out = (k & 1u) ? qa.p : qb.p;
      k_collapse8<<<(unsigned)std::min<uint64_t>((bound + 15) / 16, (uint64_t)ctx->sm_count * 16u), 128, 0, st>>>(ctr.p + k, in, out, ctr.p + k + 1u,
                                                                 ctr.p + kLevels + 1u, wl, wr, plo, phi, wlo, whi, pos,
                                                                 choice.p, nodes.p, max_nodes, ctr.p + kLevels + 2u);
      VP_CUDA(cudaGetLastError());
      bound = std::min<uint64_t>(bound * 8u, max_nodes);
    }
    VP_CUDA(cudaMemcpyAsync(c, ctr.p, sizeof(c), cudaMemcpyDeviceToHost, st));
    VP_CUDA(cudaStreamSynchronize(st));
    if (c[kLevels + 2u] != 0u || c[k] == 0u || k == kLevels) break;
    bound = c[k];
  }
  if (c[kLevels + 2u] != 0u || c[k] != 0u) return VP_OK;
  uint32_t levels = 0;
  while (c[levels] != 0u) ++levels;
  if (levels + 1u > kMaxDepth8) return VP_OK;
  nodes8 = c[kLevels + 1u];
  if ((s = dev_alloc(&sc->nodes8, (size_t)nodes8 * kNode8Words, st))) return s;
  VP_CUDA(cudaMemcpyAsync(sc->nodes8, nodes.p, 4ull * kNode8Words * nodes8, cudaMemcpyDeviceToDevice, st));
  depth8 = levels + 1u;
  return VP_OK;
}

vp_status build_scene(vp_context* ctx, const vp_gaussians* g, float sigma_multiplier, const vp_scene_options& opt,
                      vp_scene* sc) {
  cudaStream_t st = ctx->stream;
  const uint32_t n = g->count;
  if (n >= (1u << 26)) return fail(VP_ERROR_LIMIT, "scene exceeds 2^26 Gaussians");
  if (!(sigma_multiplier > 0.f) || !std::isfinite(sigma_multiplier))
    return fail(VP_ERROR_INVALID_ARGUMENT, "sigma_multiplier must be positive and finite");
  if (n == 0) return build_empty_scene(ctx, g, sigma_multiplier, opt, sc);
  if (!g->mean || !g->scale || !g->quat_wxyz || !g->density)
    return fail(VP_ERROR_INVALID_ARGUMENT, "vp_gaussians: mean, scale, quat_wxyz and density are required");

  VP_CUDA(cudaEventRecord(ctx->ev0, st));
  // Inputs on the device.
  Scratch<float> d_mean(st), d_scale(st), d_quat(st), d_dens(st), d_alb(st);
  const float *mean = g->mean, *scale = g->scale, *quat = g->quat_wxyz, *dens = g->density,
              *alb = g->albedo;
  if (g->memory == VP_MEMORY_HOST) {
    vp_status s;
    if ((s = dev_alloc(&d_mean.p, 3ull * n, st))) return s;
    if ((s = dev_alloc(&d_scale.p, 3ull * n, st))) return s;
    if ((s = dev_alloc(&d_quat.p, 4ull * n, st))) return s;
    if ((s = dev_alloc(&d_dens.p, 1ull * n, st))) return s;
    VP_CUDA(cudaMemcpyAsync(d_mean.p, mean, 12ull * n, cudaMemcpyHostToDevice, st));
    VP_CUDA(cudaMemcpyAsync(d_scale.p, scale, 12ull * n, cudaMemcpyHostToDevice, st));
    VP_CUDA(cudaMemcpyAsync(d_quat.p, quat, 16ull * n, cudaMemcpyHostToDevice, st));
    VP_CUDA(cudaMemcpyAsync(d_dens.p, dens, 4ull * n, cudaMemcpyHostToDevice, st));
    mean = d_mean.p;
    scale = d_scale.p;
    quat = d_quat.p;
    dens = d_dens.p;
    if (alb) {
      if ((s = dev_alloc(&d_alb.p, 3ull * n, st))) return s;
      VP_CUDA(cudaMemcpyAsync(d_alb.p, alb, 12ull * n, cudaMemcpyHostToDevice, st));
      alb = d_alb.p;
    }
  } else if (g->memory != VP_MEMORY_DEVICE) {
    return fail(VP_ERROR_INVALID_ARGUMENT, "vp_gaussians.memory must be VP_MEMORY_HOST or VP_MEMORY_DEVICE");
  }

  vp_status s;
  Scratch<float4> rec0(st), lo0(st), hi0(st), plo(st), phi(st);
  Scratch<ErrorWords> errw(st);
  Scratch<unsigned int> bounds(st);
  if ((s = dev_alloc(&rec0.p, 4ull * n, st))) return s;
  if ((s = dev_alloc(&lo0.p, n, st))) return s;
  if ((s = dev_alloc(&hi0.p, n, st))) return s;
  if ((s = dev_alloc(&errw.p, 1, st))) return s;
  if ((s = dev_alloc(&bounds.p, 12, st))) return s;
  {
    ErrorWords e0{0x7FFFFFFF, 0x7FFFFFFF, 0x7FFFFFFF, 0u, 0u, 0u, {0.f, 0.f, 0.f}, 0.f};
    VP_CUDA(cudaMemcpyAsync(errw.p, &e0, sizeof(e0), cudaMemcpyHostToDevice, st));
    unsigned int b0[12];
    for (int k = 0; k < 3; ++k) {
      b0[k] = 0xFFFFFFFFu;
      b0[3 + k] = 0u;
      b0[6 + k] = 0xFFFFFFFFu;
      b0[9 + k] = 0u;
    }
    VP_CUDA(cudaMemcpyAsync(bounds.p, b0, sizeof(b0), cudaMemcpyHostToDevice, st));
  }
  const int TB = 256;
  const unsigned nb = (n + TB - 1) / TB;
  k_precompute<<<nb, TB, 0, st>>>(n, mean, scale, quat, dens, alb, g->scale_is_log, sigma_multiplier,
                                  rec0.p, lo0.p, hi0.p, errw.p);
  VP_CUDA(cudaGetLastError());
  k_bounds<<<std::min(nb, 1184u), TB, 0, st>>>(n, mean, lo0.p, hi0.p, bounds.p);
  VP_CUDA(cudaGetLastError());
  k_overlap<<<1, 1024, 0, st>>>(n, mean, lo0.p, hi0.p, errw.p);
  VP_CUDA(cudaGetLastError());
  ErrorWords eh{};
  unsigned int bh[12];
  VP_CUDA(cudaMemcpyAsync(&eh, errw.p, sizeof(eh), cudaMemcpyDeviceToHost, st));
  VP_CUDA(cudaMemcpyAsync(bh, bounds.p, sizeof(bh), cudaMemcpyDeviceToHost, st));
  VP_CUDA(cudaStreamSynchronize(st));
  if (eh.bad_scale != 0x7FFFFFFF)
    return fail(VP_ERROR_INVALID_ARGUMENT, "Gaussian " + std::to_string(eh.bad_scale) +
                                               ": invalid scale - all components must be finite and > 0");
  if (eh.bad_density != 0x7FFFFFFF)
    return fail(VP_ERROR_INVALID_ARGUMENT, "Gaussian " + std::to_string(eh.bad_density) +
                                               ": invalid density - must be finite and > 0");
  if (eh.bad_center != 0x7FFFFFFF)
    return fail(VP_ERROR_INVALID_ARGUMENT, "Gaussian " + std::to_string(eh.bad_center) +
                                               ": NaN/Inf in centre or rotation");

  // Morton codes + radix sort (stable: ties keep the caller's order).
  Scratch<uint64_t> codes(st);
  Scratch<uint32_t> idx(st), pos(st);
  Scratch<unsigned char> sort_tmp(st);
  if ((s = dev_alloc(&codes.p, n, st))) return s;
  if ((s = dev_alloc(&idx.p, n, st))) return s;
  if ((s = dev_alloc(&pos.p, n, st))) return s;
  k_morton<<<nb, TB, 0, st>>>(n, mean, bounds.p, codes.p, idx.p);
  VP_CUDA(cudaGetLastError());
  // Stable radix sort of the 63-bit codes (ties keep the caller's order), in place: codes become
  // the sorted codes and idx the Morton order.
  const size_t tmp_bytes = radix_sort_tmp_bytes_u64(n);
  if ((s = dev_alloc(&sort_tmp.p, tmp_bytes, st))) return s;
  if ((s = radix_sort_pairs(codes.p, idx.p, n, 63, sort_tmp.p, tmp_bytes, st))) return s;
  const uint64_t* codes_sorted = codes.p;
  const uint32_t* morton = idx.p;
  if ((s = dev_alloc(&plo.p, n, st))) return s;
  if ((s = dev_alloc(&phi.p, n, st))) return s;
  k_gather_boxes<<<nb, TB, 0, st>>>(n, morton, lo0.p, hi0.p, plo.p, phi.p);
  VP_CUDA(cudaGetLastError());

  // PLOC clustering: the binary tree of the BVH32 and of the megakernel unless the options ask for
  // the Karras tree for both (a BVH32 that is a single leaf needs no tree).
  const uint32_t ni = n > 1 ? n - 1 : 1;
  const uint32_t kLeafMax = opt.leaf_max;
  bool wide_ploc = n > kLeafMax && opt.wide_builder == VP_TREE_PLOC;
  bool use_ploc = n > 1u && (wide_ploc || opt.binary_builder == VP_TREE_PLOC);
  Scratch<uint32_t> pleft(st), pright(st), nn(st), totals(st);
  Scratch<float4> pnlo(st), pnhi(st), ca(st), cb(st), oa(st), ob(st);
  Scratch<unsigned long long> counts(st);
  uint32_t wroot = 0u, ploc_height = 0u;
  if (use_ploc) {
    const uint32_t tiles = (n + kPlocBlock - 1) / kPlocBlock, n_super = (tiles + kPlocSuper - 1) / kPlocSuper;
    if ((s = dev_alloc(&pleft.p, ni, st))) return s;
    if ((s = dev_alloc(&pright.p, ni, st))) return s;
    if ((s = dev_alloc(&pnlo.p, ni, st))) return s;
    if ((s = dev_alloc(&pnhi.p, ni, st))) return s;
    if ((s = dev_alloc(&nn.p, n, st))) return s;
    if ((s = dev_alloc(&totals.p, 8, st))) return s;
    if ((s = dev_alloc(&ca.p, n, st))) return s;
    if ((s = dev_alloc(&cb.p, n, st))) return s;
    if ((s = dev_alloc(&oa.p, n, st))) return s;
    if ((s = dev_alloc(&ob.p, n, st))) return s;
    if ((s = dev_alloc(&counts.p, (size_t)tiles + 2u * n_super, st))) return s;
    unsigned long long* super_c[2] = {counts.p + tiles, counts.p + tiles + n_super};
    VP_CUDA(cudaMemsetAsync(super_c[0], 0, sizeof(unsigned long long) * n_super, st));
    k_ploc_init<<<nb, TB, 0, st>>>(n, plo.p, phi.p, ca.p, cb.p);
    VP_CUDA(cudaGetLastError());
    {
      const uint32_t c0[8] = {n, 0u, 0u, 0u, n, 0u, 0u, 0u};
      VP_CUDA(cudaMemcpyAsync(totals.p, c0, sizeof(c0), cudaMemcpyHostToDevice, st));
    }
    // Passes run in chunks between host reads of the count; the count only falls, so the last
    // value read bounds the grids of the next chunk.
    // A chain of nested boxes (concentric Gaussians of growing size) merges about one pair per
    // pass; past kMaxPasses the build drops the clustering and uses the Karras tree instead.
    constexpr int kChunk = 16;
    constexpr int kMaxPasses = 1024;
    uint32_t m = n, made = 0u, passes = 0u;
    int launch = 0;
    while (m > 1u && passes < (uint32_t)kMaxPasses) {
      for (int k = 0; k < kChunk && m > kPlocTail; ++k, ++launch) {
        const uint32_t* cin = totals.p + 4 * (launch & 1);
        uint32_t* cout = totals.p + 4 * ((launch + 1) & 1);
        const unsigned grid = (m + kPlocBlock - 1) / kPlocBlock;
        k_ploc_pair<<<grid, kPlocBlock + 2 * kPlocRadius, 0, st>>>(cin, ca.p, cb.p, nn.p, counts.p, super_c[launch & 1]);
        VP_CUDA(cudaGetLastError());
        k_ploc_merge<<<grid, kPlocBlock, 0, st>>>(cin, cout, nn.p, counts.p, super_c[launch & 1],
                                                 super_c[(launch + 1) & 1], n_super, ca.p, cb.p, oa.p, ob.p, pleft.p,
                                                 pright.p, pnlo.p, pnhi.p);
        VP_CUDA(cudaGetLastError());
        std::swap(ca.p, oa.p);
        std::swap(cb.p, ob.p);
      }
      uint32_t* cur = totals.p + 4 * (launch & 1);
      k_ploc_tail<<<1, kPlocTail, 0, st>>>(cur, (uint32_t)kMaxPasses, ca.p, cb.p, pleft.p, pright.p, pnlo.p, pnhi.p);
      VP_CUDA(cudaGetLastError());
      uint32_t th[4];
      VP_CUDA(cudaMemcpyAsync(th, cur, sizeof(th), cudaMemcpyDeviceToHost, st));
      VP_CUDA(cudaStreamSynchronize(st));
      if (th[0] >= m && m > 1u && th[2] < (uint32_t)kMaxPasses)
        return fail(VP_ERROR_INTERNAL, "PLOC clustering made no progress");
      if (th[0] + th[1] != n || th[1] > ni) return fail(VP_ERROR_INTERNAL, "PLOC clustering lost a cluster");
      m = th[0];
      made = th[1];
      passes = th[2];
      ploc_height = th[3];
    }
    if (m > 1u) {
      use_ploc = false;
      wide_ploc = false;
      ploc_height = 0u;
    } else {
      wroot = made - 1u;  // the last merge made the root (node n - 2)
    }
  }
  // Karras radix tree + refit over the Morton order: the BVH32's source when the options ask for it,
  // and the megakernel's binary tree when they ask for it or the PLOC tree is deeper than the
  // megakernel's thread-private stack.
  Scratch<uint32_t> left(st), right(st), first(st), last(st), par_i(st), par_l(st);
  Scratch<float4> nlo(st), nhi(st);
  Scratch<unsigned int> flags(st);
  const bool bin_from_ploc = use_ploc && opt.binary_builder == VP_TREE_PLOC && ploc_height + 1u < (uint32_t)kBinStack;
  const bool need_karras = !wide_ploc || !bin_from_ploc;
  if (need_karras) {
    if ((s = dev_alloc(&left.p, ni, st))) return s;
    if ((s = dev_alloc(&right.p, ni, st))) return s;
    if ((s = dev_alloc(&first.p, ni, st))) return s;
    if ((s = dev_alloc(&last.p, ni, st))) return s;
    if ((s = dev_alloc(&par_i.p, ni, st))) return s;
    if ((s = dev_alloc(&par_l.p, n, st))) return s;
    if ((s = dev_alloc(&nlo.p, ni, st))) return s;
    if ((s = dev_alloc(&nhi.p, ni, st))) return s;
    if ((s = dev_alloc(&flags.p, ni, st))) return s;
    if (n > 1) {
      VP_CUDA(cudaMemsetAsync(flags.p, 0, sizeof(unsigned int) * ni, st));
      k_karras<<<(ni + TB - 1) / TB, TB, 0, st>>>((int)n, codes_sorted, left.p, right.p, first.p, last.p,
                                                  par_i.p, par_l.p);
      VP_CUDA(cudaGetLastError());
      k_refit<<<nb, TB, 0, st>>>((int)n, left.p, right.p, par_i.p, par_l.p, plo.p, phi.p, nlo.p, nhi.p, flags.p);
      VP_CUDA(cudaGetLastError());
    }
  }

  const uint32_t wide_root = wide_ploc ? wroot : 0u;
  const uint32_t* wl = wide_ploc ? pleft.p : left.p;
  const uint32_t* wr = wide_ploc ? pright.p : right.p;
  const float4* wlo = wide_ploc ? pnlo.p : nlo.p;
  const float4* whi = wide_ploc ? pnhi.p : nhi.p;

  // Collapse to BVH32; its depth-first leaf order defines the scene order (pos).
  // Upper bound on BVH32 nodes: childless nodes hold > L disjoint Gaussians (<= n/(L+1)), nodes
  // with one node child hold 31 leaves of their own (<= n/31), branching nodes are fewer than
  // childless ones (<= n/(L+1)).
  const uint32_t max_wide = n / 31u + 2u * (n / (kLeafMax + 1u)) + 4u;
  float4* wide = nullptr;
  if ((s = dev_alloc(&wide, 64ull * max_wide, st))) return s;
  sc->wide = wide;
  uint32_t depth = 1, wide_nodes = 1, leaves = 1;
  bool dp_used = false;
  Scratch<uint32_t> par(st), par_leaf(st);
  if (n > 1u) {
    if ((s = dev_alloc(&par.p, n - 1u, st))) return s;
    if ((s = dev_alloc(&par_leaf.p, n, st))) return s;
    k_parents<<<(n - 1u + TB - 1) / TB, TB, 0, st>>>(n - 1u, wl, wr, par.p, par_leaf.p);
    VP_CUDA(cudaGetLastError());
  }
  if (n <= kLeafMax) {
    k_single_leaf_root<<<1, 32, 0, st>>>(n, plo.p, phi.p, wide);
    VP_CUDA(cudaGetLastError());
    k_iota<<<nb, TB, 0, st>>>(n, pos.p);
    VP_CUDA(cudaGetLastError());
  } else {
    // SAH-optimal slot tables (k_dp_cost) when asked for and the scene is at most 2^24 Gaussians.
    const uint32_t nint = n - 1u;
    Scratch<float> dp_cost(st);
    Scratch<uint8_t> dp_split(st), dp_best(st), dp_leaf(st);
    Scratch<uint32_t> dp_single(st);
    Scratch<unsigned int> dp_flags(st);
    DpTables T{nullptr, nullptr, nullptr, nullptr, nullptr};
    bool dp = opt.wide_collapse == VP_COLLAPSE_SAH && n <= (1u << 24);
    if (dp) {
      if ((s = dev_alloc(&dp_cost.p, 32ull * nint, st))) return s;
      if ((s = dev_alloc(&dp_split.p, 32ull * nint, st))) return s;
      if ((s = dev_alloc(&dp_best.p, 32ull * nint, st))) return s;
      if ((s = dev_alloc(&dp_leaf.p, nint, st))) return s;
      if ((s = dev_alloc(&dp_single.p, nint, st))) return s;
      if ((s = dev_alloc(&dp_flags.p, nint, st))) return s;
      VP_CUDA(cudaMemsetAsync(dp_flags.p, 0, sizeof(unsigned int) * nint, st));
      T = DpTables{dp_cost.p, dp_split.p, dp_best.p, dp_single.p, dp_leaf.p};
      k_dp_cost<<<nb, TB, 0, st>>>(n, wide_root, wl, wr, plo.p, phi.p, wlo, whi, par.p, par_leaf.p, dp_flags.p, T,
                                   kLeafMax);
      VP_CUDA(cudaGetLastError());
    }
    Scratch<CollapseItem> qa(st), qb(st);
    Scratch<unsigned int> ctr(st), lvl(st);
    constexpr int kMaxLevels = 512;  // BVH32 depth bound (a PLOC chain of 1,024 passes stays far below)
    constexpr int kLevelChunk = 8;   // levels between host reads
    if ((s = dev_alloc(&qa.p, max_wide, st))) return s;
    if ((s = dev_alloc(&qb.p, max_wide, st))) return s;
    if ((s = dev_alloc(&ctr.p, 3, st))) return s;
    if ((s = dev_alloc(&lvl.p, kMaxLevels + 1, st))) return s;
    // A level-by-level collapse: lvl[k] = items (BVH32 nodes to fill) at level k, counted on the
    // device; the host reads the counts every kLevelChunk levels.  An SAH cut that needs more
    // nodes than the greedy bound is redone greedily.
    for (int attempt = 0; attempt < 2; ++attempt) {
      CollapseItem root{wide_root, 0u, 0u, 0u};
      VP_CUDA(cudaMemcpyAsync(qa.p, &root, sizeof(root), cudaMemcpyHostToDevice, st));
      const unsigned int c0[3] = {1u, 0u, 0u};  // next free slot, leaves, overflow
      VP_CUDA(cudaMemcpyAsync(ctr.p, c0, sizeof(c0), cudaMemcpyHostToDevice, st));
      VP_CUDA(cudaMemsetAsync(lvl.p, 0, sizeof(unsigned int) * (kMaxLevels + 1), st));
      const unsigned int one = 1u;
      VP_CUDA(cudaMemcpyAsync(lvl.p, &one, sizeof(one), cudaMemcpyHostToDevice, st));
      uint64_t bound = 1;  // upper bound of the items at the next level to launch
      int k = 0;
      bool done = false, over = false;
      std::vector<unsigned int> counts;
      while (!done) {
        for (int c = 0; c < kLevelChunk; ++c, ++k) {
          if (k >= kMaxLevels) return fail(VP_ERROR_INTERNAL, "BVH32 deeper than 512 levels");
          const unsigned grid = (unsigned)std::min<uint64_t>((bound + 3) / 4, (uint64_t)ctx->sm_count * 16u);
          CollapseItem* qin = (k & 1) ? qb.p : qa.p;
          CollapseItem* qout = (k & 1) ? qa.p : qb.p;
          if (dp)
            k_collapse<true><<<grid, 128, 0, st>>>(lvl.p + k, qin, qout, lvl.p + k + 1, ctr.p, wl, wr, plo.p, phi.p,
                                                   wlo, whi, wide, kLeafMax, pos.p, ctr.p + 1, T, max_wide, ctr.p + 2);
          else
            k_collapse<false><<<grid, 128, 0, st>>>(lvl.p + k, qin, qout, lvl.p + k + 1, ctr.p, wl, wr, plo.p, phi.p,
                                                    wlo, whi, wide, kLeafMax, pos.p, ctr.p + 1, T, max_wide, ctr.p + 2);
          VP_CUDA(cudaGetLastError());
          bound = std::min<uint64_t>(bound * 32u, max_wide);  // each item makes at most 32 children
        }
        unsigned int ch[3];
        counts.resize((size_t)k + 1u);
        VP_CUDA(cudaMemcpyAsync(ch, ctr.p, sizeof(ch), cudaMemcpyDeviceToHost, st));
        VP_CUDA(cudaMemcpyAsync(counts.data(), lvl.p, sizeof(unsigned int) * counts.size(), cudaMemcpyDeviceToHost, st));
        VP_CUDA(cudaStreamSynchronize(st));
        wide_nodes = ch[0];
        leaves = ch[1];
        over = ch[2] != 0u;
        bound = counts.back();
        done = over || bound == 0u;
      }
      if (!over) {
        depth = 0;
        while (depth < (uint32_t)k && counts[depth] != 0u) ++depth;
        dp_used = dp;
        break;
      }
      if (!dp) return fail(VP_ERROR_INTERNAL, "BVH32 node budget exceeded");
      dp = false;
    }
  }
  // Scene order, then the records, boxes and adjoint inputs gathered into it.
  uint32_t* perm = nullptr;
  if ((s = dev_alloc(&perm, n, st))) return s;
  sc->perm = perm;
  k_compose<<<nb, TB, 0, st>>>(n, morton, pos.p, perm);
  VP_CUDA(cudaGetLastError());
  float4* prims = nullptr;
  if ((s = dev_alloc(&prims, 4ull * n, st))) return s;
  sc->prims = prims;
  float4* pbox = nullptr;
  if ((s = dev_alloc(&pbox, 2ull * n, st))) return s;
  sc->pbox = pbox;
  k_gather<<<nb, TB, 0, st>>>(n, perm, rec0.p, lo0.p, hi0.p, prims, pbox);
  VP_CUDA(cudaGetLastError());
  dev_free(rec0.p, st);
  dev_free(lo0.p, st);
  dev_free(hi0.p, st);
  float4* raw = nullptr;
  if ((s = dev_alloc(&raw, 2ull * n, st))) return s;
  sc->raw = raw;
  sc->scale_is_log = g->scale_is_log ? 1 : 0;
  sc->sigma_multiplier = sigma_multiplier;
  k_gather_raw<<<nb, TB, 0, st>>>(n, perm, scale, quat, dens, raw);
  VP_CUDA(cudaGetLastError());
  float4* bin = nullptr;
  if ((s = dev_alloc(&bin, 4ull * ni, st))) return s;
  sc->bin = bin;
  uint32_t bin_root = 0u;
  if (bin_from_ploc) {
    k_binary_nodes<<<(ni + TB - 1) / TB, TB, 0, st>>>((int)n, pleft.p, pright.p, plo.p, phi.p, pnlo.p, pnhi.p, pos.p,
                                                      bin);
    bin_root = wroot;
  } else if (n > 1) {
    k_binary_nodes<<<(ni + TB - 1) / TB, TB, 0, st>>>((int)n, left.p, right.p, plo.p, phi.p, nlo.p, nhi.p, pos.p,
                                                      bin);
  } else {
    k_single_binary_root<<<1, 1, 0, st>>>(plo.p, phi.p, bin);
  }
  VP_CUDA(cudaGetLastError());
  if (wide_nodes < max_wide) {  // keep only the nodes in use
    float4* tight = nullptr;
    if ((s = dev_alloc(&tight, 64ull * wide_nodes, st))) return s;
    VP_CUDA(cudaMemcpyAsync(tight, wide, 1024ull * wide_nodes, cudaMemcpyDeviceToDevice, st));
    dev_free(wide, st);
    wide = tight;
    sc->wide = wide;
  }
  // Last, so that a device with room for the rest only goes without it.
  uint32_t depth8 = 0, nodes8 = 0;
  sc->overlap = eh.overlap;
  if (n <= 8u || eh.overlap <= kMaxOverlap8) {
    s = build_bvh8(ctx, n, wide_root, wl, wr, plo.p, phi.p, wlo, whi, par.p, par_leaf.p, pos.p, sc, depth8, nodes8);
    if (s == VP_ERROR_OUT_OF_MEMORY) {
      dev_free(sc->nodes8, st);
      depth8 = nodes8 = 0u;
    } else if (s) {
      return s;
    }
  }
  VP_CUDA(cudaEventRecord(ctx->ev1, st));
  VP_CUDA(cudaEventSynchronize(ctx->ev1));
  float ms = 0.f;
  VP_CUDA(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));

  sc->ctx = ctx;
  SceneView& v = sc->view;
  v.prims = prims;
  v.perm = perm;
  v.wide = wide;
  v.bin = bin;
  v.pbox = pbox;
  v.nodes8 = sc->nodes8;
  v.depth8 = depth8;
  v.count = n;
  v.wide_root = 0u;
  v.bin_root = bin_root;
  v.stack_cap = 31u * depth + 2u;
  v.argmin_cap = v.stack_cap + kArgminBestFirstStack + 64u;
  v.albedo_all_zero = eh.any_albedo ? 0 : 1;
  v.one_albedo = eh.mixed_albedo ? 0 : 1;
  v.albedo = make_float3(eh.albedo0[0], eh.albedo0[1], eh.albedo0[2]);
  // AUTO: nearest first where rays need many translucent Gaussians to become opaque and the tree
  // has levels below the root's children to order (on a two-level tree the ranking pass costs
  // more than it saves)
  const int32_t tau_order = opt.tau_order != VP_TAU_ORDER_AUTO ? opt.tau_order
                            : (2ull * eh.opaque_cores < n && depth >= 3u) ? VP_TAU_ORDER_NEAREST
                                                                         : VP_TAU_ORDER_LANE;
  v.tau_nearest = tau_order == VP_TAU_ORDER_NEAREST ? 1 : 0;
  vp_scene_info& info = sc->info;
  info.count = n;
  info.wide_nodes = wide_nodes;
  info.wide_depth = depth;
  info.binary_nodes = n > 1 ? n - 1 : 1;
  info.leaves = leaves;
  info.wide_builder = n <= kLeafMax ? opt.wide_builder : (wide_ploc ? VP_TREE_PLOC : VP_TREE_LBVH);
  info.binary_builder = bin_from_ploc ? VP_TREE_PLOC : VP_TREE_LBVH;
  info.binary_height = ploc_height;
  info.leaf_max = kLeafMax;
  info.wide_collapse = dp_used ? VP_COLLAPSE_SAH : VP_COLLAPSE_GREEDY;
  info.albedo_all_zero = v.albedo_all_zero;
  info.tau_order = tau_order;
  info.build_ms = ms;
  for (int k = 0; k < 3; ++k) {
    auto o2f = [](unsigned int u) {
      unsigned int b = (u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u;
      float f;
      std::memcpy(&f, &b, 4);
      return f;
    };
    info.bounds_min[k] = o2f(bh[6 + k]);
    info.bounds_max[k] = o2f(bh[9 + k]);
  }
  // records, order, per-Gaussian boxes, adjoint inputs, BVH32, binary tree, BVH8
  info.device_bytes = 64ull * n + 4ull * n + 32ull * n + 32ull * n + 1024ull * wide_nodes + 64ull * ni +
                      4ull * kNode8Words * nodes8;
  return VP_OK;
}

}  // namespace vp
