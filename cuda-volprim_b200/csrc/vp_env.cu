// Environment-map build on the device: RGBA texels for the bilinear lookup, the
// luminance x sin(theta) sampling weights in FP64, a Vose alias table per row and one over the
// rows.  Replaces the reference's host FP32 2-D CDF (EnvironmentMap::buildCdf,
// include/thesis/host/params/environment_map.h:45-101) and texture upload (:105-151); the
// sampled distribution and its pdf are the same (proportional to joint texel weight).
#include <algorithm>
#include <cmath>
#include <vector>

#include "vp_internal.h"

namespace vp {
namespace {

// Texel weight = Rec.709 luminance x sin(theta at the row centre), environment_map.h:51-66.
__global__ void k_env_texels(uint32_t W, uint32_t H, uint32_t ch, const float* __restrict__ rgb,
                             float4* __restrict__ tex, double* __restrict__ wts,
                             float* __restrict__ joint) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)W * H) return;
  const uint32_t v = (uint32_t)(i / W);
  const float* px = rgb + i * ch;
  const float r = px[0];
  const float g = ch >= 2 ? px[1] : r;
  const float b = ch >= 3 ? px[2] : r;
  const float a = ch >= 4 ? px[3] : 1.0f;
  tex[i] = make_float4(r, g, b, a);
  const double theta = ((double)v + 0.5) / (double)H * 3.14159265358979323846;
  const double lum = 0.2126 * (double)r + 0.7152 * (double)g + 0.0722 * (double)b;
  const double wgt = lum * sin(theta);
  wts[i] = wgt;
  joint[i] = (float)wgt;
}

__global__ void k_row_sums(uint32_t W, const double* __restrict__ wts, double* __restrict__ rows) {
  const uint32_t v = blockIdx.x;
  double s = 0.0;
  for (uint32_t u = threadIdx.x; u < W; u += blockDim.x) s += wts[(size_t)v * W + u];
  __shared__ double red[256];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) rows[v] = red[0];
}

// Vose's alias method over n weights by one warp, FP64 probabilities.  p and idx (n entries each) are scratch,
// in shared memory where a table fits (kAliasSmem), else global.
//
// Entries below 1 ("small") and the others ("large") are stacks in index order; each step pairs the top
// small l with the top large g, which loses what l lacks and, once below 1, becomes the top small.  So one
// lane runs the chain p[g] = (p[g] + p[l]) - 1 with p[g], and p[l] while it is such a g, in registers: what
// is serial is two FP64 additions and a shared-memory load a step.  The warp scales the weights and splits
// them beforehand and writes what is left over afterwards.  A thread per table with its stacks in global
// memory took 1.25 ms for 1024 rows of 2048; this takes 0.13.
constexpr size_t kAliasSmem = 200 * 1024;
constexpr uint32_t kNoEntry = 0xFFFFFFFFu;

__device__ void vose(uint32_t n, const double* __restrict__ w, double sum, double* p, uint32_t* idx,
                     float2* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  if (!(sum > 0.0)) {
    for (uint32_t u = lane; u < n; u += 32u) out[u] = make_float2(1.0f, __uint_as_float(u));
    return;
  }
  // idx: smalls from the front, larges from the back
  uint32_t ns = 0, nl = 0;
  const double scale = (double)n / sum;
  for (uint32_t b = 0; b < n; b += 32u) {
    const uint32_t u = b + lane;
    double v = 0.0;
    if (u < n) p[u] = v = w[u] * scale;
    const unsigned sm = __ballot_sync(0xFFFFFFFFu, u < n && v < 1.0), in = __ballot_sync(0xFFFFFFFFu, u < n);
    const unsigned lm = in & ~sm, lt = (1u << lane) - 1u;
    if ((sm >> lane) & 1u) idx[ns + __popc(sm & lt)] = u;
    if ((lm >> lane) & 1u) idx[n - 1u - (nl + __popc(lm & lt))] = u;
    ns += __popc(sm);
    nl += __popc(lm);
  }
  __syncwarp();
  uint32_t g = kNoEntry, carry = kNoEntry;  // the top large; a g that became small
  if (lane == 0 && ns > 0u && nl > 0u) {
    double pg = 0.0, pc = 0.0;
    g = idx[n - nl--];
    pg = p[g];
    while (ns > 0u || carry != kNoEntry) {
      uint32_t l;
      double pl;
      if (carry != kNoEntry) {
        l = carry;
        pl = pc;
        carry = kNoEntry;
      } else {
        l = idx[--ns];
        pl = p[l];
      }
      out[l] = make_float2((float)pl, __uint_as_float(g));
      pg = (pg + pl) - 1.0;
      if (pg < 1.0) {
        carry = g;
        pc = pg;
        g = kNoEntry;
        if (nl == 0u) break;
        g = idx[n - nl--];
        pg = p[g];
      }
    }
  }
  ns = __shfl_sync(0xFFFFFFFFu, ns, 0);
  nl = __shfl_sync(0xFFFFFFFFu, nl, 0);
  if (lane == 0) {
    if (g != kNoEntry) out[g] = make_float2(1.0f, __uint_as_float(g));
    if (carry != kNoEntry) out[carry] = make_float2(1.0f, __uint_as_float(carry));
  }
  for (uint32_t k = lane; k < nl; k += 32u) {
    const uint32_t u = idx[n - nl + k];
    out[u] = make_float2(1.0f, __uint_as_float(u));
  }
  for (uint32_t k = lane; k < ns; k += 32u) {
    const uint32_t u = idx[k];
    out[u] = make_float2(1.0f, __uint_as_float(u));
  }
}

// Block v < H: the table of row v; block H: the marginal table over the rows and the total weight.  kSmem: the
// scratch of every table is in shared memory; else in p and idx, H rows of W and then one of H.
template <bool kSmem>
__global__ void __launch_bounds__(32) k_alias(uint32_t W, uint32_t H, const double* __restrict__ wts,
                        const double* __restrict__ rows, double* __restrict__ p, uint32_t* __restrict__ idx,
                        float2* __restrict__ cond, float2* __restrict__ marg, double* __restrict__ total) {
  extern __shared__ __align__(16) unsigned char scratch[];
  const uint32_t v = blockIdx.x;
  const uint32_t n = v < H ? W : H;
  const size_t o = (size_t)v * W;
  double* pp = kSmem ? reinterpret_cast<double*>(scratch) : p + o;
  uint32_t* ii = kSmem ? reinterpret_cast<uint32_t*>(scratch + sizeof(double) * n) : idx + o;
  if (v < H) {
    vose(W, wts + o, rows[v], pp, ii, cond + o);
    return;
  }
  for (uint32_t u = threadIdx.x; u < H; u += 32u) pp[u] = rows[u];
  __syncwarp();
  double s = 0.0;
  for (uint32_t u = 0; u < H; ++u) s += pp[u];  // every lane, in row order
  if (threadIdx.x == 0) *total = s;
  __syncwarp();
  vose(H, rows, s, pp, ii, marg);
}

}  // namespace

vp_status build_env(vp_context* ctx, const float* rgb, uint32_t W, uint32_t H, uint32_t ch,
                    int32_t memory, vp_env* env) {
  cudaStream_t st = ctx->stream;
  if (!rgb || W == 0 || H == 0) return fail(VP_ERROR_INVALID_ARGUMENT, "environment map is empty");
  if (ch < 1 || ch > 4) return fail(VP_ERROR_INVALID_ARGUMENT, "environment channels must be 1..4");
  if ((uint64_t)W * H >= (1ull << 31)) return fail(VP_ERROR_LIMIT, "environment map too large");
  const size_t n = (size_t)W * H;
  VP_CUDA(cudaEventRecord(ctx->ev0, st));
  vp_status s;
  float* d_rgb = nullptr;
  const float* src = rgb;
  if (memory == VP_MEMORY_HOST) {
    if ((s = dev_alloc(&d_rgb, n * ch, st))) return s;
    VP_CUDA(cudaMemcpyAsync(d_rgb, rgb, n * ch * sizeof(float), cudaMemcpyHostToDevice, st));
    src = d_rgb;
  } else if (memory != VP_MEMORY_DEVICE) {
    return fail(VP_ERROR_INVALID_ARGUMENT, "memory must be VP_MEMORY_HOST or VP_MEMORY_DEVICE");
  }
  double *wts = nullptr, *rows = nullptr, *p = nullptr, *total = nullptr;
  uint32_t* idx = nullptr;
  const size_t alias_smem = (size_t)std::max(W, H) * (sizeof(double) + sizeof(uint32_t));
  const bool in_smem = alias_smem <= kAliasSmem;
  auto cleanup = [&]() {
    dev_free(d_rgb, st);
    dev_free(wts, st);
    dev_free(rows, st);
    dev_free(p, st);
    dev_free(total, st);
    dev_free(idx, st);
  };
  if ((s = dev_alloc(&env->texels, n, st)) || (s = dev_alloc(&env->joint, n, st)) ||
      (s = dev_alloc(&env->cond, n, st)) || (s = dev_alloc(&env->marg, H, st)) ||
      (s = dev_alloc(&wts, n, st)) || (s = dev_alloc(&rows, H, st)) || (s = dev_alloc(&total, 1, st)) ||
      (!in_smem && ((s = dev_alloc(&p, n + H, st)) || (s = dev_alloc(&idx, n + H, st))))) {
    cleanup();
    return s;
  }
  k_env_texels<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(W, H, ch, src, env->texels, wts, env->joint);
  k_row_sums<<<H, 256, 0, st>>>(W, wts, rows);
  cudaError_t e = cudaSuccess;
  auto alias = in_smem ? k_alias<true> : k_alias<false>;
  if (in_smem && alias_smem > 48 * 1024)
    e = cudaFuncSetAttribute(alias, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)alias_smem);
  if (e == cudaSuccess) {
    alias<<<H + 1u, 32, in_smem ? alias_smem : 0, st>>>(W, H, wts, rows, p, idx, env->cond, env->marg, total);
    e = cudaGetLastError();
  }
  double tot = 0.0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&tot, total, sizeof(double), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaEventRecord(ctx->ev1, st);
  cleanup();
  if (e == cudaSuccess) e = cudaEventSynchronize(ctx->ev1);
  if (e != cudaSuccess) return cuda_fail(e, "environment build");
  float ms = 0.f;
  VP_CUDA(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
  env->ctx = ctx;
  env->build_ms = ms;
  EnvView& v = env->view;
  v.texels = env->texels;
  v.cond = env->cond;
  v.marg = env->marg;
  v.joint = env->joint;
  v.width = W;
  v.height = H;
  v.total = (float)tot;
  v.inv_total = tot > 0.0 ? (float)(1.0 / tot) : 0.0f;
  return VP_OK;
}

}  // namespace vp
