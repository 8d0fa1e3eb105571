// Router of an inference MoE layer: logits = x . W^T in f32 (x bf16 as it is, W f32), softmax over the experts,
// top-k, weights renormalised over the chosen experts
// (`DeepEP_Megatron/test_deepep_moe_dispatch_combine.py:731-742` draws its routing at random instead).
// Two launches: partial products of a part of the reduction per CTA, then one warp per token that adds the
// parts in order, takes the softmax and picks the experts. The f32 arithmetic stays f32 (no tensor cores).
// Bound: f32 FMA rate for many tokens, latency for few. The library path cast x to f32, ran one 64 x 64
// tile per CTA over the whole reduction (16 CTAs for 1024 tokens x 64 experts) and five more kernels: 70 us, now
// 21 us (one B200, 1024 x 2048, 64 experts, top-8).
#include <cuda_bf16.h>
#include "../common.cuh"
#include "gemm_api.h"

namespace b200ep {

namespace router {

constexpr int TT = 64, TE = 64, KC = 32, LD = TT + 4;      // tokens, experts and reduction indices of a tile; smem row

// part[s][t][e] = sum over the reduction indices of split s. Thread (ty, tx): 4 tokens x 4 experts.
__global__ void __launch_bounds__(256)
partial_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ w, float* __restrict__ part,
               int T, int E, int H, int k_per) {
  __shared__ __align__(16) float xs[KC][LD], ws[KC][LD];
  const int t0 = blockIdx.x * TT, e0 = blockIdx.y * TE, s = blockIdx.z;
  const int k_lo = s * k_per, k_hi = min(H, k_lo + k_per);
  const int row = threadIdx.x & 63, q = threadIdx.x >> 6;   // loader: row of the tile, 8 reduction indices from 8 * q
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  const bool t_ok = t0 + row < T, e_ok = e0 + row < E;
  const __nv_bfloat16* xr = x + (size_t)(t0 + row) * H;
  const float* wr = w + (size_t)(e0 + row) * H;
  uint4 xv, wv0, wv1;
  auto fetch = [&](int k0) {
    const int k = k0 + 8 * q;                               // (H and k_per are multiples of 8)
    xv = wv0 = wv1 = make_uint4(0, 0, 0, 0);
    if (k < k_hi) {
      if (t_ok) xv = ld_global_nc_v4(xr + k);
      if (e_ok) { wv0 = ld_global_nc_v4(wr + k); wv1 = ld_global_nc_v4(wr + k + 4); }
    }
  };
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  fetch(k_lo);
  for (int k0 = k_lo; k0 < k_hi; k0 += KC) {
    const uint32_t xu[4] = {xv.x, xv.y, xv.z, xv.w};
    const uint32_t wu[8] = {wv0.x, wv0.y, wv0.z, wv0.w, wv1.x, wv1.y, wv1.z, wv1.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      xs[8 * q + 2 * i][row] = __uint_as_float(xu[i] << 16);
      xs[8 * q + 2 * i + 1][row] = __uint_as_float(xu[i] & 0xffff0000u);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) ws[8 * q + i][row] = __uint_as_float(wu[i]);
    __syncthreads();
    if (k0 + KC < k_hi) fetch(k0 + KC);                     // in flight while this chunk is multiplied
#pragma unroll
    for (int k = 0; k < KC; ++k) {
      const float4 a = *reinterpret_cast<const float4*>(&xs[k][4 * ty]);
      const float4 b = *reinterpret_cast<const float4*>(&ws[k][4 * tx]);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = t0 + 4 * ty + i;
    if (t >= T) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (e0 + 4 * tx + j < E) part[((size_t)s * T + t) * E + e0 + 4 * tx + j] = acc[i][j];
  }
}

// Total order of the logits as unsigned keys: NaN above everything (as torch.topk ranks it), 0 is taken or absent.
__device__ __forceinline__ uint32_t key_of(float v) {
  if (v != v) return 0xffffffffu;
  const uint32_t u = __float_as_uint(v);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// One warp per token; lane l holds the logits of experts l, l + 32, ... Softmax is monotone, so the largest
// probabilities are those of the largest logits; equal logits go to the lower expert id.
template <int VPL>
__global__ void __launch_bounds__(256)
topk_kernel(const float* __restrict__ part, int splits, int T, int E, int K, long long* __restrict__ idx,
            float* __restrict__ prob) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * 8 + warp;
  if (t >= T) return;
  float v[VPL];
  uint32_t key[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) v[i] = 0.f;
  for (int s = 0; s < splits; ++s) {
    const float* p = part + ((size_t)s * T + t) * E;
#pragma unroll
    for (int i = 0; i < VPL; ++i)
      if (i * 32 + lane < E) v[i] += p[i * 32 + lane];
  }
  float top = -INFINITY;
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const bool in = i * 32 + lane < E;
    key[i] = in ? key_of(v[i]) : 0u;
    if (in) top = fmaxf(top, v[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < VPL; ++i)
    if (i * 32 + lane < E) { v[i] = expf(v[i] - top); sum += v[i]; }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  float mine = 0.f, chosen = 0.f;                           // lane k: probability of choice k; sum over the choices
  int mine_e = 0;
  for (int k = 0; k < K; ++k) {
    uint32_t best = 0;
    int at = 0;
#pragma unroll
    for (int i = 0; i < VPL; ++i)
      if (key[i] > best) { best = key[i]; at = i; }
    const uint32_t high = __reduce_max_sync(0xffffffffu, best);
    const uint32_t e = __reduce_min_sync(0xffffffffu, best == high ? (uint32_t)(at * 32 + lane) : 0xffffffffu);
    float p = 0.f;
    if ((int)(e & 31) == lane) {
#pragma unroll
      for (int i = 0; i < VPL; ++i)
        if (i == (int)(e >> 5)) { p = v[i] / sum; key[i] = 0u; }
    }
    p = __shfl_sync(0xffffffffu, p, e & 31);
    chosen += p;
    if (lane == k) { mine = p; mine_e = (int)e; }
  }
  if (lane < K) {
    idx[(size_t)t * K + lane] = mine_e;
    prob[(size_t)t * K + lane] = mine / chosen;
  }
}

// Backward of topk_kernel for one token and warp. The renormalised weights are a softmax over the chosen logits alone:
// d logit_k = w_k * (g_k - sum_j w_j g_j), nothing for the others (not a number for all of them where the sum is none).
// With topk_kernel in the forward: 55.5 us of library kernels a training step -> 8.4 (4095 tokens, top-2 of 8; one B200).
__global__ void __launch_bounds__(256)
topk_bwd_kernel(const long long* __restrict__ idx, const float* __restrict__ w, const float* __restrict__ gw, int T, int E,
                int K, float* __restrict__ dlogits) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * 8 + warp;
  if (t >= T) return;
  float wk = 0.f, gk = 0.f;
  int e = -1;
  if (lane < K) {
    const size_t at = (size_t)t * K + lane;
    wk = w[at];
    gk = gw[at];
    const long long i = idx[at];
    e = i >= 0 && i < E ? (int)i : -1;
  }
  float s = lane < K ? wk * gk : 0.f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  float* row = dlogits + (size_t)t * E;
  const float rest = s - s;                                 // 0, or not a number
  for (int i = lane; i < E; i += 32) row[i] = rest;
  __syncwarp();
  if (e >= 0) row[e] = wk * (gk - s);
}

}  // namespace router

int launch_router_topk_bwd(const long long* idx, const float* w, const float* gw, int T, int E, int K, float* dlogits, cudaStream_t st) {
  if (T < 0 || E < 1 || K < 1 || K > 32) return 1;
  if (T > 0) router::topk_bwd_kernel<<<(T + 7) / 8, 256, 0, st>>>(idx, w, gw, T, E, K, dlogits);
  return 0;
}

int router_splits(int T, int E, int H) {
  // parts of the reduction: enough CTAs for two on every SM, each with at least 128 indices
  const long long tiles = (long long)((T + router::TT - 1) / router::TT) * ((E + router::TE - 1) / router::TE);
  int s = (int)(296 / (tiles > 0 ? tiles : 1));
  const int most = H / 128 < 1 ? 1 : (H / 128 > 32 ? 32 : H / 128);
  s = s < 1 ? 1 : (s > most ? most : s);
  const int per = ((H + s - 1) / s + router::KC - 1) / router::KC * router::KC;
  return (H + per - 1) / per;
}

int launch_router_logits(const void* x, const float* w, float* part, int splits, int T, int E, int H, cudaStream_t st) {
  if (T < 0 || E < 1 || H < 8 || H % 8 || splits < 1) return 1;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) return 1;
  if (T == 0) return 0;
  const int per = ((H + splits - 1) / splits + router::KC - 1) / router::KC * router::KC;
  const dim3 grid((T + router::TT - 1) / router::TT, (E + router::TE - 1) / router::TE, splits);
  router::partial_kernel<<<grid, 256, 0, st>>>(static_cast<const __nv_bfloat16*>(x), w, part, T, E, H, per);
  return 0;
}

int launch_router_topk(const float* part, int splits, int T, int E, int K, long long* idx, float* prob, cudaStream_t st) {
  if (T < 0 || E < 1 || E > kRouterMaxExperts || K < 1 || K > 32 || K > E || splits < 1) return 1;
  if (T == 0) return 0;
  const int grid = (T + 7) / 8;
  if (E <= 64) router::topk_kernel<2><<<grid, 256, 0, st>>>(part, splits, T, E, K, idx, prob);
  else if (E <= 256) router::topk_kernel<8><<<grid, 256, 0, st>>>(part, splits, T, E, K, idx, prob);
  else router::topk_kernel<32><<<grid, 256, 0, st>>>(part, splits, T, E, K, idx, prob);
  return 0;
}

}  // namespace b200ep
