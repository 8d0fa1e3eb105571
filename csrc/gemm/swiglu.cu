// SwiGLU x routing-probability, forward and backward, as operations of their own (the expert MLP has both in epilogues
// of its GEMMs, which these are compared with), and the ungated activations, whose backward the expert MLP takes from here.
//   h = [gate | linear]  (bf16 [rows, 2F]),  act = silu(gate) * linear * p[row]
// Backward, given dact:  dp[row] = sum_f dact * silu(gate) * linear
//                         dlinear = dact * p * silu(gate)
//                         dgate   = dact * p * linear * sig(gate) * (1 + gate * (1 - sig(gate)))
// 16-byte accesses; a CTA per row forward, a warp (or a few) per row backward. Replaces the separate activation / multiply / cast kernels of
// `DeepEP_Megatron/test_deepep_moe_dispatch_combine.py:539-540,597-598` and their autograd twins.
#include <cuda_bf16.h>
#include "../common.cuh"
#include "gemm_api.h"
#include "act.cuh"

namespace b200ep {

__device__ __forceinline__ void unpack8(const uint4& v, float* f) {
  const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) { f[2 * q] = __uint_as_float(u[q] << 16); f[2 * q + 1] = __uint_as_float(u[q] & 0xffff0000u); }
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  uint4 o;
  uint32_t* u = &o.x;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * q], f[2 * q + 1]);
    u[q] = *reinterpret_cast<uint32_t*>(&h);
  }
  return o;
}

__global__ void __launch_bounds__(256)
swiglu_fwd_kernel(const char* __restrict__ h, const float* __restrict__ p, char* __restrict__ act,
                  const int* __restrict__ n_rows_ptr, int max_rows, int F) {
  const int rows = n_rows_ptr ? min(*n_rows_ptr, max_rows) : max_rows;
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    const float pr = p ? p[r] : 1.f;
    const char* g = h + (size_t)r * F * 4;          // 2F bf16 per row
    const char* l = g + (size_t)F * 2;
    char* o = act + (size_t)r * F * 2;
    for (int v = threadIdx.x; v < F / 8; v += blockDim.x) {
      float fg[8], fl[8], fo[8];
      unpack8(ld_global_nc_v4(g + ((size_t)v << 4)), fg);
      unpack8(ld_global_nc_v4(l + ((size_t)v << 4)), fl);
#pragma unroll
      for (int i = 0; i < 8; ++i) fo[i] = fg[i] / (1.f + __expf(-fg[i])) * fl[i] * pr;
      st_global_v4(o + ((size_t)v << 4), pack8(fo));
    }
  }
}

int launch_swiglu_fwd(const void* h, const float* p, void* act, const int* n_rows_ptr, int max_rows, int F,
                      cudaStream_t st) {
  if (F <= 0 || F % 8 || max_rows < 0) return 1;
  if (max_rows == 0) return 0;
  swiglu_fwd_kernel<<<min(max_rows, 148 * 16), 256, 0, st>>>(static_cast<const char*>(h), p, static_cast<char*>(act),
                                                             n_rows_ptr, max_rows, F);
  return 0;
}

// ---------------------------------------------------------------------------------------
// Ungated activations (gelu / silu / relu) x routing probability, forward and backward:
//   act = f(h) * p[row],   dh = dact * p * f'(h),   dp[row] = sum_f dact * f(h)
// kind: 0 gelu (erf form, as torch.nn.functional.gelu), 1 silu, 2 relu.
// (`DeepEP_Megatron/test_deepep_moe_dispatch_combine.py:516-526` offers these beside swiglu.)
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
act_fwd_kernel(const char* __restrict__ h, const float* __restrict__ p, char* __restrict__ act,
               const int* __restrict__ n_rows_ptr, int max_rows, int F, int kind) {
  const int rows = n_rows_ptr ? min(*n_rows_ptr, max_rows) : max_rows;
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    const float pr = p ? p[r] : 1.f;
    const char* g = h + (size_t)r * F * 2;
    char* o = act + (size_t)r * F * 2;
    for (int v = threadIdx.x; v < F / 8; v += blockDim.x) {
      float fg[8], fo[8];
      unpack8(ld_global_nc_v4(g + ((size_t)v << 4)), fg);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float f, df;
        act_eval(kind, fg[i], &f, &df);
        fo[i] = f * pr;
      }
      st_global_v4(o + ((size_t)v << 4), pack8(fo));
    }
  }
}

// ---------------------------------------------------------------------------------------
// Backward of both families. WPR warps share a row (a power of two up to the CTA's 8 warps); the sum of a
// row is a warp shuffle, plus one pass through shared memory when several warps share it.
// Bound: memory bandwidth (5 elements moved per output element with SwiGLU, 3 without). One warp per row
// keeps all loads of two vectors per operand in flight and needs no block barrier: with a CTA per row and two
// barriers 12001 rows of F = 1408 took 49.7 us and 8190 of F = 2048 39.4 us, now 37.3 and 35.3 (4.5 and 4.8 TB/s);
// 16384 of F = 14336 398 -> 389 us (6.0 TB/s), 512 of it 26.1 -> 25.1 (events around the call, inputs beyond L2). The
// gated forms of up to four warps a row spill 16 to 28 bytes a thread at the 64 registers that four CTAs per SM leave.
// ---------------------------------------------------------------------------------------
template <bool GATED>
__device__ __forceinline__ float bwd_vec(const uint4& vg, const uint4& vl, const uint4& vd, float pr, int kind, uint4* og, uint4* ol) {
  float fg[8], fl[8], fd[8], dg[8], dl[8], acc = 0.f;
  unpack8(vg, fg);
  if (GATED) unpack8(vl, fl);
  unpack8(vd, fd);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (GATED) {
      const float sig = 1.f / (1.f + __expf(-fg[i]));
      const float s = fg[i] * sig;
      acc += fd[i] * s * fl[i];
      const float da = fd[i] * pr;
      dl[i] = da * s;
      dg[i] = da * fl[i] * sig * (1.f + fg[i] * (1.f - sig));
    } else {
      float f, df;
      act_eval(kind, fg[i], &f, &df);
      acc += fd[i] * f;
      dg[i] = fd[i] * pr * df;
    }
  }
  *og = pack8(dg);
  if (GATED) *ol = pack8(dl);
  return acc;
}

constexpr int kBwdWarps = 8;

template <bool GATED, int WPR>
__global__ void __launch_bounds__(kBwdWarps * 32, 4)
act_bwd_rows_kernel(const char* __restrict__ h, const float* __restrict__ p, const char* __restrict__ dact,
                    char* __restrict__ dh, float* __restrict__ dp, const int* __restrict__ n_rows_ptr,
                    int max_rows, int F, int kind) {
  __shared__ float s_part[kBwdWarps];
  constexpr int ROWS = kBwdWarps / WPR;                      // rows of a CTA at a time
  const int rows = n_rows_ptr ? min(*n_rows_ptr, max_rows) : max_rows;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = warp % WPR;
  const int nvec = F / 8;
  const size_t ld = (size_t)F * (GATED ? 4 : 2);             // bytes of a row of h / dh
  for (int r0 = blockIdx.x * ROWS; r0 < rows; r0 += gridDim.x * ROWS) {
    const int r = r0 + warp / WPR;
    float acc = 0.f;
    if (r < rows) {
      const float pr = p ? p[r] : 1.f;
      const char* g = h + (size_t)r * ld;
      const char* l = g + (size_t)F * 2;
      const char* d = dact + (size_t)r * F * 2;
      char* og = dh + (size_t)r * ld;
      char* ol = og + (size_t)F * 2;
      constexpr int U = WPR == kBwdWarps ? 1 : 2, STEP = 32 * WPR;     // a CTA per row: more CTAs rather than deeper loads (512 x 14336, kernel alone: 16.5 -> 15.9 us)
      for (int v0 = sub * 32 + lane; v0 < nvec; v0 += U * STEP) {
        uint4 vg[U], vl[U], vd[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const size_t at = (size_t)(v0 + u * STEP) << 4;
          if (v0 + u * STEP < nvec) {
            vg[u] = ld_global_nc_v4(g + at);
            if (GATED) vl[u] = ld_global_nc_v4(l + at);
            vd[u] = ld_global_nc_v4(d + at);
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const size_t at = (size_t)(v0 + u * STEP) << 4;
          if (v0 + u * STEP < nvec) {
            uint4 o1, o2;
            acc += bwd_vec<GATED>(vg[u], vl[u], vd[u], pr, kind, &o1, &o2);
            st_global_v4(og + at, o1);
            if (GATED) st_global_v4(ol + at, o2);
          }
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (WPR > 1) {
      if (lane == 0) s_part[warp] = acc;
      __syncthreads();
      if (sub == 0) {
        acc = 0.f;
#pragma unroll
        for (int w = 0; w < WPR; ++w) acc += s_part[warp + w];
      }
      __syncthreads();
    }
    if (sub == 0 && lane == 0 && r < rows && dp != nullptr) dp[r] = acc;
  }
}

template <bool GATED>
static void launch_bwd_rows(const void* h, const float* p, const void* dact, void* dh, float* dp, const int* n_rows_ptr,
                            int max_rows, int F, int kind, cudaStream_t st) {
  const char *hc = static_cast<const char*>(h), *dc = static_cast<const char*>(dact);
  char* oc = static_cast<char*>(dh);
  // Warps per row: one as long as the rows alone fill the GPU (16 warps on each of 148 SMs), more for fewer rows, no
  // more than the row has batches of 32 vectors.
  int wpr = 1;
  while (wpr < kBwdWarps && (long long)max_rows * wpr < 148 * 16 && F / 8 > 32 * wpr) wpr *= 2;
  const int per = kBwdWarps / wpr;
  const int grid = min((max_rows + per - 1) / per, 148 * 8);
  if (wpr == 1) act_bwd_rows_kernel<GATED, 1><<<grid, kBwdWarps * 32, 0, st>>>(hc, p, dc, oc, dp, n_rows_ptr, max_rows, F, kind);
  else if (wpr == 2) act_bwd_rows_kernel<GATED, 2><<<grid, kBwdWarps * 32, 0, st>>>(hc, p, dc, oc, dp, n_rows_ptr, max_rows, F, kind);
  else if (wpr == 4) act_bwd_rows_kernel<GATED, 4><<<grid, kBwdWarps * 32, 0, st>>>(hc, p, dc, oc, dp, n_rows_ptr, max_rows, F, kind);
  else act_bwd_rows_kernel<GATED, 8><<<grid, kBwdWarps * 32, 0, st>>>(hc, p, dc, oc, dp, n_rows_ptr, max_rows, F, kind);
}

int launch_swiglu_bwd(const void* h, const float* p, const void* dact, void* dh, float* dp, const int* n_rows_ptr,
                      int max_rows, int F, cudaStream_t st) {
  if (F <= 0 || F % 8 || max_rows < 0) return 1;
  if (max_rows == 0) return 0;
  launch_bwd_rows<true>(h, p, dact, dh, dp, n_rows_ptr, max_rows, F, 0, st);
  return 0;
}

// The parts of a row are 128 columns each, one row of `part` per part, so that neighbouring threads read neighbouring
// words: 12001 rows x 11 parts are half a megabyte, a launch of 3.9 us.
__global__ void __launch_bounds__(256)
sum_parts_kernel(const float* __restrict__ part, int parts, int rows, float* __restrict__ dp) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  float s = 0.f;
#pragma unroll 8
  for (int b = 0; b < parts; ++b) s += __ldg(part + (size_t)b * rows + r);
  dp[r] = s;
}

int launch_sum_parts(const float* part, int parts, int rows, float* dp, cudaStream_t st) {
  if (parts < 1 || rows < 0) return 1;
  if (rows > 0) sum_parts_kernel<<<(rows + 255) / 256, 256, 0, st>>>(part, parts, rows, dp);
  return 0;
}

int launch_act_fwd(const void* h, const float* p, void* act, const int* n_rows_ptr, int max_rows, int F, int kind,
                   cudaStream_t st) {
  if (F <= 0 || F % 8 || max_rows < 0 || kind < 0 || kind > 2) return 1;
  if (max_rows == 0) return 0;
  act_fwd_kernel<<<min(max_rows, 148 * 16), 256, 0, st>>>(static_cast<const char*>(h), p, static_cast<char*>(act),
                                                          n_rows_ptr, max_rows, F, kind);
  return 0;
}

int launch_act_bwd(const void* h, const float* p, const void* dact, void* dh, float* dp, const int* n_rows_ptr,
                   int max_rows, int F, int kind, cudaStream_t st) {
  if (F <= 0 || F % 8 || max_rows < 0 || kind < 0 || kind > 2) return 1;
  if (max_rows == 0) return 0;
  launch_bwd_rows<false>(h, p, dact, dh, dp, n_rows_ptr, max_rows, F, kind, st);
  return 0;
}

}  // namespace b200ep
