// One launch that copies up to eight buffers of this GPU: the owned copies of a dispatch's rows and side
// arrays (DeepEP's outputs are tensors of the caller, `DeepEP_v1/deepep_v1_dispatch.py:212-230`, here they
// first arrive in the symmetric region).
// Bound: memory bandwidth for the rows, launch latency for the rest: four separate device copies cost four
// launches, and rows of 67 MB took 24 us; this launch takes 19 us for them (7 TB/s), and 1.8 us instead
// of 7 for the four small arrays of 96 tokens (one B200).
#include "api.h"

namespace b200ep {

constexpr int kCloneThreads = 256, kCloneVecs = 4;
constexpr int kCloneChunk = kCloneThreads * kCloneVecs * 16;      // bytes that a CTA copies at a time

__global__ void __launch_bounds__(kCloneThreads)
clone_kernel(const __grid_constant__ CloneArgs a) {
  stream_order_wait();
  stream_order_next();
  const int total = a.first_chunk[a.n];
  for (int c = blockIdx.x; c < total; c += gridDim.x) {
    int s = 0;
    while (c >= a.first_chunk[s + 1]) ++s;
    const long long off = (long long)(c - a.first_chunk[s]) * kCloneChunk;
    const long long left = a.bytes[s] - off;
    const char* src = a.src[s] + off;
    char* dst = a.dst[s] + off;
    const int nvec = (int)((left < kCloneChunk ? left : kCloneChunk) >> 4);
    uint4 v[kCloneVecs];
#pragma unroll
    for (int u = 0; u < kCloneVecs; ++u) {
      const int i = u * kCloneThreads + threadIdx.x;
      if (i < nvec) v[u] = ld_global_v4(src + ((size_t)i << 4));      // peers wrote the region: coherent path
    }
#pragma unroll
    for (int u = 0; u < kCloneVecs; ++u) {
      const int i = u * kCloneThreads + threadIdx.x;
      if (i < nvec) st_global_v4(dst + ((size_t)i << 4), v[u]);
    }
    if (left < kCloneChunk)                                            // bytes behind the last whole vector
      for (int i = (nvec << 4) + threadIdx.x; i < (int)left; i += kCloneThreads) dst[i] = src[i];
  }
}

int launch_clone(CloneArgs a, cudaStream_t st) {
  if (a.n < 0 || a.n > kMaxClones) return 1;
  long long chunks = 0;
  for (int s = 0; s < a.n; ++s) {
    if (a.bytes[s] < 0 || ((reinterpret_cast<uintptr_t>(a.src[s]) | reinterpret_cast<uintptr_t>(a.dst[s])) & 15)) return 1;
    a.first_chunk[s] = (int)chunks;
    chunks += (a.bytes[s] + kCloneChunk - 1) / kCloneChunk;
    if (chunks > 0x7fffffff) return 1;
  }
  a.first_chunk[a.n] = (int)chunks;
  if (chunks == 0) return 0;
  const int grid = (int)(chunks < 148 * 8 ? chunks : 148 * 8);
  launch_ordered(clone_kernel, grid, kCloneThreads, 0, st, 1, a);
  return 0;
}

}  // namespace b200ep
