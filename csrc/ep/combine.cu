// Normal-mode combine. Replaces `Buffer.combine` as consumed by
// `DeepEP_v1/deepep_v1_combine.py:241-247` and the index_add_ unpermute of
// `DeepEP_Megatron/test_deepep_moe_dispatch_combine.py:390-403`. Two forms:
//
// PULL (rows inside the producer's symmetric region, e.g. the zero-copy output of dispatch):
//   every rank announces where its rows are, waits (bounded) for the peers' announcements and
//   LOADS the rows of its own tokens over NVLink, reducing them in fp32 registers on the way:
//   one pass, no slot region, nothing left to do when the last row has arrived.
// PUSH (rows anywhere): every received row is stored into its slot on the source rank with LSU
//   peer stores; when its own rows are out a CTA waits (bounded) for the peers' flags and reduces
//   the slots of this rank's tokens. Rows whose source is this rank itself take no slot: they are
//   read where they lie, so a group of one neither sends nor waits. The fc2 GEMM epilogue of
//   csrc/gemm stores its tiles into the same slots and is followed by the reduce role alone.
//
// What was measured and dropped: cutting the push into token chunks with one flag per chunk, so
// that the reduction of chunk c overlaps the arrival of chunk c+1. Any release fence on an SM
// whose store queue is full of NVLink stores drains that queue first (tens of microseconds at a
// per-SM share of the link of about 5 GB/s); with 8 ranks the send went from 413 to 587 us with
// one fence per CTA and chunk and to 654 us with the reduction running beside it, against 519 us
// for send-then-reduce. The pull form gets the overlap without any fence.
//
// Bound: memory (or NVLink) bandwidth; every reduction asks for the indices of a warp's next item
// before it loads the rows of the current one, and few tokens are cut into more parts per row on
// smaller CTAs. Measured on one B200, before and after: push of 2047 tokens x 8 rows of 14 KiB
// 133 -> 57 us (the slot round trip is gone) -> 49 us (rows not allocated in L1; 5.4 TB/s), push of 96
// rows of 2 KiB 14.7 -> 3.7 us, pull of 4096 rows of 14 KiB 27.3 -> 22.8 -> 21.7 us. Tried and slower: half the
// warps with one or two steps of loads requested ahead (58 us for the first), rows brought to a ring in shared memory by bulk
// copies (55). Twice the loads in flight leave the push at 49 us: with the 117 MB that the dispatch before it left to be
// written back it is HBM that bounds it. One CTA of up to 1024 threads per SM: 64 registers a thread, at which the 16-bit
// forms for up to four contributors spill 8 to 84 bytes a thread (76 to 84 for two). With several virtual ranks on one
// GPU the halves that wait for peers are launched after the halves they wait for (all announcements / sends first).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include "ep.cuh"
#include "api.h"

namespace b200ep {

constexpr int kCombWarps = 32;   // one CTA of 1024 threads per SM
constexpr int kCUnroll = 4;
// Loads that a lane has in flight in a reduction, and the running sums that go with them, as a token's contributors J
// allow: U vectors of each of G contributors, 64 registers a thread in all. One contributor needs no sums (4096 rows of
// 14 KiB, pull: 24.8 -> 22.8 us on a device timeline); eight rows of a vector at a time need the sums of that vector only (1024
// tokens x 8 rows of 4 KiB: 10.7 -> 8.5 us; 2047 x 8 of 14 KiB stay at 49, HBM with what the dispatch left to be written back).
template <int FORM> struct Batch;
template <> struct Batch<0> { static constexpr int U = 4, G = 1; };     // J == 2
template <> struct Batch<1> { static constexpr int U = 8, G = 1; };     // J == 1
template <> struct Batch<2> { static constexpr int U = 2, G = 4; };     // J == 3, 4
template <> struct Batch<3> { static constexpr int U = 1, G = 8; };     // J >= 5
static int batch_form(int J) { return J == 1 ? 1 : J == 2 ? 0 : J <= 4 ? 2 : 3; }

// ---- element helpers -------------------------------------------------------------------
template <typename T> struct Vec16;
template <> struct Vec16<__nv_bfloat16> {
  static constexpr int N = 8;
  static __device__ __forceinline__ void acc(float* a, const uint4& v, float w) {
    const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      a[2 * q] += w * __uint_as_float(u[q] << 16);
      a[2 * q + 1] += w * __uint_as_float(u[q] & 0xffff0000u);
    }
  }
  static __device__ __forceinline__ uint4 pack(const float* a) {
    uint4 o;
    uint32_t* u = &o.x;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      __nv_bfloat162 h = __floats2bfloat162_rn(a[2 * q], a[2 * q + 1]);
      u[q] = *reinterpret_cast<uint32_t*>(&h);
    }
    return o;
  }
};
template <> struct Vec16<__half> {
  static constexpr int N = 8;
  static __device__ __forceinline__ void acc(float* a, const uint4& v, float w) {
    const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const __half2 h = *reinterpret_cast<const __half2*>(&u[q]);
      const float2 f = __half22float2(h);
      a[2 * q] += w * f.x;
      a[2 * q + 1] += w * f.y;
    }
  }
  static __device__ __forceinline__ uint4 pack(const float* a) {
    uint4 o;
    uint32_t* u = &o.x;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      __half2 h = __floats2half2_rn(a[2 * q], a[2 * q + 1]);
      u[q] = *reinterpret_cast<uint32_t*>(&h);
    }
    return o;
  }
};
template <> struct Vec16<float> {
  static constexpr int N = 4;
  static __device__ __forceinline__ void acc(float* a, const uint4& v, float w) {
    a[0] += w * __uint_as_float(v.x);
    a[1] += w * __uint_as_float(v.y);
    a[2] += w * __uint_as_float(v.z);
    a[3] += w * __uint_as_float(v.w);
  }
  static __device__ __forceinline__ uint4 pack(const float* a) {
    return make_uint4(__float_as_uint(a[0]), __float_as_uint(a[1]), __float_as_uint(a[2]),
                      __float_as_uint(a[3]));
  }
};


// ---- push form: send role ------------------------------------------------------------------
__device__ __forceinline__ void combine_copy_row(const CombineArgs& a, const EpGeom& g, const EpRegions& rg,
                                                 const PeerPtrs& peers, int row, int lane, int* status) {
  const int2 meta = a.recv_meta[row];
  const int slot = meta.x, s = meta.y;
  if (a.send_row != nullptr && s == g.rank) return;      // the reduce role reads it in place
  if (s < 0 || s >= g.R || slot < 0 || slot >= g.slot_cap) {
    if (lane == 0) set_status(status, kOverflowSlots);
    return;
  }
  const int nvec = a.row_bytes >> 4;
  char* pb = peers.base[s];
  char* dst = pb + rg.comb_x + (size_t)slot * a.row_bytes;
  const char* src = a.x + (size_t)row * a.row_bytes;
  for (int v0 = 0; v0 < nvec; v0 += 32 * kCUnroll) {
    uint4 buf[kCUnroll];
#pragma unroll
    for (int u = 0; u < kCUnroll; ++u) {
      const int v = v0 + u * 32 + lane;
      if (v < nvec) buf[u] = ld_global_nc_v4(src + ((size_t)v << 4));
    }
#pragma unroll
    for (int u = 0; u < kCUnroll; ++u) {
      const int v = v0 + u * 32 + lane;
      if (v < nvec) st_global_v4(dst + ((size_t)v << 4), buf[u]);
    }
  }
  // side values returned with the row: K floats per row in rank mode, one in expert mode
  const int wk = g.mode == 0 ? g.K : 1;
  if (a.topk_w != nullptr && lane < wk)
    reinterpret_cast<float*>(pb + rg.comb_w)[(size_t)slot * wk + lane] = a.topk_w[(size_t)row * wk + lane];
}

__device__ void combine_send_role(const CombineArgs& a, const EpGeom& g, const EpRegions& rg,
                                  const PeerPtrs& peers, int* status) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  // item index: neighbouring rows (same peer: rows are grouped by source rank or by expert) land on
  // DIFFERENT CTAs, so every SM stores to a mix of peers instead of one SM group per peer; a warp's
  // rows are spread over the whole range, so at any instant all peers are addressed in proportion
  const int gw = warp * gridDim.x + blockIdx.x, nw = gridDim.x * nwarps;
  int n = *a.n_recv_ptr;
  if (n > g.cap) n = g.cap;
  for (int i = gw; i < n; i += nw) combine_copy_row(a, g, rg, peers, i, lane, status);
  if (last_block_arrive(a.block_counter, gridDim.x)) {
    if ((int)threadIdx.x < g.R) {
      int* flag = reinterpret_cast<int*>(peers.base[threadIdx.x] + rg.flags) +
                  kChCombine * kMaxRanks + g.rank;
      st_release_sys(flag, g.epoch);
    }
  }
}

// ---- reduction --------------------------------------------------------------------------------
// Work item = (token, part of the row): out[t] = sum_j w[t][j] * row_j(t), j in ascending order.
// Lane j < J looks after contributor j: Index holds what it reads for an item, `fetch(t)` issues
// those loads and `resolve(t, index, &side)` turns them into the address of the row (null: none)
// and of its side values. fetch runs one item ahead.
struct Index { int row, slot; float w; };

__device__ __forceinline__ int reduce_first(int parts, int warp) { return (warp / parts) * gridDim.x + blockIdx.x; }

template <typename T, int FORM, typename Fetch, typename Resolve>
__device__ __forceinline__ void reduce_items(const EpGeom& g, int parts, char* out, float* out_topk_w,
                                             Fetch fetch, Resolve resolve) {
  __shared__ const char* s_row[kCombWarps][kMaxItemsPerToken];
  __shared__ const float* s_side[kCombWarps][kMaxItemsPerToken];
  __shared__ float s_w[kCombWarps][kMaxItemsPerToken];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const int J = g.J;
  const int row_bytes = g.H * (int)sizeof(T);
  const int nvec = row_bytes >> 4;
  const int part = warp % parts;
  const int part_vec = (nvec + parts - 1) / parts;
  const int v_end = min(nvec, (part + 1) * part_vec);
  // neighbouring items land on different CTAs, so every SM reads from a mix of peers
  const int per_round = gridDim.x * (nwarps / parts);
  int t = reduce_first(parts, warp);
  Index ix = fetch(t);
  for (; t < g.T; t += per_round) {
    const float* side = nullptr;
    const char* mine = nullptr;
    if (lane < J) mine = resolve(t, ix, &side);
    // the contributors that there are, closed up in ascending order
    const unsigned vmask = __ballot_sync(0xffffffffu, mine != nullptr);
    const int n = __popc(vmask);
    if (mine != nullptr) {
      const int at = __popc(vmask & ((1u << lane) - 1u));
      s_row[warp][at] = mine;
      s_side[warp][at] = side;
      s_w[warp][at] = ix.w;
    }
    __syncwarp();
    ix = fetch(t + per_round);
    constexpr int U = Batch<FORM>::U, G = Batch<FORM>::G, N = Vec16<T>::N;
    for (int v0 = part * part_vec + lane; v0 < v_end; v0 += 32 * U) {
      if (FORM == 1) {
        uint4 val[U];
        const char* rowp = s_row[warp][0];
        const float w = s_w[warp][0];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (n != 0 && v0 + u * 32 < v_end) val[u] = ld_global_once_v4(rowp + ((size_t)(v0 + u * 32) << 4));
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (v0 + u * 32 >= v_end) continue;
          float acc[N];
#pragma unroll
          for (int q = 0; q < N; ++q) acc[q] = 0.f;
          if (n != 0) Vec16<T>::acc(acc, val[u], w);
          st_global_v4(out + (size_t)t * row_bytes + ((size_t)(v0 + u * 32) << 4), Vec16<T>::pack(acc));
        }
        continue;
      }
      float acc[U][N];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int q = 0; q < N; ++q) acc[u][q] = 0.f;
      for (int k0 = 0; k0 < n; k0 += G) {
        uint4 val[G][U];
#pragma unroll
        for (int c = 0; c < G; ++c) {
          if (k0 + c >= n) continue;
          const char* rowp = s_row[warp][k0 + c];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int v = v0 + u * 32;
            if (v < v_end) val[c][u] = ld_global_once_v4(rowp + ((size_t)v << 4));   // coherent path: another GPU may have written it
          }
        }
#pragma unroll
        for (int c = 0; c < G; ++c) {
          if (k0 + c >= n) continue;
          const float w = s_w[warp][k0 + c];
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (v0 + u * 32 < v_end) Vec16<T>::acc(acc[u], val[c][u], w);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int v = v0 + u * 32;
        if (v < v_end) st_global_v4(out + (size_t)t * row_bytes + ((size_t)v << 4), Vec16<T>::pack(acc[u]));
      }
    }
    if (out_topk_w != nullptr && part == 0) {
      if (g.mode == 0) {
        // rank mode: [T,K] = sum over destination ranks of the K side values of each row
        if (lane < g.K) {
          float s = 0.f;
          for (int k = 0; k < n; ++k) s += s_side[warp][k][lane];
          out_topk_w[(size_t)t * g.K + lane] = s;
        }
      } else if (lane < J) {
        // expert mode: [T,K], entry k is the single side value returned for item (t,k)
        out_topk_w[(size_t)t * J + lane] = mine != nullptr ? *side : 0.f;
      }
    }
    __syncwarp();
  }
}

// ---- push form: reduce role ----------------------------------------------------------------
template <typename T, int FORM>
__device__ void combine_reduce_role(const CombineArgs& a, const EpGeom& g, const EpRegions& rg,
                                    char* self_base, int* status) {
  __shared__ int s_ok;
  const int lane = threadIdx.x & 31;
  if (a.wait) {
    if (threadIdx.x == 0) s_ok = 1;
    __syncthreads();
    if ((int)threadIdx.x < g.R) {
      const int* flags = reinterpret_cast<const int*>(self_base + rg.flags) + kChCombine * kMaxRanks;
      if (!wait_flag_ge(flags + threadIdx.x, g.epoch, g.timeout_ns, status, kTimeoutCombine)) s_ok = 0;
    }
    __syncthreads();
    if (!s_ok) return;
  }
  const int J = g.J;
  const int row_bytes = g.H * (int)sizeof(T);
  const int wk = g.mode == 0 ? g.K : 1;              // side values per row
  const char* comb = self_base + rg.comb_x;
  const float* comb_w = reinterpret_cast<const float*>(self_base + rg.comb_w);
  const bool in_place = a.send_row != nullptr;
  const int n_rows = in_place ? min(*a.n_recv_ptr, g.cap) : 0;
  // slots of own rows: lane `rank` in rank mode, a range in expert mode (one bucket after the other)
  int own_lo = lane == g.rank ? 0 : 0x7fffffff, own_hi = 0x7fffffff;
  if (in_place && g.mode == 1) {
    own_lo = a.comb_base[g.rank * g.El];
    if (g.rank + 1 < g.R) own_hi = a.comb_base[(g.rank + 1) * g.El];
  }
  auto fetch = [&](int t) {
    Index ix{-1, -1, 1.f};
    if (t < g.T && lane < J) {
      const size_t at = (size_t)t * J + lane;
      ix.slot = a.send_slot[at];
      if (in_place) ix.row = a.send_row[at];
      if (a.weights) ix.w = a.weights[at];
    }
    return ix;
  };
  auto resolve = [&](int t, const Index& ix, const float** side) -> const char* {
    if (ix.slot < 0 || ix.slot >= g.slot_cap) return nullptr;
    if (in_place && ix.slot >= own_lo && ix.slot < own_hi) {
      if (ix.row < 0 || ix.row >= n_rows) return nullptr;
      *side = a.topk_w + (size_t)ix.row * wk;
      return a.x + (size_t)ix.row * row_bytes;
    }
    *side = comb_w + (size_t)ix.slot * wk;
    return comb + (size_t)ix.slot * row_bytes;
  };
  reduce_items<T, FORM>(g, a.parts, a.out, a.out_topk_w, fetch, resolve);
}

template <typename T, int FORM>
__global__ void __launch_bounds__(kCombWarps * 32, 1)
combine_kernel(EpGeom g, EpRegions rg, const __grid_constant__ PeerPtrs peers, CombineArgs a, int* status) {
  stream_order_wait();
  if (g.R == 1) stream_order_next();
  if (a.role != kCombineReduceOnly) combine_send_role(a, g, rg, peers, status);
  if (a.role != kCombineSendOnly) combine_reduce_role<T, FORM>(a, g, rg, peers.base[g.rank], status);
}

int combine_max_ctas() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) return 1;
  return sms;
}

// How a reduction of T tokens is cut: parts per row (a power of two, at least 2 KiB each; more, down to 512 bytes,
// while the grid has warps to spare), warps per CTA and CTAs no more than the items need.
struct ReduceShape { int parts, warps, blocks; };
static ReduceShape reduce_shape(long long T, int row_bytes, int blocks, bool may_shrink) {
  const int nvec = row_bytes >> 4;
  ReduceShape s{1, kCombWarps, blocks};
  while (s.parts < 4 && nvec / (s.parts * 2) >= 128) s.parts *= 2;
  while (s.parts < 16 && nvec / (s.parts * 2) >= 32 && T * s.parts * 2 <= (long long)blocks * kCombWarps) s.parts *= 2;
  if (!may_shrink) return s;
  const long long items = (T > 0 ? T : 1) * s.parts;
  while (s.warps > 4 && s.warps / 2 >= s.parts && (long long)blocks * (s.warps / 2) >= items) s.warps /= 2;
  const long long need = (items + s.warps - 1) / s.warps;
  if (need < s.blocks) s.blocks = (int)need;
  return s;
}

void launch_combine(const EpGeom& g, const EpRegions& rg, const PeerPtrs& peers, const CombineArgs& args,
                    int dtype_code, int* status, int blocks, cudaStream_t st) {
  if (blocks < 1) blocks = 1;
  CombineArgs a = args;
  // A group of one with its rows at hand has nothing to send and nobody to wait for.
  if (g.R == 1 && a.send_row != nullptr && a.role == kCombineBoth) { a.role = kCombineReduceOnly; a.wait = 0; }
  const ReduceShape rs = reduce_shape(g.T, g.H * (dtype_code == 2 ? 4 : 2), blocks, a.role == kCombineReduceOnly);
  a.parts = rs.parts;
  auto go = [&](auto... forms) {
    decltype(&combine_kernel<float, 0>) all[] = {forms...};
    launch_ordered(all[batch_form(g.J)], rs.blocks, rs.warps * 32, 0, st, 1, g, rg, peers, a, status);
  };
  if (dtype_code == 0) go(combine_kernel<__nv_bfloat16, 0>, combine_kernel<__nv_bfloat16, 1>, combine_kernel<__nv_bfloat16, 2>, combine_kernel<__nv_bfloat16, 3>);
  else if (dtype_code == 1) go(combine_kernel<__half, 0>, combine_kernel<__half, 1>, combine_kernel<__half, 2>, combine_kernel<__half, 3>);
  else go(combine_kernel<float, 0>, combine_kernel<float, 1>, combine_kernel<float, 2>, combine_kernel<float, 3>);
}

// ---- pull form -----------------------------------------------------------------------------
template <typename T, int FORM>
__global__ void __launch_bounds__(kCombWarps * 32, 1)
combine_pull_kernel(EpGeom g, EpRegions rg, const __grid_constant__ PeerPtrs peers, CombinePullArgs a, int* status) {
  __shared__ long long s_info[kMaxRanks][4];
  __shared__ int s_first[kMaxRanks];
  __shared__ int s_ok;
  stream_order_wait();
  if (g.R == 1) stream_order_next();
  const int lane = threadIdx.x & 31;
  char* self_base = peers.base[g.rank];
  if (a.publish && blockIdx.x == 0 && (int)threadIdx.x < g.R) {
    // rows were written by earlier kernels of this stream: complete and visible at this point
    long long* info = reinterpret_cast<long long*>(peers.base[threadIdx.x] + rg.pull_info) + g.rank * 4;
    info[0] = a.x_off;
    info[1] = a.w_off;
    info[2] = a.n_rows;
    int* flag = reinterpret_cast<int*>(peers.base[threadIdx.x] + rg.flags) + kChCombine * kMaxRanks + g.rank;
    st_release_sys(flag, g.epoch);
  }
  if (!a.pull) return;
  if (threadIdx.x == 0) s_ok = 1;
  __syncthreads();
  if ((int)threadIdx.x < g.R) {
    if (g.R == 1 && a.publish) {             // a group of one: what it announces is at hand
      s_info[0][0] = a.x_off; s_info[0][1] = a.w_off; s_info[0][2] = a.n_rows;
    } else {
      const int* flags = reinterpret_cast<const int*>(self_base + rg.flags) + kChCombine * kMaxRanks;
      if (a.wait && !wait_flag_ge(flags + threadIdx.x, g.epoch, g.timeout_ns, status, kTimeoutCombine)) s_ok = 0;
      const long long* info = reinterpret_cast<const long long*>(self_base + rg.pull_info) + threadIdx.x * 4;
      for (int q = 0; q < 3; ++q) s_info[threadIdx.x][q] = __ldcg(&info[q]);
    }
    if (g.mode == 1) s_first[threadIdx.x] = a.comb_base[threadIdx.x * g.El];
  }
  __syncthreads();
  if (!s_ok) return;
  const int J = g.J;
  const int row_bytes = g.H * (int)sizeof(T);
  const int wk = g.mode == 0 ? g.K : 1;
  auto fetch = [&](int t) {
    Index ix{-1, -1, 1.f};
    if (t < g.T && lane < J) {
      const size_t at = (size_t)t * J + lane;
      ix.row = a.send_row[at];
      if (g.mode == 1) ix.slot = a.send_slot[at];
      if (a.weights) ix.w = a.weights[at];
    }
    return ix;
  };
  auto resolve = [&](int t, const Index& ix, const float** side) -> const char* {
    if (ix.row < 0) return nullptr;
    const int d = g.mode == 0 ? lane : rank_of_slot(s_first, g.R, ix.slot);
    if ((long long)ix.row >= s_info[d][2] || s_info[d][0] < 0) {
      set_status(status, kOverflowSlots);       // the peer did not announce that many rows
      return nullptr;
    }
    *side = reinterpret_cast<const float*>(peers.base[d] + s_info[d][1]) + (size_t)ix.row * wk;
    return peers.base[d] + s_info[d][0] + (size_t)ix.row * row_bytes;
  };
  reduce_items<T, FORM>(g, a.parts, a.out, a.out_topk_w, fetch, resolve);
}

void launch_combine_pull(const EpGeom& g, const EpRegions& rg, const PeerPtrs& peers,
                         const CombinePullArgs& args, int dtype_code, int* status, int blocks, cudaStream_t st) {
  if (blocks < 1) blocks = 1;
  CombinePullArgs a = args;
  ReduceShape rs = reduce_shape(g.T, g.H * (dtype_code == 2 ? 4 : 2), blocks, true);
  if (!a.pull) rs = ReduceShape{1, 1, 1};
  a.parts = rs.parts;
  auto go = [&](auto... forms) {
    decltype(&combine_pull_kernel<float, 0>) all[] = {forms...};
    launch_ordered(all[batch_form(g.J)], rs.blocks, rs.warps * 32, 0, st, 1, g, rg, peers, a, status);
  };
  if (dtype_code == 0) go(combine_pull_kernel<__nv_bfloat16, 0>, combine_pull_kernel<__nv_bfloat16, 1>, combine_pull_kernel<__nv_bfloat16, 2>, combine_pull_kernel<__nv_bfloat16, 3>);
  else if (dtype_code == 1) go(combine_pull_kernel<__half, 0>, combine_pull_kernel<__half, 1>, combine_pull_kernel<__half, 2>, combine_pull_kernel<__half, 3>);
  else go(combine_pull_kernel<float, 0>, combine_pull_kernel<float, 1>, combine_pull_kernel<float, 2>, combine_pull_kernel<float, 3>);
}

// Signal only (used when a fused GEMM epilogue has already stored the rows).
__global__ void signal_kernel(PeerPtrs peers, long long flags_off, int channel, int rank, int R,
                              int epoch) {
  if ((int)threadIdx.x < R) {
    fence_acq_rel_sys();
    int* flag = reinterpret_cast<int*>(peers.base[threadIdx.x] + flags_off) +
                channel * kMaxRanks + rank;
    st_release_sys(flag, epoch);
  }
}
void launch_signal(const PeerPtrs& peers, long long flags_off, int channel, int rank, int R,
                   int epoch, cudaStream_t st) {
  signal_kernel<<<1, 32, 0, st>>>(peers, flags_off, channel, rank, R, epoch);
}

}  // namespace b200ep
