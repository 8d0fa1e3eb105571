// Grouped expert GEMMs on the 5th-generation tensor cores (tcgen05 + TMEM), bf16 -> f32.
//
//   out[r, :] = epilogue( A[r, :] . W[e(r)]^T )    A: [rows, K] rows grouped by local expert,
//                                                  W: [E_local, N_w, K] (K-major, as nn.Linear)
// Replaces the library grouped GEMM / per-expert F.linear loop of the reference
// (`DeepEP_Megatron/test_deepep_moe_dispatch_combine.py:528-541,590-600`) and, through the
// epilogues, the element-wise kernels and the unpermute + combine send that follow them:
//   EPI_PLAIN   : bf16 store.
//   EPI_SWIGLU  : W holds [gate rows | linear rows]; a CTA multiplies 64 gate and the matching 64
//                 linear rows, the epilogue writes silu(gate) * linear * prob[r] as bf16 and, for
//                 training, the pre-activation too.
//   EPI_ACT     : the same for gelu / silu / relu: f(result) * prob and, for training, the pre-activation. Three groups of
//                 epilogue warps (8191 rows, 8 experts, 4096 x 4096: GEMM, activation kernel and fc2 with silu 441 us, in
//                 the epilogue 415; forward and backward of 12001 rows, 16 experts, 2048 x 1408: 440 -> 428, with two
//                 groups 437).
//   EPI_DSWIGLU : (data gradient of fc2) the result is the gradient of silu(gate) * linear * prob; the epilogue
//                 reads the kept pre-activation and writes its gradient, so the gradient of the activation never
//                 goes to memory and no element-wise kernel follows. The sums for the probabilities' gradients
//                 leave as one part per 128 columns (fixed order; sum_parts_kernel adds them). It has three groups
//                 of epilogue warps: with two the element-wise work of a tile takes longer than its MMAs (12001 rows, 16 experts,
//                 2048 x 1408: GEMM and element-wise kernel apart 68 + 34.4 us, in one with two groups 126, with three
//                 75 + 4.0 for the sums). Not for gelu / silu / relu, whose element-wise backward moves 3 elements where
//                 this moves 5: in one launch the same step with silu took 453 us, apart 433.
//   EPI_COMBINE : the fc2 result rows are stored straight into the combine slot of each token's
//                 SOURCE rank over NVLink (LSU stores), so no separate unpermute/combine-send
//                 kernel runs; the source reduces its slots on arrival.
//
// The WEIGHTS are the M operand of the tensor core (128 accumulator lanes per CTA = 128 weight rows)
// and the TOKENS its N operand. N can be any multiple of 16 (32 for a pair) up to 256 per tile, so an
// expert's rows are cut into equal tiles that fit them: 8 rows cost a 32-column MMA, 260 rows two of
// 160 and 128. With tokens on M every expert was padded to a multiple of 128 or 256 rows: at 8 rows per
// expert 31/32 of the MMA work and half of the operand traffic were padding, at 1000 rows 12 %.
// Structure: persistent CTAs, one per SM; warp 0 = TMA producer (plain tile loads of this GPU's
// memory; every CTA fetches its own tiles), warp 1 = MMA issuer and TMEM owner, the others = epilogue.
// 2 TMEM accumulators (128 lanes x 256 f32 columns each) so the epilogue of tile i overlaps the MMAs
// of tile i+1. Bound: few rows per expert: the weights, read once (32 experts x 8 rows, hidden 7168, FFN
// 2048: fc1 + fc2 623-657 -> 437-450 us = 6.4 TB/s); many rows: the tensor pipe under the power cap
// (8 x 1100 rows, hidden 4096, FFN 14336: fc1 1871 -> 1642 us; 8 x 1024, which fills 256-row tiles
// either way: 1462 -> 1465 us = 1313 TFLOP/s, in a loop). Two forms of the same kernel (template CG):
//   CG = 1: one CTA per 128 weight rows x 256 tokens; 4-stage ring of 16 KiB weights + 32 KiB tokens.
//   CG = 2: a CTA pair (cluster of two SMs, `cta_group::2`) per 256 weight rows x 256 tokens. Each CTA
//           loads its own 128 weight rows and HALF of the token tile; the leader CTA issues one MMA
//           that reads both halves from the two CTAs' shared memory and writes 128 accumulator lanes
//           into each CTA's TMEM. A token tile is thus fetched once per pair and the shared-memory
//           traffic per flop halves for it; 6-stage ring of 32 KiB.
// Epilogue: an accumulator lane is a weight row (an output column), so 16 token columns at a time go
// through a f32 staging tile in shared memory and leave as 128-byte segments of output rows. Two or
// three groups of four warps take 16-column chunks in turn.
// The tile list is derived on the device from the per-expert row offsets (no host sync).
// Every mbarrier wait is bounded; on a time-out all roles leave their loops, TMEM is freed.
#include <cuda_bf16.h>
#include "tc05.cuh"
#include "tmap.h"
#include "gemm_api.h"
#include "act.cuh"

namespace b200ep {

using namespace tc;

constexpr int WM = 128, TN = 256, BK = 64;                    // weight rows per CTA, tokens per tile, reduction block
constexpr int W_BYTES = WM * BK * 2, T_HALF_BYTES = 128 * BK * 2;
// per-CTA stage: weight tile + the part of the token tile this CTA holds (all of it, or one half)
template <int CG> struct Ring;
template <> struct Ring<1> { static constexpr int STAGES = 4, STAGE_BYTES = W_BYTES + 2 * T_HALF_BYTES; };
template <> struct Ring<2> { static constexpr int STAGES = 6, STAGE_BYTES = W_BYTES + T_HALF_BYTES; };
constexpr int MAX_STAGES = 6;
constexpr int RING_BYTES = 4 * (W_BYTES + 2 * T_HALF_BYTES);
static_assert(Ring<1>::STAGES * Ring<1>::STAGE_BYTES == RING_BYTES && Ring<2>::STAGES * Ring<2>::STAGE_BYTES == RING_BYTES, "");
constexpr int CHUNK = 16;                                     // token columns per staging pass
constexpr int STG_LD = WM + 4;                                // f32 per staged token (pad: bank spread)
constexpr int STG_BYTES = CHUNK * STG_LD * 4;
// groups of four epilogue warps
template <int EPI> struct Epi {
  static constexpr int GROUPS = EPI == EPI_DSWIGLU || EPI == EPI_ACT ? 3 : 2, WARPS = 4 * GROUPS;
  static constexpr int THREADS = 64 + 32 * WARPS, SMEM_BYTES = RING_BYTES + GROUPS * STG_BYTES + 1024 /*align slack*/;
};
constexpr int kMaxLocalExperts = 256;
constexpr int TOKEN_BOXES = 4;                                // token boxes of 16, 32, 64 and 128 rows

struct TokenMaps { CUtensorMap m[TOKEN_BOXES]; };

// An expert's rows are cut into ceil(rows / 256) token tiles of equal size in units of G = 16 * CG rows (the
// first ones get what does not divide). Equal tiles matter beyond the rows saved: units take tiles in a
// fixed stride, and with all the short tiles at one place of every expert some units would meet none.
__device__ __forceinline__ int token_tiles(int rows) { return (rows + TN - 1) / TN; }

struct Tile { int e, row0, rows, n, wt; };   // expert, first row, valid rows, MMA columns, weight tile

// Tile t -> token tile and weight tile. `e` is kept from call to call (t only grows). Order inside one
// expert: bands of `gm` token tiles; inside a band the token tile runs fastest, then the weight tile,
// so the tiles in flight at one time cover a band of activation rows times a few weight tiles, the
// band stays in L2 while all weight tiles pass over it, and an expert whose activations exceed L2 is
// not re-read from HBM once per weight tile.
template <int G>
__device__ __forceinline__ bool decode_tile(int t, const int* s_tile_off, const int* s_row_off, int El,
                                            int w_tiles, int gm, int& e, Tile& out) {
  if (t >= s_tile_off[El]) return false;
  while (e + 1 < El && t >= s_tile_off[e + 1]) ++e;
  const int local = t - s_tile_off[e];
  const int rows = s_row_off[e + 1] - s_row_off[e];
  const int t_tiles = token_tiles(rows);
  const int per_band = gm * w_tiles;
  const int band = local / per_band;
  const int idx = local - band * per_band;
  const int band_t = min(gm, t_tiles - band * gm);
  const int tt = band * gm + idx % band_t;
  out.e = e;
  out.wt = idx / band_t;
  const int units = (rows + G - 1) / G, each = units / t_tiles, more = units - each * t_tiles;
  const int first = (tt * each + min(tt, more)) * G;
  out.n = (each + (tt < more ? 1 : 0)) * G;
  out.row0 = s_row_off[e] + first;
  out.rows = min(out.n, rows - first);
  return true;
}

__device__ __forceinline__ float silu(float v) { return v / (1.f + __expf(-v)); }
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ float bf_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf_hi(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }
// Backward of silu(g) * l * prob for one element: d = gradient of the product; the gradients of g and l come back in
// place of g and l, the element's share of the probability's gradient is returned.
__device__ __forceinline__ float dswiglu(float d, float pr, float& g, float& l) {
  const float sig = sigmoid(g);
  const float s = g * sig, da = d * pr, share = d * s * l;
  g = da * l * sig * (1.f + g * (1.f - sig));
  l = da * s;
  return share;
}
// four columns: d against bf16 pairs of gate and linear, both replaced by their gradients
__device__ __forceinline__ float dswiglu4(const float4& d, float pr, uint2& hg, uint2& hl) {
  float g[4] = {bf_lo(hg.x), bf_hi(hg.x), bf_lo(hg.y), bf_hi(hg.y)};
  float l[4] = {bf_lo(hl.x), bf_hi(hl.x), bf_lo(hl.y), bf_hi(hl.y)};
  const float dd[4] = {d.x, d.y, d.z, d.w};
  float share = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) share += dswiglu(dd[i], pr, g[i], l[i]);
  hg = make_uint2(pack_bf16(g[0], g[1]), pack_bf16(g[2], g[3]));
  hl = make_uint2(pack_bf16(l[0], l[1]), pack_bf16(l[2], l[3]));
  return share;
}
__device__ __forceinline__ float act_only(int kind, float x) {
  float f, df;
  act_eval(kind, x, &f, &df);
  return f;
}
__device__ __forceinline__ void st_global_v2(void* p, uint32_t a, uint32_t b) {
  asm volatile("st.global.L1::no_allocate.v2.u32 [%0], {%1,%2};" ::"l"(p), "r"(a), "r"(b) : "memory");
}

// WMN: the weights are stored [E_local, K, N] (N contiguous) instead of [E_local, N, K]; they are
// then read as an M-major operand (64 x 64 boxes, one 128-byte row of 64 outputs per reduction
// index), which is how the data gradients use the forward weights without a transposed copy.
template <int EPI, int CG, bool WMN>
__global__ void __launch_bounds__(Epi<EPI>::THREADS, 1)
grouped_gemm_kernel(const __grid_constant__ TokenMaps map_t, const __grid_constant__ CUtensorMap map_w,
                    const __grid_constant__ GemmParams p, const __grid_constant__ PeerPtrs peers) {
  constexpr int EPI_GROUPS = Epi<EPI>::GROUPS, EPI_WARPS = Epi<EPI>::WARPS;
  constexpr int STAGES = Ring<CG>::STAGES, STAGE_BYTES = Ring<CG>::STAGE_BYTES, G = 16 * CG;
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t full_bar[MAX_STAGES], empty_bar[MAX_STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  __shared__ int s_tile_off[kMaxLocalExperts + 1], s_row_off[kMaxLocalExperts + 1];

  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* abort = &s_abort;
  // work unit = CTA (CG 1) or CTA pair (CG 2); in a pair, rank 0 leads: it owns the barriers the
  // MMA thread waits on and issues every MMA; both CTAs load, both run an epilogue on their own TMEM
  const int cta_rank = CG == 2 ? (int)cluster_cta_rank() : 0;
  const bool leader = cta_rank == 0;
  const int unit = CG == 2 ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int n_units = CG == 2 ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  const int gm = max(1, p.band_rows / TN);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], EPI_WARPS * CG); }
    s_abort = 0;
    fence_barrier_init();
    prefetch_tmap(&map_w);
    for (int b = 0; b < TOKEN_BOXES; ++b) prefetch_tmap(&map_t.m[b]);
  }
  if (warp == 1) {
    if (CG == 2) tmem_alloc_pair(&s_tmem, 512); else tmem_alloc(&s_tmem, 512);
  }
  if (warp == 2) {
    // device-side tile table: rows per expert come from the dispatch metadata
    int acc = 0;
    for (int e0 = 0; e0 < p.El; e0 += 32) {
      const int e = e0 + lane;
      int r0 = 0, r1 = 0, tiles = 0;
      if (e < p.El) {
        r0 = max(0, min(p.expert_off[e], p.max_rows));
        r1 = max(r0, min(p.expert_off[e + 1], p.max_rows));
        tiles = token_tiles(r1 - r0) * p.n_tiles;
      }
      int incl = tiles;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
      }
      if (e < p.El) {
        s_tile_off[e] = acc + incl - tiles;
        s_row_off[e] = r0;
        if (e == p.El - 1) s_row_off[p.El] = r1;
      }
      acc += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) s_tile_off[p.El] = acc;
  }
  fence_before_sync();
  __syncthreads();
  __syncwarp();
  if (CG == 2) cluster_sync_all();      // the peer's barriers are initialised before anything arrives on them
  fence_after_sync();
  const uint32_t tmem_base = s_tmem;
  const int k_blocks = (p.K + BK - 1) / BK;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (elect_one()) {
      uint32_t it = 0;
      int e = 0;
      Tile tl;
      for (int t = unit; decode_tile<G>(t, s_tile_off, s_row_off, p.El, p.n_tiles, gm, e, tl) && !*abort; t += n_units) {
        // weight rows of this CTA: [gate 64 | linear 64] for swiglu, 128 consecutive rows otherwise
        const int f0 = (tl.wt * CG + cta_rank) * (EPI == EPI_SWIGLU ? 64 : WM);       // first output column
        const int w_first = tl.e * p.w_rows + f0;
        // my token rows: all n of them, or my half; one box that covers them (two of 128 above 128 rows)
        const int nb = tl.n / CG;
        const int tok0 = tl.row0 + cta_rank * nb;
        const int box = nb <= 16 ? 0 : nb <= 32 ? 1 : nb <= 64 ? 2 : 3;
        const int boxes = (CG == 1 && nb > 128) ? 2 : 1;
        const CUtensorMap* mt = &map_t.m[box];
        const uint32_t bytes = W_BYTES + boxes * (16u << box) * BK * 2;
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (it >= STAGES && !mbar_wait(&empty_bar[s], ph ^ 1, p.status, abort)) break;
          unsigned char* st = smem + s * STAGE_BYTES;
          // (a pair's bytes are all counted on the leader's barrier; only the leader announces them)
          if (leader) mbar_expect_tx(&full_bar[s], CG * bytes);
          auto load = [&](unsigned char* dst, const CUtensorMap* map, int x, int y) {
            if (CG == 1) tma_load_2d(dst, map, x, y, &full_bar[s]); else tma_load_2d_pair(dst, map, x, y, &full_bar[s]);
          };
          if (WMN) {
            // weights [K, N] per expert: boxes of 64 reduction rows x 64 output columns. A reduction
            // tail that runs into the next expert's rows meets zero-filled columns of the tokens.
            const int krow = tl.e * p.w_rows + kb * BK;
            load(st, &map_w, f0, krow);
            load(st + W_BYTES / 2, &map_w, f0 + 64, krow);
          } else if (EPI == EPI_SWIGLU) {
            load(st, &map_w, kb * BK, w_first);
            load(st + W_BYTES / 2, &map_w, kb * BK, w_first + p.N);
          } else {
            load(st, &map_w, kb * BK, w_first);
          }
          load(st + W_BYTES, mt, kb * BK, tok0);
          if (boxes == 2) load(st + W_BYTES + T_HALF_BYTES, mt, kb * BK, tok0 + 128);
        }
      }
      if (*abort) {
        // let the loads that are still in flight land before the CTA's shared memory goes away
        // (a pair's follower cannot observe its own loads: they complete on the leader's barrier)
        if (CG == 1 || leader) {
          int quiet = 0;
          for (uint32_t n = it > STAGES ? it - STAGES : 0; n < it; ++n)
            mbar_wait(&full_bar[n % STAGES], (n / STAGES) & 1, nullptr, &quiet);
        }
      } else if (CG == 2) {
        // a pair's CTA must not leave while the leader's last commits can still arrive on its barriers
        for (uint32_t n = it > STAGES ? it - STAGES : 0; n < it; ++n)
          if (!mbar_wait(&empty_bar[n % STAGES], (n / STAGES) & 1, p.status, abort)) break;
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (the leader CTA of a pair) ----------------
    if (leader && elect_one()) {
      uint32_t it = 0, tile_n = 0;
      int e = 0;
      Tile tl;
      for (int t = unit; decode_tile<G>(t, s_tile_off, s_row_off, p.El, p.n_tiles, gm, e, tl) && !*abort; t += n_units, ++tile_n) {
        const int buf = tile_n & 1;
        const uint32_t use = tile_n >> 1;
        const uint32_t idesc = instr_desc_bf16(WM * CG, tl.n, WMN, false);
        if (use > 0 && !mbar_wait(&acc_empty[buf], (use - 1) & 1, p.status, abort)) break;
        fence_after_sync();
        const uint32_t d_tmem = tmem_base + buf * TN;
        bool ok = true;
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(&full_bar[s], ph, p.status, abort)) { ok = false; break; }
          fence_after_sync();
          const uint32_t w_addr = smem_u32(smem + s * STAGE_BYTES);
          const uint64_t w_desc = WMN ? smem_desc_mn_sw128(w_addr, W_BYTES / 2) : smem_desc_sw128(w_addr);
          const uint64_t t_desc = smem_desc_sw128(w_addr + W_BYTES);
          // per MMA step of 16 reduction indices: K-major +32 bytes (2 units), M-major +16 rows of 128 bytes (128 units)
          constexpr int W_STEP = WMN ? 128 : 2;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            if (CG == 1) mma_bf16(d_tmem, w_desc + W_STEP * k, t_desc + 2 * k, idesc, (kb | k) ? 1u : 0u);
            else mma_bf16_pair(d_tmem, w_desc + W_STEP * k, t_desc + 2 * k, idesc, (kb | k) ? 1u : 0u);
          }
          // frees the smem stage (in both CTAs of a pair) when these MMAs retire
          if (CG == 1) mma_commit(&empty_bar[s]); else mma_commit_pair(&empty_bar[s]);
        }
        if (!ok) break;
        // accumulator complete (announced to both epilogues of a pair)
        if (CG == 1) mma_commit(&acc_full[buf]); else mma_commit_pair(&acc_full[buf]);
      }
    }
  } else {
    // ---------------- epilogue: two or three groups of 4 warps, one TMEM lane quarter per warp ----------------
    const int q = warp & 3;                        // TMEM lanes [32q, 32q+32)
    const int grp = (warp - 2) >> 2;
    const int bar_id = 1 + grp;                    // the group's barrier (128 threads)
    const int gtid = ((warp - 2) & 3) * 32 + lane; // thread of the group
    float* stg = reinterpret_cast<float*>(smem + RING_BYTES + grp * STG_BYTES);
    float* my_stg = stg + q * 32 + lane;
    const int oct = gtid & 15, tok_in = gtid >> 4; // reader: output columns 4*oct.. and 64 + 4*oct.. of tokens tok_in, tok_in + 8
    uint32_t tile_n = 0;
    int e = 0;
    Tile tl;
    for (int t = unit; decode_tile<G>(t, s_tile_off, s_row_off, p.El, p.n_tiles, gm, e, tl); t += n_units, ++tile_n) {
      const int buf = tile_n & 1;
      // all four warps take the same way out: a warp that left alone would strand the others at the group's barrier
      if (!group_all(bar_id, !*abort && mbar_wait(&acc_full[buf], (tile_n >> 1) & 1, p.status, abort))) break;
      fence_after_sync();
      const uint32_t t_addr = tmem_base + buf * TN + ((uint32_t)(q * 32) << 16);
      const int col0 = (tl.wt * CG + cta_rank) * (EPI == EPI_SWIGLU ? 64 : WM) + 4 * oct;
      float prob[2] = {1.f, 1.f};
      // what the reader needs to know about its two tokens of chunk c, requested one chunk ahead
      int2 meta[2];
      uint2 pre[2][4];                             // dswiglu: gate and linear of my columns, then of those 64 on
      const bool ok_a = col0 < p.N, ok_b = col0 + 64 < p.N;      // (a last tile may hang over the expert's outputs)
      auto fetch = [&](int c) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int tok = c * CHUNK + tok_in + 8 * i;
          if (EPI != EPI_PLAIN && EPI != EPI_COMBINE && p.row_prob != nullptr && tok < tl.rows) prob[i] = p.row_prob[tl.row0 + tok];
          if (EPI == EPI_DSWIGLU && ok_a && tok < tl.rows) {
            const char* h = reinterpret_cast<const char*>(p.pre_out) + ((size_t)(tl.row0 + tok) * p.pre_ld + col0) * 2;
            pre[i][0] = __ldg(reinterpret_cast<const uint2*>(h));
            pre[i][1] = __ldg(reinterpret_cast<const uint2*>(h + (size_t)p.N * 2));
            pre[i][2] = __ldg(reinterpret_cast<const uint2*>(h + 128));
            pre[i][3] = __ldg(reinterpret_cast<const uint2*>(h + (size_t)p.N * 2 + 128));
          }
          if (EPI == EPI_COMBINE && tok < tl.rows) meta[i] = p.recv_meta[tl.row0 + tok];
        }
      };
      const int chunks = tl.n / CHUNK;
      uint32_t v[CHUNK];
      if (grp < chunks) { fetch(grp); tmem_ld16(t_addr + grp * CHUNK, v); }
      for (int c = grp; c < chunks; c += EPI_GROUPS) {
        tmem_ld_wait();
        tmem_ld_pin16(v);
        group_sync(bar_id);                        // the readers of the previous chunk are done
#pragma unroll
        for (int i = 0; i < CHUNK; ++i) my_stg[i * STG_LD] = __uint_as_float(v[i]);
        group_sync(bar_id);
        const float pr0 = prob[0], pr1 = prob[1];
        int2 mt[2];
        if (EPI == EPI_COMBINE) { mt[0] = meta[0]; mt[1] = meta[1]; }
        uint2 hv[2][4];
        if (EPI == EPI_DSWIGLU) {
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int u = 0; u < 4; ++u) hv[i][u] = pre[i][u];
        }
        if (c + EPI_GROUPS < chunks) { fetch(c + EPI_GROUPS); tmem_ld16(t_addr + (c + EPI_GROUPS) * CHUNK, v); }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int tok = tok_in + 8 * i;
          if (c * CHUNK + tok >= tl.rows) continue;
          const float4 a = *reinterpret_cast<const float4*>(stg + tok * STG_LD + 4 * oct);
          const float4 b = *reinterpret_cast<const float4*>(stg + tok * STG_LD + 64 + 4 * oct);
          const size_t grow = (size_t)(tl.row0 + c * CHUNK + tok);
          if (EPI == EPI_DSWIGLU) {
            // a and b are the gradient of the activation; it goes no further than these registers
            const int block = tl.wt * CG + cta_rank;     // my CTA's 128 columns: all there or, behind an odd number, none
            if (!ok_b) continue;
            const float pr = i == 0 ? pr0 : pr1;
            float share = dswiglu4(a, pr, hv[i][0], hv[i][1]) + dswiglu4(b, pr, hv[i][2], hv[i][3]);
            char* o = reinterpret_cast<char*>(p.out) + (grow * p.out_ld + col0) * 2;
            st_global_v2(o, hv[i][0].x, hv[i][0].y);
            st_global_v2(o + 128, hv[i][2].x, hv[i][2].y);
            o += (size_t)p.N * 2;
            st_global_v2(o, hv[i][1].x, hv[i][1].y);
            st_global_v2(o + 128, hv[i][3].x, hv[i][3].y);
            // the 16 lanes of a token hold its 128 columns
            const unsigned half_mask = 0xffffu << (lane & 16);
#pragma unroll
            for (int m = 8; m > 0; m >>= 1) share += __shfl_xor_sync(half_mask, share, m);
            if (oct == 0) p.dp_part[(size_t)block * p.max_rows + grow] = share;
          } else if (EPI == EPI_ACT) {
            const float pr = i == 0 ? pr0 : pr1;
            const int k = p.act_kind;
            char* o = reinterpret_cast<char*>(p.out) + (grow * p.out_ld + col0) * 2;
            if (ok_a) st_global_v2(o, pack_bf16(act_only(k, a.x) * pr, act_only(k, a.y) * pr), pack_bf16(act_only(k, a.z) * pr, act_only(k, a.w) * pr));
            if (ok_b) st_global_v2(o + 128, pack_bf16(act_only(k, b.x) * pr, act_only(k, b.y) * pr), pack_bf16(act_only(k, b.z) * pr, act_only(k, b.w) * pr));
            if (p.pre_out != nullptr) {
              char* h = reinterpret_cast<char*>(p.pre_out) + (grow * p.pre_ld + col0) * 2;
              if (ok_a) st_global_v2(h, pack_bf16(a.x, a.y), pack_bf16(a.z, a.w));
              if (ok_b) st_global_v2(h + 128, pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
            }
          } else if (EPI == EPI_SWIGLU) {
            const float pr = i == 0 ? pr0 : pr1;
            char* o = reinterpret_cast<char*>(p.out) + (grow * p.out_ld + col0) * 2;
            st_global_v2(o, pack_bf16(silu(a.x) * b.x * pr, silu(a.y) * b.y * pr),
                         pack_bf16(silu(a.z) * b.z * pr, silu(a.w) * b.w * pr));
            if (p.pre_out != nullptr) {
              // training forward: also keep the pre-activation [gate | linear] (bf16) for the backward pass
              char* h = reinterpret_cast<char*>(p.pre_out) + (grow * p.pre_ld + col0) * 2;
              st_global_v2(h, pack_bf16(a.x, a.y), pack_bf16(a.z, a.w));
              st_global_v2(h + (size_t)p.N * 2, pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
            }
          } else {
            char* o;
            if (EPI == EPI_COMBINE) {
              const bool good = mt[i].y >= 0 && mt[i].y < p.R && mt[i].x >= 0 && mt[i].x < p.slot_cap;
              if (!good) { set_status(p.status, kOverflowSlots); continue; }
              o = peers.base[mt[i].y] + p.comb_off + ((size_t)mt[i].x * p.N_out + col0) * 2;
            } else {
              o = reinterpret_cast<char*>(p.out) + (grow * p.out_ld + col0) * 2;
            }
            if (col0 < p.N_out) st_global_v2(o, pack_bf16(a.x, a.y), pack_bf16(a.z, a.w));
            if (col0 + 64 < p.N_out) st_global_v2(o + 128, pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
          }
        }
      }
      fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        if (CG == 1) mbar_arrive(&acc_empty[buf]); else mbar_arrive_cluster_tmem(&acc_empty[buf], 0);
      }
    }
  }

  // ---------------- teardown: every path arrives here ----------------
  fence_before_sync();
  __syncthreads();
  __syncwarp();
  if (CG == 2) cluster_sync_all();      // both epilogues are done with TMEM, nobody addresses the peer any more
  if (warp == 1) {
    fence_after_sync();
    if (CG == 2) tmem_dealloc_pair(tmem_base, 512); else tmem_dealloc(tmem_base, 512);
  }
  if (EPI == EPI_COMBINE && p.signal_flag_off >= 0) {
    // all CTAs' peer stores done -> the last CTA raises this rank's combine flag on every peer
    if (last_block_arrive(p.block_counter, gridDim.x)) {
      if (threadIdx.x < p.R) {
        int* flag = reinterpret_cast<int*>(peers.base[threadIdx.x] + p.signal_flag_off) + p.rank;
        st_release_sys(flag, p.epoch);
      }
    }
  }
}

// ---- host side -----------------------------------------------------------------------------
// Number of CTA pairs that can be resident at once (the SMs of a pair share a GPC, so this can be
// below SMs / 2); cached per epilogue. 0 if the query fails.
template <int EPI, bool WMN>
static int max_resident_pairs() {
  static int cached = -1;
  if (cached < 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2, 1, 1);
    cfg.blockDim = dim3(Epi<EPI>::THREADS, 1, 1);
    cfg.dynamicSmemBytes = Epi<EPI>::SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, grouped_gemm_kernel<EPI, 2, WMN>, &cfg) != cudaSuccess) n = 0;
    cached = n;
  }
  return cached;
}

template <int EPI, bool WMN>
static int launch_one(const TokenMaps& ma, const CUtensorMap& mb, const GemmParams& p, const PeerPtrs& peers,
                      int ctas, bool pair, cudaStream_t st) {
  if (!pair) {
    if (cudaFuncSetAttribute(grouped_gemm_kernel<EPI, 1, WMN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Epi<EPI>::SMEM_BYTES) != cudaSuccess)
      return 4;
    grouped_gemm_kernel<EPI, 1, WMN><<<ctas, Epi<EPI>::THREADS, Epi<EPI>::SMEM_BYTES, st>>>(ma, mb, p, peers);
    return 0;
  }
  if (cudaFuncSetAttribute(grouped_gemm_kernel<EPI, 2, WMN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Epi<EPI>::SMEM_BYTES) != cudaSuccess)
    return 4;
  int pairs = ctas / 2;
  const int resident = max_resident_pairs<EPI, WMN>();
  if (resident < 1) return 5;
  if (pairs > resident) pairs = resident;
  if (pairs < 1) pairs = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs, 1, 1);
  cfg.blockDim = dim3(Epi<EPI>::THREADS, 1, 1);
  cfg.dynamicSmemBytes = Epi<EPI>::SMEM_BYTES;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, grouped_gemm_kernel<EPI, 2, WMN>, ma, mb, p, peers) == cudaSuccess ? 0 : 5;
}

int launch_grouped_gemm(const void* a, long long a_rows, const void* w, int epi, GemmParams p,
                        const PeerPtrs& peers, int ctas, bool pair, cudaStream_t st) {
  if (p.El < 1 || p.El > kMaxLocalExperts || p.K <= 0 || p.K % 8 || p.N <= 0 || p.N_out % 8) return 1;
  if (reinterpret_cast<uintptr_t>(a) % 16 || reinterpret_cast<uintptr_t>(w) % 16) return 1;
  if ((epi == EPI_SWIGLU || epi == EPI_DSWIGLU) && (p.N % 128)) return 1;
  if (epi == EPI_ACT && (p.act_kind < 0 || p.act_kind > 2)) return 1;
  if (p.b_mn && epi != EPI_PLAIN && epi != EPI_DSWIGLU) return 1;
  // No rows (no tokens, or a rank that none was sent to): nothing to compute, and a tensor map may not be empty. The combine
  // epilogue has its flag to raise all the same: its map names one row of the weights, which no tile reads.
  const long long map_rows = a_rows > 0 ? a_rows : 1;
  if (a_rows == 0) {
    if (epi != EPI_COMBINE || p.signal_flag_off < 0) return 0;
    a = w;
  }
  if (epi == EPI_DSWIGLU && (!p.b_mn || p.pre_out == nullptr || p.dp_part == nullptr)) return 1;
  // 64-column boxes (one 128-byte swizzle row): the tokens in four heights, so that a small tile fetches no more
  // rows than it needs; the weights 128 rows high, 64 where a CTA's rows come from two places
  TokenMaps ma;
  CUtensorMap mb;
  for (int b = 0; b < TOKEN_BOXES; ++b)
    if (make_tmap_bf16(&ma.m[b], a, map_rows, p.K, BK, 16 << b)) return 3;
  if (p.b_mn) {
    if (make_tmap_bf16(&mb, w, (long long)p.El * p.w_rows, p.N, 64, BK)) return 3;
  } else if (make_tmap_bf16(&mb, w, (long long)p.El * p.w_rows, p.K, BK, epi == EPI_SWIGLU ? 64 : WM)) return 3;
  const int tile_cols = (pair ? 2 : 1) * (epi == EPI_SWIGLU ? 64 : WM);       // output columns per tile
  p.n_tiles = (p.N + tile_cols - 1) / tile_cols;
  p.max_rows = (int)a_rows;
  if (p.band_rows <= 0) p.band_rows = 2048;
  if (ctas < 1) ctas = 1;
  if (epi == EPI_PLAIN && p.b_mn) return launch_one<EPI_PLAIN, true>(ma, mb, p, peers, ctas, pair, st);
  if (epi == EPI_DSWIGLU) return launch_one<EPI_DSWIGLU, true>(ma, mb, p, peers, ctas, pair, st);
  if (epi == EPI_ACT) return launch_one<EPI_ACT, false>(ma, mb, p, peers, ctas, pair, st);
  if (epi == EPI_PLAIN) return launch_one<EPI_PLAIN, false>(ma, mb, p, peers, ctas, pair, st);
  if (epi == EPI_SWIGLU) return launch_one<EPI_SWIGLU, false>(ma, mb, p, peers, ctas, pair, st);
  if (epi == EPI_COMBINE) return launch_one<EPI_COMBINE, false>(ma, mb, p, peers, ctas, pair, st);
  return 1;
}

}  // namespace b200ep
