// Packed variable-length causal GQA prefill attention on the Blackwell tensor cores (tcgen05 + TMEM + tensor-map TMA).
//   b200_gqa_varlen_causal       <-> triton_kernels/gqa_attention_varlen_causal.py:214-278 (kernel :99-210)
//   b200_fused_prefill_attention <-> the chain of engine/runner.py:339-384: partial_rope(q), partial_rope(k),
//                                    gqa_attention_varlen_causal, attention_gate_pack, paged_kv_fill_varlen
//
// Calls that are over in one wave of CTAs run on a kernel without pairs (prefill_short.cu); here is the other one.
// Two CTAs of a cluster work on one item after another: (sequence, kv head, block of 64 query tokens), 32 tokens each.  The 4 Q heads
// of the group are stacked into the 128 rows of a CTA's half of an M=256 tile (row = token*4 + head, the stacking idea of
// gqa_attention_varlen_causal.py:151-160).  Per 128-token KV tile, cta_group::2, operands split over the pair:
//     S[256 x 128]  = Q[256 x 256] . K^T          tcgen05.mma, both operands K-major in shared memory, D in TMEM
//     P = exp2(S*scale*log2e - m)                  a thread per row, TMEM -> TMEM
//     O[256 x 256] += P[256 x 128] . V[128 x 256]  tcgen05.mma, P from TMEM, V as an MN-major operand, O stays in TMEM
// Each CTA holds 64 tokens of a K tile and 128 columns of a V tile, so a pair fetches a tile once (one CTA per tile fetched twice as
// much, 35 bytes a cycle and SM, and had room for one K and one V tile only; now two of each).  Why not more rows per CTA: O and two
// buffers of S fill the 512 columns of tensor memory.  Roles of the 16 warps:
//   0-3, 4-7  exponentials of the even and of the odd tiles, a thread per row; the row's reference maximum goes from one to the other
//             through shared memory.  (Two threads per row of every tile: the exponential units idle while S, the row maximum and the
//             store of P are waited for, 2950 cycles a tile.)
//   8-11      rotate the next item's Q in shared memory, then take O of this one through gate and copy engine to the output
//   12, 15    issue S and PV (even CTA only; the odd one's 12 passes its rotated Q on), 13 loads K, 14 deals the items and loads Q and V
// P is stored as packed bf16 over the first 64 columns of the S buffer just read; S of tile j+2 waits for PV of tile j to complete.  O is
// rescaled in TMEM only when a row maximum grows by more than 2^8 (the running reference maximum may lag; p then stays <= 256, exact
// for bf16 and fp32 l).
// Bound: the tensor pipe, 2137 of 2765 cycles a tile (68 % of a launch of 8 x 4096 tokens by counter); the rest is the completion of PV that
// S of the buffer waits for.  The chip's power cap comes before it in long runs (1560 MHz).  us with rope and gate, one CTA per 32 queries and
// pairs: 8 x 4096 tokens 623 -> 575, in bursts 533 -> 497; 64 x 512 227 -> 174; 32 of 16 to 512 67.5 -> 61.4.  Short prompts are bound by what
// comes first: loads from HBM by all SMs at once and the fetch of instructions, some 200 cycles for every eight (therefore loops where unrolled
// code would run once).
// The reference's rounding points are kept where they matter for the 2e-2 bar: p is rounded to bf16 for the PV
// product while l sums the fp32 p; scores are scaled in fp32 (the reference pre-scales q and re-rounds it to bf16).
// Every mbarrier wait is bounded; on expiry the role sets the device error flag and the CTA drains and exits.
#include "prefill.cuh"

namespace b200 {

constexpr int PU_PAIR_Q = 2 * PU_BQ;
constexpr int PU_SOFTMAX_WARPS = 8;
constexpr int PU_OUT_WARPS = 4;
constexpr int PU_THREADS = 512;
constexpr int PU_Q_BYTES = 128 * HEAD_DIM * 2;      // 64 KiB: 4 column blocks of [128 rows][64]
constexpr int PU_KV_BYTES = PU_TKV * HEAD_DIM;      // 32 KiB: half a tile, K 64 tokens, V 128 columns
constexpr int PU_STAGE = 3, PU_STAGE_BYTES = 32 * 64;  // buffers of an output warp: 32 columns of its 32 rows, first the gates, then the output
constexpr int PU_SMEM = PU_Q_BYTES + 4 * PU_KV_BYTES + PU_OUT_WARPS * PU_STAGE * PU_STAGE_BYTES;
constexpr int PU_ITEMS = 4;                         // work items in flight per pair
constexpr int PU_GROUP = 64;                        // most sequences whose items are dealt together
constexpr int PU_REGS_SOFTMAX = 160, PU_REGS_OUT = 120, PU_REGS_ISSUE = 64;
constexpr int PU_REGS = 65536 / PU_THREADS;         // what __launch_bounds__ leaves a thread, and ptxas gives (the host checks)
static_assert(2 * PU_REGS_SOFTMAX + PU_REGS_OUT + PU_REGS_ISSUE <= PU_THREADS / 128 * PU_REGS, "shares of the registers the CTA is launched with");
constexpr float PU_LOG2E = 1.4426950408889634f;

// Fused path, first kernel: rotate K at its position, scatter K (rotated) and V into the paged cache and keep a
// packed copy of the rotated K [T, H_kv, 256] for the attention kernel's TMA loads (so the rotation is computed once
// per token, not once per consumer tile).  One warp per (token, kv head) row, each lane 8 consecutive dims;
// grid = (pages of the longest sequence, H_kv, B).
__global__ void __launch_bounds__(128)
rope_scatter_kernel(const __nv_bfloat16* __restrict__ k, int64_t k_t, int64_t k_h, const __nv_bfloat16* __restrict__ v,
                    int64_t v_t, int64_t v_h, __nv_bfloat16* __restrict__ k_cache, __nv_bfloat16* __restrict__ v_cache,
                    int64_t kc_p, int64_t kc_h, int64_t kc_s, int64_t vc_p, int64_t vc_h, int64_t vc_s,
                    const int32_t* __restrict__ block_table, int64_t bt_b, const int32_t* __restrict__ cu_seqlens,
                    const void* __restrict__ position_ids, int ids_are_int64, const float* __restrict__ inv_freq,
                    int rotary_half, __nv_bfloat16* __restrict__ k_rot, int num_kv_heads) {
  const int lp = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_trigger();  // the attention kernel behind this one may start: it waits for this grid before it reads k_rot
  const int seq_start = cu_seqlens[b];
  const int seq_len = cu_seqlens[b + 1] - seq_start;
  if (lp * PAGE >= seq_len) return;
  const int64_t phys = block_table[b * bt_b + lp];
  const int lanes_half = rotary_half / 8;
  const bool in_rot = lane < 2 * lanes_half;
  const bool first = lane < lanes_half;
  const int partner = first ? lane + lanes_half : lane - lanes_half;
  const int dbase = (in_rot ? (first ? lane : partner) : 0) * 8;
  const float freq = lane < rotary_half ? inv_freq[lane] : 0.f;  // rotary_half <= 32: one angle per lane
  // a warp's four token rows (slots warp, warp + 4, ...): every row's loads are requested before the first is used
  constexpr int ROWS = PAGE / 4;
  uint4 kraw[ROWS], vraw[ROWS];
  int64_t pid[ROWS];
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    const int tok = lp * PAGE + warp + 4 * i;
    if (tok < seq_len) {
      const int64_t t = seq_start + tok;
      kraw[i] = *reinterpret_cast<const uint4*>(k + t * k_t + h * k_h + lane * 8);
      vraw[i] = *reinterpret_cast<const uint4*>(v + t * v_t + h * v_h + lane * 8);
      pid[i] = rotary_half == 0 ? 0
               : ids_are_int64 ? static_cast<const int64_t*>(position_ids)[t]
                               : static_cast<int64_t>(static_cast<const int32_t*>(position_ids)[t]);
    }
  }
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    const int slot = warp + 4 * i;
    const int tok = lp * PAGE + slot;
    if (tok >= seq_len) break;
    const int64_t t = seq_start + tok;
    uint32_t kw[4] = {kraw[i].x, kraw[i].y, kraw[i].z, kraw[i].w};
    if (rotary_half > 0) {
      // the warp computes the row's angles once, one sincosf per lane, and hands them round by shuffles (the same
      // full-range sincosf of float(pos) * inv_freq as before, so the rotated bytes do not change)
      float sn = 0.f, cs = 1.f;
      if (lane < rotary_half) sincosf(static_cast<float>(pid[i]) * freq, &sn, &cs);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t other = __shfl_sync(0xffffffffu, kw[j], in_rot ? partner : lane);
        const float s0 = __shfl_sync(0xffffffffu, sn, dbase + 2 * j), c0 = __shfl_sync(0xffffffffu, cs, dbase + 2 * j);
        const float s1 = __shfl_sync(0xffffffffu, sn, dbase + 2 * j + 1), c1 = __shfl_sync(0xffffffffu, cs, dbase + 2 * j + 1);
        if (in_rot) {
          const uint32_t fa = first ? kw[j] : other;
          const uint32_t fb = first ? other : kw[j];
          float f0, g0, f1, g1;
          rope_pair(bf16_lo(fa), bf16_lo(fb), s0, c0, f0, g0);
          rope_pair(bf16_hi(fa), bf16_hi(fb), s1, c1, f1, g1);
          kw[j] = first ? pack_bf16(f0, f1) : pack_bf16(g0, g1);
        }
      }
    }
    const uint4 krot = make_uint4(kw[0], kw[1], kw[2], kw[3]);
    *reinterpret_cast<uint4*>(k_cache + phys * kc_p + h * kc_h + slot * kc_s + lane * 8) = krot;
    *reinterpret_cast<uint4*>(k_rot + (t * num_kv_heads + h) * HEAD_DIM + lane * 8) = krot;
    *reinterpret_cast<uint4*>(v_cache + phys * vc_p + h * vc_h + slot * vc_s + lane * 8) = vraw[i];
  }
}



// ---- the pair's ring of work items: what every role of a CTA reads, written by its last warp
struct PrefillItem {
  int start, len, q0, h, tiles;  // first packed row and length of the sequence, the pair's first query, kv head, kv tiles (0: no more)
};

// SLOTS: sequences of a group per lane of the warp that deals them
template <bool FUSED, int SLOTS>
__global__ void __launch_bounds__(PU_THREADS, 1)
prefill_pair_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_gate,
                    const __grid_constant__ CUtensorMap map_out, const __grid_constant__ PrefillUmmaParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // `lead_*`: waited for by the issuer, the even CTA of the pair; the others are each CTA's own
  __shared__ uint64_t lead_k[2], lead_v[2], lead_q, lead_p[2][2], lead_o, lead_s[2], bar_q, bar_rot, bar_s[2], bar_pv[2], bar_m[4][2][2], bar_g[PU_OUT_WARPS][PU_STAGE], bar_l[PU_ITEMS], item_full[PU_ITEMS], item_free[PU_ITEMS];
  __shared__ uint32_t tmem_slot;
  __shared__ PrefillItem items[PU_ITEMS];
  __shared__ float row_ref[2][2][128];                // [tile parity][item parity][row]: the reference of the last tile of that parity
  __shared__ float row_end[PU_ITEMS][2][2][128];      // [item][tile parity][reference, sum][row]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_ctarank();
  uint8_t* q_s = smem_raw;
  uint8_t* k_s = q_s + PU_Q_BYTES;
  uint8_t* v_s = k_s + 2 * PU_KV_BYTES;
  uint8_t* out_s = v_s + 2 * PU_KV_BYTES;
  const bool aligned = (smem_u32(smem_raw) & 1023u) == 0;  // swizzled tiles need it; always so with __align__(1024)

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&lead_k[i], 1);
      mbar_init(&lead_v[i], 1);
      mbar_init(&lead_p[i][0], PU_SOFTMAX_WARPS);
      mbar_init(&lead_p[i][1], PU_SOFTMAX_WARPS);  // the warps of one parity in both CTAs
      mbar_init(&bar_s[i], 1);
      mbar_init(&bar_pv[i], 1);
    }
    mbar_init(&lead_q, FUSED ? PU_OUT_WARPS + 1 : 1);
    mbar_init(&bar_rot, PU_OUT_WARPS);
    mbar_init(&lead_o, 2 * PU_OUT_WARPS);
    mbar_init(&lead_s[0], 1);
    mbar_init(&lead_s[1], 1);
    mbar_init(&bar_q, 1);
    for (int i = 0; i < 4; ++i) {
      for (int n = 0; n < 4; ++n) mbar_init(&bar_m[i][n >> 1][n & 1], 1);
      for (int n = 0; n < PU_STAGE; ++n) mbar_init(&bar_g[i][n], 1);
    }
    for (int i = 0; i < PU_ITEMS; ++i) {
      mbar_init(&bar_l[i], PU_SOFTMAX_WARPS);
      mbar_init(&item_full[i], 1);
      mbar_init(&item_free[i], PU_SOFTMAX_WARPS + PU_OUT_WARPS + 1 + (rank == 0 ? 2 : FUSED ? 1 : 0));
    }
    mbar_fence_init();
  }
  // ---- the items (warp 14).  They are dealt to the pairs forth and back, group by group of sequences, in a group longest first: all blocks in
  // the highest of its levels of 64 queries, then those in the next, and so on.  A group's lengths are read once, and a level is found by
  // halving: `above(l)` counts the (sequence, level) blocks from level l on.  Walked level by level, 32 lengths read at a time and from the
  // longest level that the caller names on, the list took 1024 prompts of 16 tokens 371 us where that was 4096, now 105.  The code is kept
  // short, and the first item found while the pair meets: with four sequences per lane, or loops over shared memory, 8 prompts of 1024 tokens
  // took 64.4 us (62.5 with one).
  const int pairs = gridDim.x >> 1, me = blockIdx.x >> 1, heads = p.num_kv_heads;
  int first = 0, from[SLOTS], to[SLOTS], levels[SLOTS];  // the group's first sequence; bounds and levels of a lane's sequences
  int blocks = 0, top = 0, over_top = 0;  // blocks of the group; items to come have none of the over_top from level `top` on
  uint32_t base = 0;  // items of the groups in front (q, k, v and the output of 2^32 of them do not fit the device)
  auto above = [&](int level) {
    int n = 0;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) n += max(levels[s] - level, 0);
    return __reduce_add_sync(0xffffffffu, n);
  };
  auto open_group = [&]() {
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      const int nth = s * 32 + lane, b = first + nth;
      from[s] = to[s] = 0;
      if (nth < p.group && b < p.batch) from[s] = p.cu_seqlens[b], to[s] = p.cu_seqlens[b + 1];
    }
    top = 0;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      levels[s] = (min(max(to[s] - from[s], 0), p.max_seqlen) + PU_PAIR_Q - 1) / PU_PAIR_Q;
      top = max(top, levels[s]);
    }
    top = __reduce_max_sync(0xffffffffu, top);
    blocks = above(0);
    over_top = 0;
  };
  auto find = [&](int i, PrefillItem& it) {
    const uint32_t target = static_cast<uint32_t>(i) * pairs + ((i & 1) ? pairs - 1 - me : me);
    it.tiles = 0;
    while (first < p.batch) {
      const int block = static_cast<int>((target - base) / heads);
      if (block < blocks) {
        int level = 0;                               // above(level) > block >= over_top = above(top)
        while (top - level > 1) {
          const int mid = (level + top) >> 1, n = above(mid);
          if (n > block) level = mid;
          else top = mid, over_top = n;
        }
        int nth = block - over_top;
        it.q0 = level * PU_PAIR_Q;
        it.h = static_cast<int>(target - base) - block * heads;
#pragma unroll
        for (int s = 0; s < SLOTS; ++s) {
          const uint32_t has = __ballot_sync(0xffffffffu, levels[s] > level);
          const int here = __popc(has);
          if (nth >= 0 && nth < here) {
            const bool mine = ((has >> lane) & 1) != 0 && __popc(has & ((1u << lane) - 1)) == nth;
            const int src = __ffs(__ballot_sync(0xffffffffu, mine)) - 1;
            it.start = __shfl_sync(0xffffffffu, from[s], src);
            it.len = __shfl_sync(0xffffffffu, to[s], src) - it.start;
          }
          nth -= here;
        }
        it.tiles = (min(it.q0 + PU_PAIR_Q, it.len) + PU_TKV - 1) / PU_TKV;
        break;
      }
      base += static_cast<uint32_t>(blocks) * heads;
      first += p.group;
      if (first < p.batch) open_group();
    }
  };
  PrefillItem it0;
  if (warp == 14) {  // while the pair meets
    open_group();
    find(0, it0);
  }
  if (warp == 12) tmem_alloc_pair(&tmem_slot, PU_TMEM_COLS);
  if (warp == 13 && lane == 0) {
    prefetch_tensormap(&map_q);
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
  }
  tc_fence_before_sync();
  cluster_sync();  // barriers of both CTAs are set up, tensor memory is there
  tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;
  const uint32_t tmem_o = tmem + 2 * PU_TKV;
  bool ok = aligned;

  // item i of this pair; the whole warp
  auto release = [&](int i) {
    __syncwarp();
    if (lane == 0) mbar_arrive(&item_free[i & (PU_ITEMS - 1)]);
  };
  auto fetch = [&](int i, PrefillItem& it, bool keep = false) {
    ok = warp_wait_bounded(&item_full[i & (PU_ITEMS - 1)], (i / PU_ITEMS) & 1, ok);
    it.tiles = 0;
    if (ok) it = items[i & (PU_ITEMS - 1)];
    if (!keep) release(i);
    return ok && it.tiles > 0;
  };

  if (warp >= 12) {
    set_registers<PU_REGS_ISSUE, PU_REGS>();
    PrefillItem it;
    if (warp == 14) {
      // ---------------------------------------------------------------- the items; TMA producer: Q, and this CTA's 128 columns of every V tile
      // One item is made while the one in front of it is loaded.
      auto make = [&](int i, PrefillItem& it) {
        if (i > 0) find(i, it);
        if (i >= PU_ITEMS) ok = warp_wait_bounded(&item_free[i & (PU_ITEMS - 1)], (i / PU_ITEMS - 1) & 1, ok);
        if (ok && lane == 0) {
          items[i & (PU_ITEMS - 1)] = it;
          mbar_arrive(&item_full[i & (PU_ITEMS - 1)]);
        }
        return ok && it.tiles > 0;
      };
      const uint32_t full[2] = {cluster_map(smem_u32(&lead_v[0]), 0), cluster_map(smem_u32(&lead_v[1]), 0)};
      const uint32_t full_q = cluster_map(smem_u32(&lead_q), 0);
      const int q_off = static_cast<int>(rank) * PU_BQ;
      PrefillItem next;
      it = it0;
      bool more = ok && make(0, it);
      for (int i = 0, g = 0; more; ++i, it = next) {
        // the last S of the item in front read Q; the V tile of that S was asked for behind PV of two tiles before it, so this
        // barrier's phase in front of it is over
        if (g >= 1) ok = warp_wait_bounded(&bar_s[(g - 1) & 1], ((g - 1) >> 1) & 1, ok);
        if (!ok) break;
        if (lane == 0) {
          if (FUSED) {
            mbar_expect_tx(&bar_q, PU_Q_BYTES);
            tma_load_5d(q_s, &map_q, 0, 0, it.h, it.start + it.q0 + q_off, 0, &bar_q);
          } else {
            if (rank == 0) mbar_expect_tx(&lead_q, 2 * PU_Q_BYTES);
            tma_load_5d_pair(q_s, &map_q, 0, 0, it.h, it.start + it.q0 + q_off, 0, full_q);
          }
        }
        for (int j = 0; j < it.tiles; ++j, ++g) {
          const int s = g & 1;
          if (g >= 2) ok = warp_wait_bounded(&bar_pv[s], ((g >> 1) - 1) & 1, ok);  // PV of tile g-2 done: its V is free
          if (!ok) break;
          if (lane == 0) {
            if (rank == 0) mbar_expect_tx(&lead_v[s], 2 * PU_KV_BYTES);
            tma_load_4d_pair(v_s + s * PU_KV_BYTES, &map_v, 0, it.start + j * PU_TKV, 2 * static_cast<int>(rank), it.h, full[s]);
          }
          if (j == (i == 0 && it.tiles > 1)) {  // (the first two V tiles wait for nobody)
            more = make(i + 1, next);
            if (more && lane == 0) tma_prefetch_5d(&map_q, 0, 0, next.h, next.start + next.q0 + q_off, 0);
          }
        }
      }
    } else if (warp == 13) {
      // ---------------------------------------------------------------- TMA producer: this CTA's 64 tokens of every K tile
      // Fused form: started while the rope + scatter kernel still runs (programmatic dependent launch).  Everything else of the
      // prologue, Q and V overlap with it; the rotated K it writes is read only after it has completed.
      if (FUSED) pdl_wait();
      const uint32_t full[2] = {cluster_map(smem_u32(&lead_k[0]), 0), cluster_map(smem_u32(&lead_k[1]), 0)};
      for (int i = 0, g = 0; fetch(i, it); ++i) {
        for (int j = 0; j < it.tiles; ++j, ++g) {
          const int s = g & 1;
          if (g >= 2) ok = warp_wait_bounded(&bar_s[s], ((g >> 1) - 1) & 1, ok);  // S of tile g-2 done: its K is free
          if (!ok) break;
          if (lane == 0) {
            if (rank == 0) mbar_expect_tx(&lead_k[s], 2 * PU_KV_BYTES);
            tma_load_4d_pair(k_s + s * PU_KV_BYTES, &map_k, 0, it.start + j * PU_TKV + static_cast<int>(rank) * (PU_TKV / 2), 0, it.h, full[s]);
          }
        }
      }
    } else if (warp == 12 && rank == 0) {
      // ---------------------------------------------------------------- issuer of S for the pair (the whole warp walks, lane 0 issues)
      const bool leader = lane == 0;
      const uint32_t idesc_s = idesc_bf16_f32(256, PU_TKV, false, false);
      const uint32_t q_addr = smem_u32(q_s), k_addr = smem_u32(k_s);
      for (int i = 0, g = 0; fetch(i, it); ++i) {
        ok = warp_wait_cluster(&lead_q, i & 1, ok);
        for (int j = 0; j < it.tiles; ++j, ++g) {
          const int s = g & 1;
          ok = ok && mbar_wait_bounded(&lead_k[s], (g >> 1) & 1);
          // S(g) overwrites the buffer whose first columns hold P(g-2): the PV product that reads them from tensor
          // memory must have COMPLETED, issue order alone does not protect an operand in tensor memory
          if (g >= 2) ok = ok && mbar_wait_bounded(&bar_pv[s], ((g >> 1) - 1) & 1);
          if (!ok) break;
          tc_fence_after_sync();
#pragma unroll
          for (int ks = 0; ks < HEAD_DIM / 16; ++ks)
            umma_ss_pair(tmem + s * PU_TKV, smem_desc_sw128(q_addr + (ks >> 2) * (128 * 128) + (ks & 3) * 32, 16, 1024),
                         smem_desc_sw128(k_addr + s * PU_KV_BYTES + (ks >> 2) * (PU_TKV / 2 * 128) + (ks & 3) * 32, 16, 1024), idesc_s, ks > 0,
                         leader);
          umma_commit_pair(&bar_s[s], leader);
          if (leader) mbar_arrive(&lead_s[s]);
        }
      }
    } else if (rank == 1) {
      // ---------------------------------------------------------------- the odd CTA's rotated Q, handed to the issuer in the even one
      // The product that reads these rows of shared memory is the other CTA's, so they are released at cluster scope.  By a warp that has no
      // stores of its own: a release waits for them (by the output warps themselves 32 prompts of 16 to 512 tokens take 63.7 us, so 61.4).
      if (FUSED && warp == 12) {
        const uint32_t ready_q = cluster_map(smem_u32(&lead_q), 0);
        for (int i = 0; fetch(i, it); ++i) {
          ok = warp_wait_bounded(&bar_rot, i & 1, ok);
          if (ok && lane == 0) mbar_arrive_cluster(ready_q);
        }
      }
    } else {
      // ---------------------------------------------------------------- issuer of PV for the pair
      // Inside an item S of the tile behind goes into the pipe first: PV has its operand later anyway, and free to overtake one another
      // the two issuers end in two tiles' S, then both PV (3025 cycles a tile of 4096-token prompts, 2765 in this order).  From one item to the next
      // nobody waits: the next S may need a Q that is still on its way.
      const bool leader = lane == 0;
      const uint32_t idesc_o = idesc_bf16_f32(256, HEAD_DIM, false, true);
      const uint32_t v_addr = smem_u32(v_s);
      for (int i = 0, g = 0; fetch(i, it); ++i) {
        for (int j = 0; j < it.tiles; ++j, ++g) {
          const int s = g & 1;
          ok = ok && mbar_wait_bounded(&lead_s[s], (g >> 1) & 1);
          if (j + 1 < it.tiles) ok = ok && mbar_wait_bounded(&lead_s[s ^ 1], ((g + 1) >> 1) & 1);
          ok = ok && mbar_wait_bounded(&lead_v[s], (g >> 1) & 1);
          if (j == 0 && i > 0) ok = ok && mbar_wait_bounded(&lead_o, (i - 1) & 1);  // O of the item in front has been read
#pragma unroll
          for (int half = 0; half < 2; ++half) {  // the second 64 tokens' exponentials are computed under the first 64's product
            ok = ok && mbar_wait_bounded(&lead_p[s][half], (g >> 1) & 1);
            if (!ok) break;
            tc_fence_after_sync();
#pragma unroll
            for (int kt = half * 4; kt < half * 4 + 4; ++kt)
              umma_ts_pair(tmem_o, tmem + s * PU_TKV + kt * 8,  // P: 16 tokens = 8 packed columns per step
                           smem_desc_sw128(v_addr + s * PU_KV_BYTES + kt * 2048, PU_TKV * 128, 1024), idesc_o, j > 0 || kt > 0, leader);
          }
          if (!ok) break;
          umma_commit_pair(&bar_pv[s], leader);
        }
      }
    }
    if (!ok) {
      if (lane == 0) atomicExch(p.err, 1);
      // copies in flight signal barriers that may be the other CTA's: give them their time before the shared memory goes away
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 100000) __nanosleep(1000);
    }
  } else if (warp >= 8) {
    // ------------------------------------------------------------------ rope of the next item's Q, output of this one
    set_registers<PU_REGS_OUT, PU_REGS>();
    
    const int row = tid - 8 * 32;              // TMEM lane; row = token*4 + head
    const uint32_t lane_base = static_cast<uint32_t>(row & ~31) << 16;
    const uint32_t read_o = cluster_map(smem_u32(&lead_o), 0);
    uint8_t* stage = out_s + (warp - 8) * (PU_STAGE * PU_STAGE_BYTES);  // of [32 rows][32 columns], 64-byte swizzle
    auto rope = [&](const PrefillItem& it, int i) {
      // rotary embedding of this row's q in place (dims [0,32) and [32,64) live in column block 0, chunks c, c+4)
      const int q_tok = it.q0 + static_cast<int>(rank) * PU_BQ + (row >> 2);
      const int64_t t = it.start + min(q_tok, it.len - 1);
      const int64_t pid = p.ids_are_int64 ? static_cast<const int64_t*>(p.position_ids)[t]
                                          : static_cast<int64_t>(static_cast<const int32_t*>(p.position_ids)[t]);
      const float posf = static_cast<float>(pid);
      // the four rows of a token share their angles: each lane of a quad computes 8 of the 32 (sin, cos) pairs
      // the gate row is the output's: asked into the L2 now
#pragma unroll
      for (int n = 0; n < 4; ++n)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p.gate + t * p.gate_t + (it.h * GROUP + (row & 3)) * HEAD_DIM + n * 64));
      // (sin, cos) of the warp's eight tokens, one frequency per lane, while Q travels; in loops: code that runs once per item is
      // fetched as slowly as it is long
      const float freq = p.inv_freq[lane];
      float2* angles = reinterpret_cast<float2*>(stage);  // [8 tokens][32]
#pragma unroll 1
      for (int n = 0; n < 8; ++n) {
        float2 sc;
        sincosf(__shfl_sync(0xffffffffu, posf, n * 4) * freq, &sc.x, &sc.y);
        angles[n * 32 + lane] = sc;
      }
      __syncwarp();
      ok = warp_wait_bounded(&bar_q, i & 1, ok);
      if (!ok) return;
      uint8_t* qrow = q_s + row * 128;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {  // chunk c holds dims [8c, 8c+8), chunk c+4 their partners [32+8c, 40+8c)
        uint4* pa = reinterpret_cast<uint4*>(qrow + ((c ^ (row & 7)) << 4));
        uint4* pb = reinterpret_cast<uint4*>(qrow + (((c + 4) ^ (row & 7)) << 4));
        const uint4 va = *pa, vb = *pb;
        uint32_t wa[4] = {va.x, va.y, va.z, va.w}, wb[4] = {vb.x, vb.y, vb.z, vb.w};
        const float4* at = reinterpret_cast<const float4*>(angles + (lane >> 2) * 32 + c * 8);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float4 sc = at[k];  // sin, cos of angle 8c + 2k and of the next
          float f0, g0, f1, g1;
          rope_pair(bf16_lo(wa[k]), bf16_lo(wb[k]), sc.x, sc.y, f0, g0);
          rope_pair(bf16_hi(wa[k]), bf16_hi(wb[k]), sc.z, sc.w, f1, g1);
          wa[k] = pack_bf16(f0, f1);
          wb[k] = pack_bf16(g0, g1);
        }
        *pa = make_uint4(wa[0], wa[1], wa[2], wa[3]);
        *pb = make_uint4(wb[0], wb[1], wb[2], wb[3]);
      }
      // The rotated rows are the tensor core's to read: fenced to its proxy, and handed to the issuer of S, in the odd CTA through warp 12
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(rank == 0 ? &lead_q : &bar_rot);
    };
    PrefillItem it, next;
    bool more = fetch(0, it, true);
    if (FUSED && more) rope(it, 0);
    for (int i = 0, g = 0, n = 0; more; ++i, it = next) {  // n: 32-column pieces so far
      g += it.tiles;
      more = fetch(i + 1, next, true);
      if (lane == 0) bulk_wait_read();  // the buffers of the item in front
      __syncwarp();
      if (FUSED && more) rope(next, i + 1);
      const int q_tok0 = it.q0 + static_cast<int>(rank) * PU_BQ + (warp - 8) * 8, tok0 = it.start + q_tok0;
      const bool whole = q_tok0 + 8 <= it.len;  // eight tokens of the sequence: a tile for the copy engine; else row by row
      auto load_gate = [&](int c) {
        uint64_t* bar = &bar_g[warp - 8][(n + c) % PU_STAGE];
        mbar_expect_tx(bar, PU_STAGE_BYTES);
        tma_load_5d(stage + (n + c) % PU_STAGE * PU_STAGE_BYTES, &map_gate, 0, 0, it.h, tok0, c, bar);
      };
      if (FUSED && lane == 0) {
        load_gate(0);
        load_gate(1);
      }
      const int slot = i & (PU_ITEMS - 1);
      ok = warp_wait_bounded(&bar_l[slot], (i / PU_ITEMS) & 1, ok);
      // bar_l is behind S of the item's last tile, S behind PV of two tiles before it: the phase in front of this one is over
      ok = warp_wait_bounded(&bar_pv[(g - 1) & 1], ((g - 1) >> 1) & 1, ok);
      tc_fence_after_sync();
      // even and odd tiles summed against references of their own; O stands at the larger, the last tile's
      const float m0 = row_end[slot][0][0][row], m1 = row_end[slot][1][0][row], m = fmaxf(m0, m1);
      const float inv_l = 1.f / (row_end[slot][0][1][row] * ex2_fast(m0 - m) + row_end[slot][1][1][row] * ex2_fast(m1 - m));
      // o sigmoid(g) = o/2 tanh(g/2) + o/2
      const uint64_t inv2 = FUSED ? f32x2(0.5f * inv_l, 0.5f * inv_l) : f32x2(inv_l, inv_l);
      const __nv_bfloat162 half = __floats2bfloat162_rn(0.5f, 0.5f);
#pragma unroll 1
      for (int c = 0; c < HEAD_DIM / 32 && ok; ++c) {
        uint8_t* buf = stage + (n + c) % PU_STAGE * PU_STAGE_BYTES;
        uint4* mine = reinterpret_cast<uint4*>(buf + lane * 64);  // chunk k of this row at k ^ (row / 2 % 4)
        uint32_t o[32];
        tmem_ld32(tmem_o + lane_base + c * 32, o);
        if (FUSED) {
          ok = warp_wait_bounded(&bar_g[warp - 8][(n + c) % PU_STAGE], ((n + c) / PU_STAGE) & 1, ok);
        } else {
          if (lane == 0) bulk_wait_read_but<PU_STAGE - 1>();
          __syncwarp();
        }
        tmem_ld_wait();
        if (c == HEAD_DIM / 32 - 1) {  // O is read: the next item's first product may overwrite it
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster_plain(read_o);
        }
        uint4 v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          uint32_t gs[4] = {}, w[4];
          if (FUSED) {
            const uint4 gv = mine[k ^ ((lane >> 1) & 3)];
            gs[0] = gv.x; gs[1] = gv.y; gs[2] = gv.z; gs[3] = gv.w;
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            uint64_t x = f32x2_mul(f32x2(o[k * 8 + e * 2], o[k * 8 + e * 2 + 1]), inv2);
            if (FUSED) {
              const __nv_bfloat162 h2 = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&gs[e]), half);
              const uint32_t hw = *reinterpret_cast<const uint32_t*>(&h2);
              x = f32x2_fma(x, f32x2(tanh_fast(bf16_lo(hw)), tanh_fast(bf16_hi(hw))), x);
            }
            w[e] = pack_bf16x2(x);
          }
          v[k] = make_uint4(w[0], w[1], w[2], w[3]);
        }
        if (whole) {
#pragma unroll
          for (int k = 0; k < 4; ++k) mine[k ^ ((lane >> 1) & 3)] = v[k];
          fence_proxy_async();
        } else if (q_tok0 + (lane >> 2) < it.len) {
          __nv_bfloat16* out = p.out + static_cast<int64_t>(tok0 + (lane >> 2)) * p.out_t + (it.h * GROUP + (lane & 3)) * p.out_h + c * 32;
#pragma unroll
          for (int k = 0; k < 4; ++k) reinterpret_cast<uint4*>(out)[k] = v[k];
        }
        __syncwarp();
        if (lane == 0) {
          if (whole) tma_store_5d(&map_out, 0, 0, it.h, tok0, c, buf);
          if (FUSED && c + 2 < HEAD_DIM / 32) {
            bulk_wait_read_but<1>();  // the piece in front has left the buffer that the one after the next comes to
            load_gate(c + 2);
          }
        }
      }
      if (!ok) break;
      n += HEAD_DIM / 32;
      // only now: the item's place in the ring is also that of its sums
      release(i);
    }
    if (lane == 0) bulk_wait_read();
    if (!ok && lane == 0) {
      atomicExch(p.err, 1);
      for (int i = 0; i < PU_STAGE; ++i) mbar_wait_bounded(&bar_g[warp - 8][i], 0, 1u << 12);  // gates in flight
    }
  } else {
    // ------------------------------------------------------------------ softmax
    set_registers<PU_REGS_SOFTMAX, PU_REGS>();
    // Warps 0-3 take the even tiles of the pair's stream, warps 4-7 the odd ones, one thread per row: while one of the two warps of a
    // scheduler waits for its scores, its row's reference or the store of P, the other has its exponentials computed.
    const int quarter = warp & 3, par = warp >> 2;
    const int row = 32 * quarter + lane;       // TMEM lane; row = token*4 + head
    const uint32_t lane_base = static_cast<uint32_t>(32 * quarter) << 16;
    const uint32_t tmem_s = tmem + lane_base + par * PU_TKV;
    const uint32_t ready_p = cluster_map(smem_u32(&lead_p[par][0]), 0);
    const float scale = p.scale_log2;
    uint32_t refs[2] = {0, 0};                 // references taken over from the other warp so far, in even and odd items
    PrefillItem it;
    for (int i = 0, g0 = 0; fetch(i, it); ++i) {
      const int q_last = min(it.q0 + static_cast<int>(rank) * PU_BQ + (row >> 2), it.len - 1);
      float m_ref = -INFINITY, l_run = 0.f;
      for (int j = (g0 ^ par) & 1; j < it.tiles; j += 2) {
        const int g = g0 + j;
        ok = warp_wait_bounded(&bar_s[par], (g >> 1) & 1, ok);
        if (!ok) break;
        tc_fence_after_sync();
        // causal and inside the sequence; only tiles on the diagonal or at the sequence end have columns to mask
        const int lim = q_last - j * PU_TKV;   // last valid column
        const bool edge = __any_sync(0xffffffffu, lim < PU_TKV - 1);
        // the row maximum of the raw scores; the scale (> 0) is folded into the exponent below
        float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll 1
        for (int c0 = 0; c0 < PU_TKV; c0 += 64) {
          uint32_t r[2][32];
          tmem_ld32(tmem_s + c0, r[0]);
          tmem_ld32(tmem_s + c0 + 32, r[1]);
          tmem_ld_wait();
          if (edge) {  // back into tensor memory, where the second pass finds it
#pragma unroll
            for (int c = 0; c < 64; ++c)
              if (c0 + c > lim) r[c >> 5][c & 31] = 0xff800000u;  // -inf
            tmem_st32(tmem_s + c0, r[0]);
            tmem_st32(tmem_s + c0 + 32, r[1]);
          }
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            mx0 = fmaxf(mx0, fmaxf(__uint_as_float(r[0][c]), __uint_as_float(r[0][c + 1])));
            mx1 = fmaxf(mx1, fmaxf(__uint_as_float(r[1][c]), __uint_as_float(r[1][c + 1])));
          }
        }
        if (edge) tmem_st_wait();
        const float m_tile = fmaxf(mx0, mx1) * scale;
        float m_use = m_tile;
        if (j > 0) {
          ok = warp_wait_bounded(&bar_m[quarter][par ^ 1][i & 1], ((i & 1) ? refs[1]++ : refs[0]++) & 1, ok);
          if (!ok) break;
          const float m_prev = row_ref[par ^ 1][i & 1][row], m_new = fmaxf(m_prev, m_tile);
          const bool need = m_new - m_prev > PU_TAU;
          m_use = need ? m_new : m_prev;
          if (j + 1 < it.tiles) {
            row_ref[par][i & 1][row] = m_use;
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_m[quarter][par][i & 1]);
          }
          if (__any_sync(0xffffffffu, need)) {
            // O must be at rest before it is rescaled: wait for the PV product of the tile in front
            ok = warp_wait_bounded(&bar_pv[par ^ 1], ((g - 1) >> 1) & 1, ok);
            if (!ok) break;
            tc_fence_after_sync();
            const float alpha = need ? ex2_fast(m_prev - m_new) : 1.f;
#pragma unroll 1
            for (int c0 = 0; c0 < HEAD_DIM; c0 += 32) {
              uint32_t o[32];
              tmem_ld32(tmem_o + lane_base + c0, o);
              tmem_ld_wait();
#pragma unroll
              for (int c = 0; c < 32; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * alpha);
              tmem_st32(tmem_o + lane_base + c0, o);
            }
          }
        } else if (it.tiles > 1) {
          row_ref[par][i & 1][row] = m_use;
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar_m[quarter][par][i & 1]);
        }
        l_run *= ex2_fast(m_ref - m_use);      // this parity's sum so far, against the reference of its last tile
        m_ref = m_use;
        // p = 2^(s*scale - m_ref): fp32 for l, bf16 for the PV product, stored as packed columns of the P tile (tokens 2c, 2c+1 in
        // column c) over the columns of S that have been read
        const uint64_t sc2 = f32x2(scale, scale), neg2 = f32x2(-m_use, -m_use);
        uint64_t sum0 = 0, sum1 = 0;
#pragma unroll 1
        for (int c0 = 0; c0 < PU_TKV; c0 += 64) {
          uint32_t r[2][32];
          tmem_ld32(tmem_s + c0, r[0]);
          tmem_ld32(tmem_s + c0 + 32, r[1]);
          tmem_ld_wait();
          uint32_t w[32];
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            const uint64_t x = f32x2_fma(f32x2(r[c >> 4][(2 * c) & 31], r[c >> 4][(2 * c + 1) & 31]), sc2, neg2);
            const uint64_t e = f32x2(ex2_fast(f32x2_lo(x)), ex2_fast(f32x2_hi(x)));
            if (c & 1) sum1 = f32x2_add(sum1, e);
            else sum0 = f32x2_add(sum0, e);
            w[c] = pack_bf16x2(e);
          }
          tmem_st32(tmem_s + (c0 >> 1), w);
          tmem_st_wait();
          tc_fence_before_sync();              // this warp's TMEM loads/stores before the arrive
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster_plain(ready_p + (c0 >> 6) * 8);
        }
        sum0 = f32x2_add(sum0, sum1);
        l_run += f32x2_lo(sum0) + f32x2_hi(sum0);
      }
      if (!ok) break;
      g0 += it.tiles;
      const int slot = i & (PU_ITEMS - 1);
      row_end[slot][par][0][row] = m_ref;
      row_end[slot][par][1][row] = l_run;
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_l[slot]);
    }
    if (!ok && lane == 0) atomicExch(p.err, 1);
  }
  tc_fence_before_sync();
  cluster_sync();  // nobody reads or signals the other CTA any more
  if (warp == 12) tmem_dealloc_pair(tmem, PU_TMEM_COLS);
}

}  // namespace b200

using namespace b200;

static bool mult8(int64_t x) { return (x & 7) == 0; }

// Sequences whose items are dealt together.  All of them balance best.  But the pairs go level by level, and between two levels of a sequence
// the K and V of all, and a level's rows of q, output and (row_tensors = 3) gate, pass through the L2 of 126 MB: beyond 80 MiB groups of 48.
// Not with six pairs or more to a (sequence, head): those read the same tiles at about the same time.  us, all together and in groups: 64 x
// 2048 tokens 1476 and 1260, 64 x 4096 4662 and 4229, 128 x 512 370 and 336, 12 x 4096 880 and 863; on the wrong side of the lines 8 x 4096
// (70 MiB) 502 and 522, 6 x 8192 1322 and 1345.
static int prefill_group(int batch, int total_tokens, int num_kv_heads, int row_tensors, int pairs) {
  const int64_t rows = total_tokens < static_cast<int64_t>(batch) * PU_PAIR_Q ? total_tokens : static_cast<int64_t>(batch) * PU_PAIR_Q;
  const int64_t pass = (2 * static_cast<int64_t>(total_tokens) + row_tensors * GROUP * rows) * num_kv_heads * HEAD_DIM * 2;
  int64_t groups = 1;
  if (pass > (80ll << 20) && static_cast<int64_t>(batch) * num_kv_heads * 6 > pairs) groups = (pass + (48ll << 20) - 1) / (48ll << 20);
  const int64_t group = (batch + groups - 1) / groups;
  return static_cast<int>(group < PU_GROUP ? group : PU_GROUP);
}

// Encodes the tensor maps and launches the attention kernel (FUSED adds rope on q and the output gate).
template <bool FUSED>
static int launch_prefill_umma(const PrefillTensors& t, PrefillUmmaParams p, int batch, int max_seqlen, cudaStream_t stream, const char* what) {
  const int num_kv_heads = t.num_kv_heads, sms = sm_count();
  B200_REQUIRE((max_seqlen + PU_BQ - 1) / PU_BQ <= 65535 && batch <= 65535 && num_kv_heads <= 65535,
               "%s: max_seqlen must be at most %d, batch and heads at most 65535 (got %d, %d, %d)", what, 65535 * PU_BQ,
               max_seqlen, batch, num_kv_heads);
  p.err = wait_timeout_flag();
  if (!p.err) return fail(ERR_RUNTIME, "%s: no error flag", what);
  p.scale_log2 = (1.0f / sqrtf(static_cast<float>(HEAD_DIM))) * PU_LOG2E;
  p.num_kv_heads = num_kv_heads;
  p.batch = batch;
  p.max_seqlen = max_seqlen;
  if (prefill_takes_short(FUSED, batch, t.tokens, max_seqlen, num_kv_heads)) return launch_prefill_short(FUSED, t, p, stream, what);
  CUtensorMap map_q, map_k, map_v, map_gate = {}, map_out;
  // of K a CTA loads 64 tokens of a head, of V 128 columns of 128 tokens
  if (!encode_prefill_q(&map_q, t) || !encode_prefill_kv(&map_k, t, t.k, t.k_t, t.k_h, PU_TKV / 2, HEAD_DIM / 64) ||
      !encode_prefill_kv(&map_v, t, t.v, t.v_t, t.v_h, PU_TKV, HEAD_DIM / 128))
    return fail(ERR_RUNTIME, "%s: cannot encode the tensor maps of q / k / v", what);
  {
    // gates and output as {32 cols, 4 heads of a group, groups, tokens, 8 column blocks}; one copy = 8 tokens of one group
    const uint64_t dims[5] = {32, GROUP, static_cast<uint64_t>(num_kv_heads), static_cast<uint64_t>(t.tokens), HEAD_DIM / 32};
    const uint64_t gs[4] = {HEAD_DIM * 2, HEAD_DIM * 2 * GROUP, static_cast<uint64_t>(p.gate_t) * 2, 64};
    const uint64_t os[4] = {static_cast<uint64_t>(p.out_h) * 2, static_cast<uint64_t>(p.out_h) * 2 * GROUP, static_cast<uint64_t>(p.out_t) * 2, 64};
    const uint32_t box[5] = {32, GROUP, 1, 8, 1};
    if ((FUSED && !encode_map_bf16_sw64(&map_gate, p.gate, 5, dims, gs, box)) || !encode_map_bf16_sw64(&map_out, p.out, 5, dims, os, box))
      return fail(ERR_RUNTIME, "%s: cannot encode the tensor maps of gate / out", what);
  }
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  const auto one = prefill_pair_kernel<FUSED, 1>, two = prefill_pair_kernel<FUSED, 2>;
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    for (const auto k : {one, two}) {
      if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, PU_SMEM) != cudaSuccess)
        return fail(ERR_RUNTIME, "%s: cannot raise dynamic shared memory to %d", what, PU_SMEM);
      cudaFuncAttributes attr;  // its warpgroups exchange registers: with fewer at the launch than they share out they would wait for good
      if (cudaFuncGetAttributes(&attr, k) != cudaSuccess || attr.numRegs != PU_REGS)
        return fail(ERR_RUNTIME, "%s: the kernel was not built with %d registers per thread", what, PU_REGS);
    }
    configured[dev] = true;
  }
  p.group = prefill_group(batch, t.tokens, num_kv_heads, FUSED ? 3 : 2, sms / 2);
  const int64_t most = static_cast<int64_t>((max_seqlen + PU_PAIR_Q - 1) / PU_PAIR_Q) * num_kv_heads * batch;
  const int pairs = static_cast<int>(most < sms / 2 ? most : sms / 2);
  // the fused form starts behind its own rope + scatter kernel while that one still runs (see the K producer)
  if (launch_pdl_cluster(FUSED, 2, p.group <= 32 ? one : two, dim3(2 * pairs), dim3(PU_THREADS), PU_SMEM, stream, map_q, map_k, map_v, map_gate,
                         map_out, p) !=
      cudaSuccess)
    return fail(ERR_LAUNCH, "%s: %s", what, cudaGetErrorString(cudaGetLastError()));
  return check_launch(what);
}

extern "C" int b200_gqa_varlen_causal(const void* q, int64_t q_stride_t, int64_t q_stride_h, const void* k,
                                      int64_t k_stride_t, int64_t k_stride_h, const void* v, int64_t v_stride_t,
                                      int64_t v_stride_h, void* out, int64_t out_stride_t, int64_t out_stride_h,
                                      const int32_t* cu_seqlens, int32_t batch, int32_t total_tokens,
                                      int32_t max_seqlen, int32_t num_q_heads, int32_t num_kv_heads, int32_t head_dim,
                                      b200_stream_t stream) {
  B200_REQUIRE(batch > 0 && batch <= 65535, "gqa_varlen_causal: batch must be in [1, 65535]");
  B200_REQUIRE(total_tokens > 0, "gqa_varlen_causal: total_tokens must be positive");
  B200_REQUIRE(head_dim == HEAD_DIM, "gqa_varlen_causal: head_dim must be %d (got %d)", HEAD_DIM, head_dim);
  B200_REQUIRE(num_kv_heads > 0 && num_q_heads == num_kv_heads * GROUP,
               "gqa_varlen_causal: needs %d Q heads per KV head (got %d/%d)", GROUP, num_q_heads, num_kv_heads);
  B200_REQUIRE(aligned16(q) && aligned16(k) && aligned16(v) && aligned16(out) && mult8(q_stride_t) &&
                   mult8(q_stride_h) && mult8(k_stride_t) && mult8(k_stride_h) && mult8(v_stride_t) &&
                   mult8(v_stride_h) && mult8(out_stride_t) && mult8(out_stride_h),
               "gqa_varlen_causal: tensors must be 16-byte aligned with strides that are multiples of 8");
  if (max_seqlen <= 0) return OK;
  PrefillUmmaParams p = {};
  p.out = static_cast<__nv_bfloat16*>(out);
  p.out_t = out_stride_t;
  p.out_h = out_stride_h;
  p.cu_seqlens = cu_seqlens;
  const PrefillTensors t = {q, k, v, q_stride_t, q_stride_h, k_stride_t, k_stride_h, v_stride_t, v_stride_h, total_tokens, num_kv_heads};
  return launch_prefill_umma<false>(t, p, batch, max_seqlen, reinterpret_cast<cudaStream_t>(stream), "gqa_varlen_causal");
}

extern "C" int b200_fused_prefill_attention(const void* q, int64_t q_stride_t, int64_t q_stride_h, const void* k,
                                            int64_t k_stride_t, int64_t k_stride_h, const void* v, int64_t v_stride_t,
                                            int64_t v_stride_h, const void* gate, int64_t gate_stride_t, void* k_cache,
                                            void* v_cache, int64_t kc_stride_p, int64_t kc_stride_h,
                                            int64_t kc_stride_s, int64_t vc_stride_p, int64_t vc_stride_h,
                                            int64_t vc_stride_s, const int32_t* block_table, int64_t bt_stride_b,
                                            const int32_t* cu_seqlens, const void* position_ids, int32_t ids_are_int64,
                                            const float* inv_freq, int32_t rotary_dim, void* k_rot_scratch, void* out,
                                            int32_t batch, int32_t total_tokens, int32_t max_seqlen,
                                            int32_t num_q_heads, int32_t num_kv_heads, int32_t head_dim,
                                            b200_stream_t stream) {
  B200_REQUIRE(batch > 0 && batch <= 65535, "fused_prefill_attention: batch must be in [1, 65535]");
  B200_REQUIRE(total_tokens > 0, "fused_prefill_attention: total_tokens must be positive");
  B200_REQUIRE(head_dim == HEAD_DIM, "fused_prefill_attention: head_dim must be %d (got %d)", HEAD_DIM, head_dim);
  B200_REQUIRE(num_kv_heads > 0 && num_q_heads == num_kv_heads * GROUP,
               "fused_prefill_attention: needs %d Q heads per KV head (got %d/%d)", GROUP, num_q_heads, num_kv_heads);
  B200_REQUIRE(rotary_dim == 64, "fused_prefill_attention: rotary_dim must be 64 (got %d)", rotary_dim);
  B200_REQUIRE(inv_freq != nullptr && position_ids != nullptr && k_rot_scratch != nullptr,
               "fused_prefill_attention: NULL rope inputs or scratch");
  B200_REQUIRE(aligned16(q) && aligned16(k) && aligned16(v) && aligned16(out) && aligned16(gate) &&
                   aligned16(k_cache) && aligned16(v_cache) && aligned16(k_rot_scratch) && mult8(q_stride_t) &&
                   mult8(q_stride_h) && mult8(k_stride_t) && mult8(k_stride_h) && mult8(v_stride_t) &&
                   mult8(v_stride_h) && mult8(gate_stride_t) && mult8(kc_stride_p) && mult8(kc_stride_h) &&
                   mult8(kc_stride_s) && mult8(vc_stride_p) && mult8(vc_stride_h) && mult8(vc_stride_s),
               "fused_prefill_attention: tensors must be 16-byte aligned with strides that are multiples of 8");
  if (max_seqlen <= 0) return OK;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const dim3 grid((max_seqlen + PAGE - 1) / PAGE, num_kv_heads, batch);
  rope_scatter_kernel<<<grid, 128, 0, st>>>(
      static_cast<const __nv_bfloat16*>(k), k_stride_t, k_stride_h, static_cast<const __nv_bfloat16*>(v), v_stride_t,
      v_stride_h, static_cast<__nv_bfloat16*>(k_cache), static_cast<__nv_bfloat16*>(v_cache), kc_stride_p, kc_stride_h,
      kc_stride_s, vc_stride_p, vc_stride_h, vc_stride_s, block_table, bt_stride_b, cu_seqlens, position_ids,
      ids_are_int64, inv_freq, rotary_dim / 2, static_cast<__nv_bfloat16*>(k_rot_scratch), num_kv_heads);
  int rc = check_launch("fused_prefill_attention (rope + scatter)");
  if (rc != OK) return rc;
  PrefillUmmaParams p = {};
  p.out = static_cast<__nv_bfloat16*>(out);
  p.out_t = static_cast<int64_t>(num_q_heads) * HEAD_DIM;
  p.out_h = HEAD_DIM;
  p.cu_seqlens = cu_seqlens;
  p.gate = static_cast<const __nv_bfloat16*>(gate);
  p.gate_t = gate_stride_t;
  p.position_ids = position_ids;
  p.ids_are_int64 = ids_are_int64;
  p.inv_freq = inv_freq;
  const PrefillTensors t = {q, k_rot_scratch, v, q_stride_t, q_stride_h, static_cast<int64_t>(num_kv_heads) * HEAD_DIM, HEAD_DIM,
                            v_stride_t, v_stride_h, total_tokens, num_kv_heads};
  return launch_prefill_umma<true>(t, p, batch, max_seqlen, st, "fused_prefill_attention");
}
