// Prefill attention (see prefill_umma.cu) of calls that one wave of CTAs takes, and of prompts no longer than one of its blocks: a CTA to
// every (sequence, kv head, block of 32 query tokens), with no partner, no list of items and no ring of them in front of its first load.  The 4 Q
// heads of the group are stacked into the 128 rows of one MMA tile (row = token*4 + head), so every K/V tile is fetched once per group.
// Per 128-token KV tile:
//     S[128 x 128]  = Q[128 x 256] . K^T          tcgen05.mma, both operands K-major in shared memory, D in TMEM
//     P = exp2(S*scale*log2e - m)                  two softmax threads per row (64 columns each), TMEM -> TMEM
//     O[128 x 256] += P[128 x 128] . V[128 x 256]  tcgen05.mma, P from TMEM, V as an MN-major operand, O stays in TMEM
// Roles: warps 0-7 softmax/epilogue (TMEM lane quarter = warp % 4, column half = warp / 4), warp 8 issues the MMAs (the whole warp walks
// the loop, lane 0 issues), warps 9 and 10 issue the K and V TMA loads (64 KiB per tile, 128-byte swizzle, no multicast; K of tile j+1 is
// requested the moment S of tile j is done).  S is double-buffered in TMEM (2 x 128 columns + 256 for O = all 512), P is stored as packed
// bf16 over the first 64 columns of the S buffer just read.  O is rescaled in TMEM only when a row maximum grows by more than 2^8.
// Bound: a chain of latencies (launch, loads, S, exponentials, PV, stores); times beside the rule in prefill_takes_short.
// Every mbarrier wait is bounded; on expiry the role sets the device error flag and the CTA drains and exits.
#include "prefill.cuh"

namespace b200 {

constexpr int PS_SOFTMAX_THREADS = 256;
constexpr int PS_THREADS = 352;                     // 8 softmax warps + MMA issuer + K producer + V producer
constexpr int PS_Q_BYTES = 128 * HEAD_DIM * 2;      // 64 KiB: 4 column blocks of [128 rows][64]
constexpr int PS_KV_BYTES = PU_TKV * HEAD_DIM * 2;  // 64 KiB: 4 column blocks of [128 rows][64]
constexpr int PS_SMEM = PS_Q_BYTES + 2 * PS_KV_BYTES;  // 192 KiB; tiles need 1024-byte alignment: the kernel checks
constexpr int PS_OUT_PITCH = HEAD_DIM * 2 + 16;     // pitch of gates and output (bytes)
static_assert(128 * PS_OUT_PITCH <= PS_Q_BYTES + PS_KV_BYTES, "gates and output must fit in the Q + K region");

template <bool FUSED>
__global__ void __launch_bounds__(PS_THREADS, 1)
prefill_short_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                     const __grid_constant__ CUtensorMap map_v, const __grid_constant__ PrefillUmmaParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ uint64_t bar_q, bar_qr, bar_k, bar_v, bar_s[2], bar_p[2], bar_pv, bar_o;  // bar_pv: PV of every tile but the last, whose is bar_o
  __shared__ uint32_t tmem_slot;
  __shared__ float xm[2][2][128];  // [tile parity][column half][row]: row maxima (at the end: row sums) exchanged
                                   // between the two threads of a row

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // the whole batch's last (heaviest) query blocks first, then the ones before them, ...
  const int qb = gridDim.y - 1 - blockIdx.y, h = blockIdx.x % p.num_kv_heads, b = blockIdx.x / p.num_kv_heads;
  const int seq_start = p.cu_seqlens[b];
  const int seq_len = p.cu_seqlens[b + 1] - seq_start;
  const int q0 = qb * PU_BQ;
  if (q0 >= seq_len) {
    if (FUSED) pdl_wait();  // every CTA orders the grid after the kernel in front of it
    return;
  }
  const int kv_end = min(q0 + PU_BQ, seq_len);
  const int n_tiles = (kv_end + PU_TKV - 1) / PU_TKV;

  uint8_t* smem = smem_raw;
  if ((smem_u32(smem) & 1023u) != 0) {  // swizzled tiles need 1024-byte alignment; never taken with __align__(1024)
    if (tid == 0) atomicExch(p.err, 1);
    return;
  }
  uint8_t* q_s = smem;
  uint8_t* k_s = smem + PS_Q_BYTES;
  uint8_t* v_s = k_s + PS_KV_BYTES;

  if (warp == 0) tmem_alloc(&tmem_slot, PU_TMEM_COLS);
  // The loads that wait for nobody leave before the CTA has met: Q and the first V tile (and, where no kernel in front writes
  // it, the first K tile) travel while tensor memory is allocated and the other barriers are set up.
  if (tid == 9 * 32) {
    mbar_init(&bar_q, 1);
    mbar_init(&bar_k, 1);
    mbar_init(&bar_v, 1);
    mbar_fence_init();
    mbar_expect_tx(&bar_q, PS_Q_BYTES);
    tma_load_5d(q_s, &map_q, 0, 0, h, seq_start + q0, 0, &bar_q);
    if (!FUSED) {
      mbar_expect_tx(&bar_k, PS_KV_BYTES);
      tma_load_4d(k_s, &map_k, 0, seq_start, 0, h, &bar_k);
    }
    mbar_expect_tx(&bar_v, PS_KV_BYTES);
    tma_load_4d(v_s, &map_v, 0, seq_start, 0, h, &bar_v);
  }
  // the gate rows are the epilogue's: asked into the L2 now, 128 rows of four lines
  if (FUSED && tid < PS_SOFTMAX_THREADS) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int line = tid + i * PS_SOFTMAX_THREADS, r = line >> 2, tok = q0 + (r >> 2);
      if (tok < seq_len)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p.gate + static_cast<int64_t>(seq_start + tok) * p.gate_t + (h * GROUP + (r & 3)) * HEAD_DIM + (line & 3) * 64));
    }
  }
  if (tid == 0) {
    mbar_init(&bar_qr, 128);
    mbar_init(&bar_s[0], 1);
    mbar_init(&bar_s[1], 1);
    mbar_init(&bar_p[0], PS_SOFTMAX_THREADS);  // one per S/P buffer: a warp may be a tile ahead of another
    mbar_init(&bar_p[1], PS_SOFTMAX_THREADS);
    mbar_init(&bar_pv, 1);
    mbar_init(&bar_o, 1);
    mbar_fence_init();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;
  const uint32_t tmem_o = tmem + 2 * PU_TKV;

  if (warp == 9) {
    // ------------------------------------------------------------------ TMA producer: the K tiles
    if (lane == 0) {
      bool ok = true;
      // fused form: started while the rope + scatter kernel still runs (programmatic dependent launch).  Everything up
      // to here - tensor-memory allocation, barriers, the Q tile, and the V tiles of the other producer - overlaps with
      // it; the rotated K it writes is read only after it has completed.
      if (FUSED) pdl_wait();
      for (int j = FUSED ? 0 : 1; j < n_tiles && ok; ++j) {
        if (j >= 1) ok = mbar_wait_bounded(&bar_s[(j - 1) & 1], ((j - 1) >> 1) & 1);  // S of tile j-1 done: K free
        if (!ok) break;
        mbar_expect_tx(&bar_k, PS_KV_BYTES);
        tma_load_4d(k_s, &map_k, 0, seq_start + j * PU_TKV, 0, h, &bar_k);
      }
      if (!ok) atomicExch(p.err, 1);
    }
  } else if (warp == 10) {
    // ------------------------------------------------------------------ TMA producer: the V tiles
    if (lane == 0) {
      bool ok = true;
      for (int j = 1; j < n_tiles && ok; ++j) {
        ok = mbar_wait_bounded(&bar_pv, (j - 1) & 1);  // PV of tile j-1 done: V free
        if (!ok) break;
        mbar_expect_tx(&bar_v, PS_KV_BYTES);
        tma_load_4d(v_s, &map_v, 0, seq_start + j * PU_TKV, 0, h, &bar_v);
      }
      if (!ok) atomicExch(p.err, 1);
    }
  } else if (warp == 8) {
    // ------------------------------------------------------------------ MMA issuer
    {
      // the whole warp walks the loop (uniform control flow), lane 0 issues
      const bool leader = lane == 0;
      const uint32_t idesc_s = idesc_bf16_f32(128, PU_TKV, false, false);
      const uint32_t idesc_o = idesc_bf16_f32(128, HEAD_DIM, false, true);
      const uint32_t q_addr = smem_u32(q_s), k_addr = smem_u32(k_s), v_addr = smem_u32(v_s);
      bool ok = FUSED ? mbar_wait_bounded(&bar_qr, 0) : mbar_wait_bounded(&bar_q, 0);
      auto issue_pv = [&](int jj) {
        ok = ok && mbar_wait_bounded(&bar_p[jj & 1], (jj >> 1) & 1);
        ok = ok && mbar_wait_bounded(&bar_v, jj & 1);
        if (!ok) return;
        tc_fence_after_sync();
#pragma unroll
        for (int kt = 0; kt < PU_TKV / 16; ++kt)
          umma_ts_leader(tmem_o, tmem + (jj & 1) * PU_TKV + kt * 8,  // P: 16 tokens = 8 packed columns per step
                         smem_desc_sw128(v_addr + kt * 2048, PU_TKV * 128, 1024), idesc_o, (jj > 0) || (kt > 0), leader);
        umma_commit_leader(jj + 1 < n_tiles ? &bar_pv : &bar_o, leader);
      };
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int s = j & 1;
        ok = mbar_wait_bounded(&bar_k, j & 1);
        // S(j) overwrites the buffer whose first columns hold P(j-2): the PV product that reads them from tensor
        // memory must have COMPLETED, issue order alone does not protect an operand in tensor memory
        if (ok && j >= 2) ok = mbar_wait_bounded(&bar_pv, (j - 2) & 1);
        if (!ok) break;
        tc_fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < HEAD_DIM / 16; ++ks) {
          const uint32_t o = (ks >> 2) * (128 * 128) + (ks & 3) * 32;
          umma_ss_leader(tmem + s * PU_TKV, smem_desc_sw128(q_addr + o, 16, 1024), smem_desc_sw128(k_addr + o, 16, 1024),
                         idesc_s, ks > 0, leader);
        }
        umma_commit_leader(&bar_s[s], leader);
        if (j >= 1) issue_pv(j - 1);
      }
      if (ok) issue_pv(n_tiles - 1);
      if (!ok && leader) atomicExch(p.err, 1);
    }
  } else {
    // ------------------------------------------------------------------ softmax + epilogue
    const int row = 32 * (warp & 3) + lane;    // TMEM lane; row = token*4 + head
    const int half = warp >> 2;                // this thread's 64 of the tile's 128 columns
    const int q_tok = q0 + (row >> 2);
    const uint32_t lane_base = static_cast<uint32_t>(32 * (warp & 3)) << 16;
    const int pair_bar = 1 + (warp & 3);       // named barrier of the two warps that share these rows
    float m_ref = -INFINITY, l_run = 0.f;
    bool ok = true;
    if (FUSED && half == 0) {
      // rotary embedding of this row's q in place (dims [0,32) and [32,64) live in column block 0, chunks c, c+4)
      const int64_t t = seq_start + min(q_tok, seq_len - 1);
      const int64_t pid = p.ids_are_int64 ? static_cast<const int64_t*>(p.position_ids)[t]
                                          : static_cast<int64_t>(static_cast<const int32_t*>(p.position_ids)[t]);
      const float posf = static_cast<float>(pid);
      // the four rows of a token share their angles: each lane of a quad computes 8 of the 32 (sin, cos) pairs
      float sn[8], cs[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) sincosf(posf * p.inv_freq[(lane & 3) * 8 + i], &sn[i], &cs[i]);
      ok = warp_wait_bounded(&bar_q, 0);
      uint8_t* qrow = q_s + row * 128;
#pragma unroll
      for (int c = 0; c < 4; ++c) {  // chunk c holds dims [8c, 8c+8), chunk c+4 their partners [32+8c, 40+8c)
        uint4* pa = reinterpret_cast<uint4*>(qrow + ((c ^ (row & 7)) << 4));
        uint4* pb = reinterpret_cast<uint4*>(qrow + (((c + 4) ^ (row & 7)) << 4));
        const uint4 va = *pa, vb = *pb;
        uint32_t wa[4] = {va.x, va.y, va.z, va.w}, wb[4] = {vb.x, vb.y, vb.z, vb.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          // angle index 8c + 2k (+1) lives in lane (quad base + c), register 2k (+1)
          const int src = (lane & ~3) + c;
          const float c0 = __shfl_sync(0xffffffffu, cs[2 * k], src), s0 = __shfl_sync(0xffffffffu, sn[2 * k], src);
          const float c1 = __shfl_sync(0xffffffffu, cs[2 * k + 1], src), s1 = __shfl_sync(0xffffffffu, sn[2 * k + 1], src);
          float f0, g0, f1, g1;
          rope_pair(bf16_lo(wa[k]), bf16_lo(wb[k]), s0, c0, f0, g0);
          rope_pair(bf16_hi(wa[k]), bf16_hi(wb[k]), s1, c1, f1, g1);
          wa[k] = pack_bf16(f0, f1);
          wb[k] = pack_bf16(g0, g1);
        }
        *pa = make_uint4(wa[0], wa[1], wa[2], wa[3]);
        *pb = make_uint4(wb[0], wb[1], wb[2], wb[3]);
      }
      fence_proxy_async();  // the rotated rows must be visible to the tensor core's reads
      mbar_arrive(&bar_qr);
    }
    // A failed (timed-out) wait clears `ok`; the loop then keeps only its barriers and arrivals, so that the partner
    // warp and the MMA issuer are never left waiting for this thread.
    for (int j = 0; j < n_tiles; ++j) {
      const int s = j & 1;
      ok = warp_wait_bounded(&bar_s[s], (j >> 1) & 1, ok);
      uint32_t r0[32], r1[32];
      float m_half = 0.f;
      if (ok) {
        tc_fence_after_sync();
        tmem_ld32(tmem + lane_base + s * PU_TKV + half * 64, r0);
        tmem_ld32(tmem + lane_base + s * PU_TKV + half * 64 + 32, r1);
        tmem_ld_wait();
        // mask (causal and inside the sequence; only tiles on the diagonal or at the sequence end need it) and take
        // the row maximum of the raw scores; the scale (> 0) is folded into the exponent below
        const int lim = min(q_tok, seq_len - 1) - j * PU_TKV - half * 64;  // last valid column of this half
        if (lim < 63) {
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            if (c > lim) r0[c] = 0xff800000u;       // -inf
            if (c + 32 > lim) r1[c] = 0xff800000u;
          }
        }
        float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
        for (int c = 0; c < 32; c += 2) {
          mx0 = fmaxf(mx0, __uint_as_float(r0[c]));
          mx1 = fmaxf(mx1, __uint_as_float(r0[c + 1]));
          mx2 = fmaxf(mx2, __uint_as_float(r1[c]));
          mx3 = fmaxf(mx3, __uint_as_float(r1[c + 1]));
        }
        m_half = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
      }
      xm[s][half][row] = m_half;
      named_barrier(pair_bar, 64);
      // after this barrier both threads of the row hold their scores in registers: the S buffer may take P
      if (ok) {
        const float m_tile = fmaxf(m_half, xm[s][half ^ 1][row]) * p.scale_log2;
        const float m_new = fmaxf(m_ref, m_tile);  // both threads of a row compute the same value
        if (j == 0) {
          m_ref = m_new;
        } else {
          const bool need = (m_new - m_ref) > PU_TAU;
          if (__any_sync(0xffffffffu, need)) {
            // O must be at rest before it is rescaled: wait for the PV product of tile j-1
            ok = warp_wait_bounded(&bar_pv, (j - 1) & 1);
            tc_fence_after_sync();
            const float alpha = need ? ex2_fast(m_ref - m_new) : 1.f;
#pragma unroll 1
            for (int c0 = 0; c0 < HEAD_DIM / 2; c0 += 32) {  // this thread's 128 columns of O
              uint32_t o[32];
              tmem_ld32(tmem_o + lane_base + half * (HEAD_DIM / 2) + c0, o);
              tmem_ld_wait();
#pragma unroll
              for (int c = 0; c < 32; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * alpha);
              tmem_st32(tmem_o + lane_base + half * (HEAD_DIM / 2) + c0, o);
            }
            tmem_st_wait();
            l_run *= alpha;
            if (need) m_ref = m_new;
          }
        }
        // p = 2^(s*scale - m_ref): fp32 for l, bf16 for the PV product, stored as this thread's 32 packed columns of
        // the P tile (tokens 2c, 2c+1 in column c) over the S buffer
        float sum0 = 0.f, sum1 = 0.f;
        const float neg_m = -m_ref, sc = p.scale_log2;
        uint32_t w[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          const float x0 = ex2_fast(fmaf(__uint_as_float(c < 16 ? r0[2 * c] : r1[2 * c - 32]), sc, neg_m));
          const float x1 = ex2_fast(fmaf(__uint_as_float(c < 16 ? r0[2 * c + 1] : r1[2 * c - 31]), sc, neg_m));
          sum0 += x0;
          sum1 += x1;
          w[c] = pack_bf16(x0, x1);
        }
        l_run += sum0 + sum1;
        tmem_st32(tmem + lane_base + s * PU_TKV + half * 32, w);
        tmem_st_wait();
      }
      tc_fence_before_sync();   // this thread's TMEM loads/stores before the arrive
      mbar_arrive(&bar_p[s]);
    }
    // ---- epilogue: O / l, gated, -> bf16 -> staged in shared memory (Q and K are dead) -> coalesced global stores.  The gates come to the
    // places of the output while the last PV product runs.
    uint8_t* orow = smem + row * PS_OUT_PITCH + half * HEAD_DIM;  // this half's 128 columns = 256 bytes
    if (FUSED && ok) {
#pragma unroll 4
      for (int i = tid; i < 128 * (HEAD_DIM / 8); i += PS_SOFTMAX_THREADS) {  // a warp brings one row of 512 bytes per step
        const int r = i >> 5, ch = i & 31, tok = q0 + (r >> 2);
        if (tok >= seq_len) break;                                  // rows behind the sequence are not written
        cp_async16(smem + r * PS_OUT_PITCH + ch * 16,
                   p.gate + static_cast<int64_t>(seq_start + tok) * p.gate_t + (h * GROUP + (r & 3)) * HEAD_DIM + ch * 8);
      }
    }
    // (a barrier of its own: by the parity of bar_pv the PV products of the last tile and of the third last look alike)
    ok = warp_wait_bounded(&bar_o, 0, ok);
    float* xl = &xm[n_tiles & 1][0][0];  // the parity slot the last tile did not use
    xl[half * 128 + row] = l_run;
    if (FUSED) {
      cp_async_wait_all();
      named_barrier(9, PS_SOFTMAX_THREADS);  // the eight softmax warps only
    } else {
      named_barrier(pair_bar, 64);
    }
    if (ok) {
      tc_fence_after_sync();
      const float inv_l = 1.f / (l_run + xl[(half ^ 1) * 128 + row]);
      // o sigmoid(g) = o/2 tanh(g/2) + o/2
      const uint64_t inv2 = FUSED ? f32x2(0.5f * inv_l, 0.5f * inv_l) : f32x2(inv_l, inv_l);
      const __nv_bfloat162 one_half = __floats2bfloat162_rn(0.5f, 0.5f);
#pragma unroll 1
      for (int c0 = 0; c0 < HEAD_DIM / 2; c0 += 64) {
        uint32_t o[2][32];                         // two loads in flight
        tmem_ld32(tmem_o + lane_base + half * (HEAD_DIM / 2) + c0, o[0]);
        tmem_ld32(tmem_o + lane_base + half * (HEAD_DIM / 2) + c0 + 32, o[1]);
        tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          const uint32_t(&v)[32] = o[g >> 2];
          uint4* at = reinterpret_cast<uint4*>(orow + (c0 + g * 8) * 2);
          uint32_t gs[4] = {}, w[4];
          if (FUSED) {
            const uint4 gv = *at;
            gs[0] = gv.x; gs[1] = gv.y; gs[2] = gv.z; gs[3] = gv.w;
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            uint64_t x = f32x2_mul(f32x2(v[(g & 3) * 8 + k * 2], v[(g & 3) * 8 + k * 2 + 1]), inv2);
            if (FUSED) {
              const __nv_bfloat162 h2 = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&gs[k]), one_half);
              const uint32_t hw = *reinterpret_cast<const uint32_t*>(&h2);
              x = f32x2_fma(x, f32x2(tanh_fast(bf16_lo(hw)), tanh_fast(bf16_hi(hw))), x);
            }
            w[k] = pack_bf16x2(x);
          }
          *at = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    } else {
      atomicExch(p.err, 1);
    }
    named_barrier(9, PS_SOFTMAX_THREADS);
    if (ok) {
#pragma unroll 4
      for (int i = tid; i < 128 * (HEAD_DIM / 8); i += PS_SOFTMAX_THREADS) {
        const int r = i >> 5, ch = i & 31, tok = q0 + (r >> 2);
        if (tok < seq_len)
          *reinterpret_cast<uint4*>(p.out + static_cast<int64_t>(seq_start + tok) * p.out_t + (h * GROUP + (r & 3)) * p.out_h + ch * 8) =
              *reinterpret_cast<const uint4*>(smem + r * PS_OUT_PITCH + ch * 16);
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, PU_TMEM_COLS);
}

}  // namespace b200

using namespace b200;

// One wave of CTAs: at most as many as SMs, by the longest length, or by the tokens and half a block of padding per sequence where that bounds
// the empty ones by another wave.  A little more than a wave where up to four (sequence, head) have a chain of tiles each that sets the time
// anyway.  And prompts of one block, of which a pair would compute one and a padded one (without rope and gate up to 256 of them: beyond, the
// pairs' copies out are worth more).  us with rope and gate / without, here and on the pairs: 1 x 2048 tokens 36.8 / 31.1 and 40.1 / 32.5, 8 x 256
// 15.9 / 10.1 and 18.3 / 11.3, 32 x 64 14.9 / 8.5 and 17.3 / 10.5, 32 of 1 to 128 16.5 / 9.5 and 23.7 / 14.2, 2 x 1500 31.8 / 25.8 and 34.8 / 28.0,
// 256 x 32 53.3 / 33.1 and 62.7 / 33.4; on the other side of the lines 8 x 300 24.1 / 15.1 and 23.7 / 14.3, 64 x 64 25.6 / 15.8 and 25.5 / 14.4,
// 4 x 700 26.4 / 17.1 and 25.4 / 18.0, 512 x 32 without 60.3 and 58.0.
bool b200::prefill_takes_short(bool fused, int batch, int total_tokens, int max_seqlen, int num_kv_heads) {
  const int64_t sms = sm_count(), segments = static_cast<int64_t>(batch) * num_kv_heads;
  if (max_seqlen <= PU_BQ) return fused || max_seqlen <= PU_BQ / 2 || segments <= 512;
  const int64_t ctas = segments * ((max_seqlen + PU_BQ - 1) / PU_BQ);
  if (ctas <= sms) return true;
  if (segments <= 4) return ctas * 4 <= sms * (fused ? 5 : 7);
  return ctas <= 2 * sms && (static_cast<int64_t>(total_tokens) + static_cast<int64_t>(batch) * (PU_BQ / 2)) * num_kv_heads <= sms * PU_BQ;
}

template <bool FUSED>
static int launch_short(const PrefillTensors& t, PrefillUmmaParams p, cudaStream_t stream, const char* what) {
  CUtensorMap map_q, map_k, map_v;
  if (!encode_prefill_q(&map_q, t) || !encode_prefill_kv(&map_k, t, t.k, t.k_t, t.k_h, PU_TKV, HEAD_DIM / 64) ||
      !encode_prefill_kv(&map_v, t, t.v, t.v_t, t.v_h, PU_TKV, HEAD_DIM / 64))
    return fail(ERR_RUNTIME, "%s: cannot encode the tensor maps of q / k / v", what);
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    if (cudaFuncSetAttribute(prefill_short_kernel<FUSED>, cudaFuncAttributeMaxDynamicSharedMemorySize, PS_SMEM) != cudaSuccess)
      return fail(ERR_RUNTIME, "%s: cannot raise dynamic shared memory to %d", what, PS_SMEM);
    configured[dev] = true;
  }
  const dim3 grid(static_cast<unsigned>(p.num_kv_heads) * p.batch, (p.max_seqlen + PU_BQ - 1) / PU_BQ);
  // the fused form starts behind its own rope + scatter kernel while that one still runs (see the K producer)
  if (launch_pdl(FUSED, prefill_short_kernel<FUSED>, grid, dim3(PS_THREADS), PS_SMEM, stream, map_q, map_k, map_v, p) != cudaSuccess)
    return fail(ERR_LAUNCH, "%s: %s", what, cudaGetErrorString(cudaGetLastError()));
  return check_launch(what);
}

int b200::launch_prefill_short(bool fused, const PrefillTensors& t, const PrefillUmmaParams& p, cudaStream_t stream, const char* what) {
  return fused ? launch_short<true>(t, p, stream, what) : launch_short<false>(t, p, stream, what);
}
