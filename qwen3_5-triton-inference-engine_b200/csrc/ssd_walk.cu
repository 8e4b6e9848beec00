// State-space prefill (ssd.cu: the chunked form's mathematics; bf16, 64 < state rows <= 128, heads of at least 48 value columns)
// in two launches.  With L_t = log a_1 + .. + log a_t inside a 32-token chunk and E its last token
//     prep   P_ts = exp(L_t - L_s) dt_s (C_t . B_s) for s <= t,   exp(L_t),   exp(L_E - L_t) dt_t     all chunks at once
//     walk   y_t = exp(L_t) S_0^T C_t + sum P_ts x_s + D x_t,     S_E = exp(L_E) S_0 + sum_s B_s (exp(L_E - L_s) dt_s x_s)^T
// The prep takes C B^T once for all heads of a group and leaves P as product fragments (bf16 high and low parts).  In the walk
// a warp owns 16 value columns of S^T as accumulators and weights its own x in registers; two copy warps bring the chunks, and
// multiplying warps wait for nothing but the copies.
// One launch (ssd.cu) went through decays, scores, weights and products in turn, 4.7 us a chunk.  32 heads of 64 columns, one
// group, before -> now: 8 sequences of 256 to 1024 tokens 153 -> 84 us, 32 of 128 64 -> 57, one of 4096 100 -> 78 (in segments),
// one of 512 45 -> 29, 32 of 48 39 -> 35; heads of 128 columns, 8 groups, ragged 139 -> 88.  Sequences of one chunk stay there.
#include "linear_rnn.cuh"

namespace b200 {
namespace {

constexpr int SW_Q = 32;                          // tokens per chunk
constexpr int SW_N = 128;                         // state rows incl. padding
constexpr int SW_NP = SW_N + 8;                   // bf16 pitch of C and B rows: ldmatrix rows in different banks
constexpr int SW_BLOCKS = 3;                      // 16 x 16 blocks of a lower triangular 32 x 32 matrix: (0,0), (1,0), (1,1)
constexpr int SW_E = SW_BLOCKS * 1024, SW_SLOT = SW_E + 2 * SW_Q * 4;   // bytes: P | exp(L_t) | exp(L_E - L_t) dt_t
constexpr int SW_PREP_WARPS = 8;
constexpr int SW_WARPS = 4, SW_COPY = 64, SW_THREADS = 32 * SW_WARPS + SW_COPY, SW_COLS = 16 * SW_WARPS;
constexpr int SW_XP = SW_COLS + 8;
constexpr int SW_STAGES = 3;

__device__ __forceinline__ int64_t first_slot(const int32_t* cu, int b) { return cu[b] / SW_Q + b; }   // as in linear_rnn_walk.cu

__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16(a, b);
  lo = pack_bf16(a - bf16_lo(hi), b - bf16_hi(hi));
}
__device__ __forceinline__ void copy16(void* dst, const void* src, bool on) {   // zeros, and nothing read, when off
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(on ? 16 : 0) : "memory");
}

// grid (slots, groups * ceil(heads of a group / 8)): C B^T of a chunk on the tensor cores, then a head per warp: a lane per token for
// the decays, a fragment's elements for P.  A latency chain: with all heads of a group in one CTA it took twice as long.
__global__ void __launch_bounds__(32 * SW_PREP_WARPS) ssd_prep_kernel(const __grid_constant__ OuterRnnParams p, int batch) {
  __shared__ __align__(16) __nv_bfloat16 c[SW_Q * SW_NP], bm[SW_Q * SW_NP];
  __shared__ float G[SW_Q][SW_Q + 2], cum[SW_PREP_WARPS][SW_Q], step[SW_PREP_WARPS][SW_Q];
  pdl_trigger();                                  // the walk waits for this grid before it reads the slots
  const int slot = blockIdx.x, parts = (p.per_group + SW_PREP_WARPS - 1) / SW_PREP_WARPS, group = blockIdx.y / parts, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int b = -1;                                     // the last sequence whose slots start at or before this one
  for (int i0 = 0; i0 < batch; i0 += 32 * SW_PREP_WARPS) b += __syncthreads_count(i0 + tid < batch && first_slot(p.cu, i0 + tid) <= slot);
  if (b < 0) return;
  const int row0 = p.cu[b] + static_cast<int>(slot - first_slot(p.cu, b)) * SW_Q, rows = min(SW_Q, p.cu[b + 1] - row0);
  if (rows <= 0) return;
  const __nv_bfloat16* base = static_cast<const __nv_bfloat16*>(p.x) + static_cast<int64_t>(row0) * p.stride + group * p.dim;
  for (int i = tid; i < SW_Q * (SW_N / 8); i += 32 * SW_PREP_WARPS) {
    const int t = i / (SW_N / 8), k = (i % (SW_N / 8)) * 8;
    const bool on = t < rows && k < p.dim;
    const __nv_bfloat16* r = base + (on ? t * p.stride + k : 0);
    copy16(&c[t * SW_NP + k], r + p.q_off, on);
    copy16(&bm[t * SW_NP + k], r + p.k_off, on);
  }
  const int in_group = blockIdx.y % parts * SW_PREP_WARPS + warp, head = group * p.per_group + in_group;
  const bool mine = in_group < p.per_group;
  float dt_raw = 0.f, dt_bias = 0.f, rate = 0.f;
  if (mine) {
    dt_raw = load1(static_cast<const __nv_bfloat16*>(p.dt) + static_cast<int64_t>(row0 + min(lane, rows - 1)) * p.dt_stride + head);
    dt_bias = p.bias[head], rate = expf(p.a_log[head]);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const int gm = warp & 1, gn = warp >> 1;        // this warp's 16 x 8 tile of C B^T
  if (gn * 8 <= gm * 16 + 15) {
    float g[4] = {};
#pragma unroll
    for (int k2 = 0; k2 < SW_N / 32; ++k2) {
      uint32_t a0[4], a1[4], bk[4];
      const uint32_t at = smem_u32(&c[(gm * 16 + (lane & 15)) * SW_NP + k2 * 32 + (lane >> 4) * 8]);
      ldmatrix_x4(a0, at);
      ldmatrix_x4(a1, at + 32);
      ldmatrix_x4(bk, smem_u32(&bm[(gn * 8 + (lane & 7)) * SW_NP + k2 * 32 + (lane >> 3) * 8]));
      mma_bf16_16816(g, a0, bk[0], bk[1]);
      mma_bf16_16816(g, a1, bk[2], bk[3]);
    }
    const int t = gm * 16 + (lane >> 2), s = gn * 8 + (lane & 3) * 2;
    *reinterpret_cast<float2*>(&G[t][s]) = make_float2(g[0], g[1]);
    *reinterpret_cast<float2*>(&G[t + 8][s]) = make_float2(g[2], g[3]);
  }
  __syncthreads();
  if (!mine) return;
  const float dt = lane < rows ? softplus_f(dt_raw + dt_bias) : 0.f;
  float run = -rate * dt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float up = __shfl_up_sync(0xffffffffu, run, o);
    if (lane >= o) run += up;
  }
  const float total = __shfl_sync(0xffffffffu, run, 31);
  uint8_t* ws = static_cast<uint8_t*>(p.chunks) + (static_cast<int64_t>(slot) * p.heads + head) * SW_SLOT;
  float* scale = reinterpret_cast<float*>(ws + SW_E);
  scale[lane] = expf(run);
  scale[SW_Q + lane] = expf(total - run) * dt;
  __syncwarp();
  cum[warp][lane] = run, step[warp][lane] = dt;
  __syncwarp();
#pragma unroll
  for (int blk = 0; blk < SW_BLOCKS; ++blk) {
    const int m = blk > 0, ks = blk == 2;
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int t = m * 16 + (lane >> 2) + (j & 1) * 8, s = ks * 16 + (lane & 3) * 2 + (j >> 1) * 8;
      const float ct = cum[warp][t];
      const float p0 = s <= t ? G[t][s] * __expf(ct - cum[warp][s]) * step[warp][s] : 0.f;
      const float p1 = s + 1 <= t ? G[t][s + 1] * __expf(ct - cum[warp][s + 1]) * step[warp][s + 1] : 0.f;
      split_pair(p0, p1, hi[j], lo[j]);
    }
    *reinterpret_cast<uint4*>(ws + blk * 1024 + lane * 16) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(ws + blk * 1024 + 512 + lane * 16) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
}

template <bool V>
struct Flag {
  static constexpr bool value = V;
};

struct WalkSmem {
  __nv_bfloat16 c[SW_STAGES][SW_Q * SW_NP], b[SW_STAGES][SW_Q * SW_NP], x[SW_STAGES][SW_Q * SW_XP];
  uint8_t slot[SW_STAGES][SW_SLOT];
  uint64_t full[SW_STAGES], empty[SW_STAGES];
};

// One CTA = up to 64 value columns of one head of one sequence or segment: few columns per CTA, so that the tensor pipes of the
// card share a ragged batch's chunks evenly (two CTAs fit an SM).  LOCAL: only the state from zero and the total decay of
// every segment.  Bound by the tensor pipe: 140 products per warp and chunk, 1.2 us; a sequence's first chunk skips those with its
// zero state.  One copy warp instead of two was the bound of a chunk (88 us against 75 of the ragged batch's walk).  grid (vdim / 64, heads, sequences * segments)
template <bool LOCAL>
__global__ void __launch_bounds__(SW_THREADS, 2) ssd_walk_kernel(const __grid_constant__ OuterRnnParams p, int* err) {
  extern __shared__ __align__(128) uint8_t sw_smem[];
  WalkSmem& sm = *reinterpret_cast<WalkSmem*>(sw_smem);
  const int seq = blockIdx.z / p.segments, seg = blockIdx.z % p.segments, head = blockIdx.y, col0 = blockIdx.x * SW_COLS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int all = p.cu[seq + 1] - p.cu[seq], seg0 = seg * p.segment;
  const int row0 = p.cu[seq] + seg0, len = min(all - seg0, p.segment);
  if (len <= 0 || (LOCAL && seg0 + len == all)) {   // nothing follows a sequence's last segment
    pdl_wait();                                   // an idle CTA still orders the grid after the preparation
    return;
  }
  if (first_slot(p.cu, seq) + (all + SW_Q - 1) / SW_Q > p.chunk_slots) {   // more tokens than the call named: nobody prepared the end
    pdl_wait();
    if (tid == 0) atomicExch(err, 1);
    return;
  }
  const int chunks = (len + SW_Q - 1) / SW_Q, cols = min(SW_COLS, p.vdim - col0);
  const __nv_bfloat16* base = static_cast<const __nv_bfloat16*>(p.x) + static_cast<int64_t>(row0) * p.stride;
  if (tid == 0) {
#pragma unroll
    for (int s = 0; s < SW_STAGES; ++s) mbar_init(&sm.full[s], SW_COPY + 1), mbar_init(&sm.empty[s], SW_WARPS);
    mbar_fence_init();
  }
  __syncthreads();
  if (warp >= SW_WARPS) {
    // ------------------------------------------------------------------------------------------------------- copies
    const uint8_t* slots = static_cast<const uint8_t*>(p.chunks) + ((first_slot(p.cu, seq) + seg0 / SW_Q) * p.heads + head) * SW_SLOT;
    const int ct = tid - 32 * SW_WARPS, bc_col = (head / p.per_group) * p.dim, x_col = p.v_off + head * p.vdim + col0;
    int i = 0;
    for (; i < chunks; ++i) {
      const int st = i % SW_STAGES, t0 = i * SW_Q;
      if (i >= SW_STAGES && !warp_wait_bounded(&sm.empty[st], (i / SW_STAGES - 1) & 1)) break;
#pragma unroll 8
      for (int k = ct; k < SW_Q * (SW_N / 8); k += SW_COPY) {
        const int t = k / (SW_N / 8), d = (k % (SW_N / 8)) * 8;
        const bool on = t0 + t < len && d < p.dim;
        const __nv_bfloat16* r = base + (on ? (t0 + t) * p.stride + bc_col + d : 0);
        if (!LOCAL) copy16(&sm.c[st][t * SW_NP + d], r + (on ? p.q_off : 0), on);
        copy16(&sm.b[st][t * SW_NP + d], r + (on ? p.k_off : 0), on);
      }
#pragma unroll
      for (int k = ct; k < SW_Q * (SW_COLS / 8); k += SW_COPY) {
        const int t = k / (SW_COLS / 8), d = (k % (SW_COLS / 8)) * 8;
        const bool on = t0 + t < len && d < cols;
        copy16(&sm.x[st][t * SW_XP + d], base + (on ? (t0 + t) * p.stride + x_col + d : 0), on);
      }
      if (i == 0) pdl_wait();                     // the slots are complete
      if (ct == 0) {
        constexpr int skip = LOCAL ? SW_E : 0;
        mbar_expect_tx(&sm.full[st], SW_SLOT - skip);
        bulk_g2s(sm.slot[st] + skip, slots + static_cast<int64_t>(i) * p.heads * SW_SLOT + skip, SW_SLOT - skip, &sm.full[st]);
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&sm.full[st])) : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (i < chunks) {                             // the other warp runs out as well: no chunk is complete without this one's part
      atomicExch(err, 1);
      // bulk copies that nobody waits for any more may still be landing in this CTA's shared memory
      if (ct == 0)
        for (int k = max(i - SW_STAGES, 0); k < i; ++k) mbar_wait_bounded(&sm.full[k % SW_STAGES], k / SW_STAGES & 1, 1u << 12);
    }
    return;
  }
  // ---------------------------------------------------------------------------------------------------------- products
  const int wcol = warp * 16;
  const bool warp_on = wcol < cols;
  // S^T: value column lane / 4 (+ 8) of the warp, state rows 8 n + (lane % 4) * 2 (+ 1)
  float S[SW_N / 8][4];
  const int64_t head_elems = static_cast<int64_t>(p.dim) * p.vdim;
  float* slot_state = p.state + (static_cast<int64_t>(p.slots[seq]) * p.heads + head) * head_elems;
  float* seg_state = p.seg_state + (static_cast<int64_t>(blockIdx.z) * p.heads + head) * head_elems;
  const float* from = p.segments > 1 ? seg_state : slot_state;
  const bool carry = !LOCAL && warp_on && (p.segments > 1 || p.start[seq] > 0);
  const int my_col = col0 + wcol + (lane >> 2);
#pragma unroll
  for (int n = 0; n < SW_N / 8; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int d = n * 8 + (lane & 3) * 2 + (j & 1), c = my_col + (j >> 1) * 8;
      S[n][j] = carry && d < p.dim ? from[static_cast<int64_t>(d) * p.vdim + c] : 0.f;
    }
  const float skip = LOCAL ? 0.f : p.skip[head];
  float total = 1.f;
  pdl_wait();                                     // before the first store
#pragma unroll 1
  for (int i = 0; i < chunks; ++i) {
    const int st = i % SW_STAGES;
    if (!warp_wait_bounded(&sm.full[st], (i / SW_STAGES) & 1)) {
      atomicExch(err, 1);
      return;
    }
    const float* scale = reinterpret_cast<const float*>(sm.slot[st] + SW_E);
    const float keep = scale[SW_Q - 1];
    total *= keep;
    if (warp_on) {
      float o[2][2][4] = {}, y[2][2][4] = {};     // (C S)^T and the rest, 16-token halves x 8-column halves
      uint32_t xh[2][4], xl[2][4];                // weighted x, as a left operand: columns x tokens
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) {
        // matrices (tokens 0-7, columns 0-7), (0-7, 8-15), (8-15, 0-7), (8-15, 8-15)
        uint32_t vm[4];
        ldmatrix_x4_trans(vm, smem_u32(&sm.x[st][(ks * 16 + (lane & 7) + (lane >> 4) * 8) * SW_XP + wcol + ((lane >> 3) & 1) * 8]));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 w = *reinterpret_cast<const float2*>(scale + SW_Q + ks * 16 + (j >> 1) * 8 + (lane & 3) * 2);
          split_pair(bf16_lo(vm[j]) * w.x, bf16_hi(vm[j]) * w.y, xh[ks][j], xl[ks][j]);
        }
        if (!LOCAL) {
#pragma unroll
          for (int m = ks; m < 2; ++m) {
            const uint8_t* f = sm.slot[st] + (m + ks) * 1024 + lane * 16;
            const uint4 h4 = *reinterpret_cast<const uint4*>(f), l4 = *reinterpret_cast<const uint4*>(f + 512);
            const uint32_t h[4] = {h4.x, h4.y, h4.z, h4.w}, l[4] = {l4.x, l4.y, l4.z, l4.w};
            mma_bf16_16816(y[m][0], h, vm[0], vm[2]);
            mma_bf16_16816(y[m][1], h, vm[1], vm[3]);
            mma_bf16_16816(y[m][0], l, vm[0], vm[2]);
            mma_bf16_16816(y[m][1], l, vm[1], vm[3]);
          }
        }
      }
      const uint32_t a_at = smem_u32(&sm.c[st][(lane & 15) * SW_NP + (lane >> 4) * 8]);
      const uint32_t b_at = smem_u32(&sm.b[st][(lane & 15) * SW_NP + (lane >> 4) * 8]);
      auto products = [&](auto enters) {          // whether a state enters the chunk
#pragma unroll
        for (int ks = 0; ks < SW_N / 16; ++ks) {
          float(&s0)[4] = S[2 * ks];
          float(&s1)[4] = S[2 * ks + 1];
          uint32_t bt[2][4];
          ldmatrix_x4_trans(bt[0], b_at + ks * 32);
          ldmatrix_x4_trans(bt[1], b_at + ks * 32 + 16 * SW_NP * 2);
          if (enters.value) {
            uint32_t a0[4], a1[4], h[2][2], l[2][2];
            ldmatrix_x4(a0, a_at + ks * 32);
            ldmatrix_x4(a1, a_at + ks * 32 + 16 * SW_NP * 2);
#pragma unroll
            for (int n = 0; n < 2; ++n) {
              split_pair(s0[2 * n], s0[2 * n + 1], h[n][0], l[n][0]);
              split_pair(s1[2 * n], s1[2 * n + 1], h[n][1], l[n][1]);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) s0[j] *= keep, s1[j] *= keep;
            mma_bf16_16816(o[0][0], a0, h[0][0], h[0][1]);
            mma_bf16_16816(o[0][1], a0, h[1][0], h[1][1]);
            mma_bf16_16816(s0, xh[0], bt[0][0], bt[0][1]);
            mma_bf16_16816(s1, xh[0], bt[0][2], bt[0][3]);
            mma_bf16_16816(o[1][0], a1, h[0][0], h[0][1]);
            mma_bf16_16816(o[1][1], a1, h[1][0], h[1][1]);
            mma_bf16_16816(s0, xl[0], bt[0][0], bt[0][1]);
            mma_bf16_16816(s1, xl[0], bt[0][2], bt[0][3]);
            mma_bf16_16816(o[0][0], a0, l[0][0], l[0][1]);
            mma_bf16_16816(o[0][1], a0, l[1][0], l[1][1]);
            mma_bf16_16816(s0, xh[1], bt[1][0], bt[1][1]);
            mma_bf16_16816(s1, xh[1], bt[1][2], bt[1][3]);
            mma_bf16_16816(o[1][0], a1, l[0][0], l[0][1]);
            mma_bf16_16816(o[1][1], a1, l[1][0], l[1][1]);
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) s0[j] *= keep, s1[j] *= keep;
            mma_bf16_16816(s0, xh[0], bt[0][0], bt[0][1]);
            mma_bf16_16816(s1, xh[0], bt[0][2], bt[0][3]);
            mma_bf16_16816(s0, xl[0], bt[0][0], bt[0][1]);
            mma_bf16_16816(s1, xl[0], bt[0][2], bt[0][3]);
            mma_bf16_16816(s0, xh[1], bt[1][0], bt[1][1]);
            mma_bf16_16816(s1, xh[1], bt[1][2], bt[1][3]);
          }
          mma_bf16_16816(s0, xl[1], bt[1][0], bt[1][1]);
          mma_bf16_16816(s1, xl[1], bt[1][2], bt[1][3]);
        }
      };
      if (!LOCAL && (carry || i > 0)) products(Flag<true>());
      else products(Flag<false>());
      if (!LOCAL) {
        __nv_bfloat16* out = static_cast<__nv_bfloat16*>(p.out) + static_cast<int64_t>(row0 + i * SW_Q) * p.out_stride + head * p.vdim + col0 + wcol + (lane & 3) * 2;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const int t = m * 16 + (lane >> 2) + half * 8;
            const float e = scale[t];
            if (i * SW_Q + t >= len) continue;
#pragma unroll
            for (int n = 0; n < 2; ++n) {
              const uint32_t x = *reinterpret_cast<const uint32_t*>(&sm.x[st][t * SW_XP + wcol + n * 8 + (lane & 3) * 2]);
              const float r0 = fmaf(o[m][n][2 * half], e, y[m][n][2 * half]), r1 = fmaf(o[m][n][2 * half + 1], e, y[m][n][2 * half + 1]);
              *reinterpret_cast<uint32_t*>(out + t * p.out_stride + n * 8) = pack_bf16(fmaf(skip, bf16_lo(x), r0), fmaf(skip, bf16_hi(x), r1));
            }
          }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.empty[st]);
  }
  if (LOCAL && blockIdx.x == 0)
    for (int d = tid; d < p.dim; d += 32 * SW_WARPS) p.seg_decay[(static_cast<int64_t>(blockIdx.z) * p.heads + head) * p.dim + d] = total;
  if ((!LOCAL && seg0 + len < all) || !warp_on) return;   // only the last segment leaves the sequence's state behind
  float* to = LOCAL ? seg_state : slot_state;
#pragma unroll
  for (int n = 0; n < SW_N / 8; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int d = n * 8 + (lane & 3) * 2 + (j & 1), c = my_col + (j >> 1) * 8;
      if (d < p.dim) to[static_cast<int64_t>(d) * p.vdim + c] = S[n][j];
    }
}

int64_t slots_of(int64_t tokens, int64_t batch) { return tokens / SW_Q + batch; }

template <bool LOCAL>
int launch_pass(const OuterRnnParams& p, dim3 grid, bool early, int* err, cudaStream_t st) {
  constexpr int smem = sizeof(WalkSmem);
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    if (cudaFuncSetAttribute(ssd_walk_kernel<LOCAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
      return fail(ERR_RUNTIME, "ssd_prefill: cannot raise dynamic shared memory to %d", smem);
    configured[dev] = true;
  }
  if (launch_pdl(early, ssd_walk_kernel<LOCAL>, grid, dim3(SW_THREADS), smem, st, p, err) != cudaSuccess)
    return fail(ERR_LAUNCH, "ssd_prefill: %s", cudaGetErrorString(cudaGetLastError()));
  return OK;
}

bool shape_walks(int dim, int vdim) { return dim > 64 && dim <= SW_N && dim % 8 == 0 && vdim % 16 == 0 && (vdim + SW_COLS - 1) / SW_COLS * SW_COLS - vdim <= 16; }

}  // namespace

bool ssd_walk_supports(const OuterRnnParams& p) { return p.chunks && shape_walks(p.dim, p.vdim); }

int ssd_walk_launch(OuterRnnParams p, int n, int tokens, cudaStream_t st) {
  int* err = wait_timeout_flag();
  if (!err) return fail(ERR_RUNTIME, "ssd_prefill: no error flag");
  const int groups = p.heads / p.per_group * ((p.per_group + SW_PREP_WARPS - 1) / SW_PREP_WARPS);   // at most heads
  p.chunk_slots = static_cast<int>(slots_of(tokens, n));
  ssd_prep_kernel<<<dim3(static_cast<unsigned>(p.chunk_slots), groups), 32 * SW_PREP_WARPS, 0, st>>>(p, n);
  const dim3 grid((p.vdim + SW_COLS - 1) / SW_COLS, p.heads, n * p.segments);
  if (p.segments > 1) {
    const int rc = launch_pass<true>(p, grid, true, err, st);
    if (rc != OK) return rc;
    outer_rnn_fold_launch(p, n, st);
  }
  const int rc = launch_pass<false>(p, grid, p.segments == 1, err, st);
  return rc != OK ? rc : check_launch("ssd_prefill (walk)");
}

}  // namespace b200

using namespace b200;

extern "C" int64_t b200_ssd_walk_workspace_bytes(int32_t tokens, int32_t batch, int32_t heads, int32_t dim, int32_t vdim) {
  if (tokens <= 0 || batch <= 0 || !shape_walks(dim, vdim)) return 0;
  const int64_t bytes = slots_of(tokens, batch) * heads * SW_SLOT;
  return bytes <= (int64_t{1} << 30) ? bytes : 0;
}
