// Prefill of the outer-product recurrences with a decay per key channel (linear_rnn.cuh, FORGET and KEYED; bf16 activations,
// 64 < dim <= 128) in two launches: what a 16-token chunk needs of itself, all chunks at once, then a walk over every
// sequence's chunks with the state in registers.  The mathematics is that of linear_rnn_chunk.cu: with B_t = f_1 .. f_t and
// R_s = f_(s+1) .. f_16 inside a chunk (products of numbers <= 1, no quotient of them is ever formed)
//     prep   q_t B_t,   k_s R_s,   A_ts = sum_d q_td k_sd f_(s+1)d .. f_td,   B_16
//     walk   o_t = S_0^T (q_t B_t) + sum_(s<=t) A_ts v_s,     S_16^T = S_0^T diag(B_16) + V^T (K R)
// A warp of the prep holds four channels per lane and takes the tokens one by one: keys decayed so far stay in registers and
// are K R when the chunk ends.  Everything leaves as tensor-core fragments, bf16 high and low parts, in an order of channels
// that makes both the stores of the prep and the loads of the walk whole 16-byte vectors without bank conflicts.
// fp32 operands are bf16 pairs with the products hi hi + hi lo + lo hi (relative error 2^-16); v is bf16 as it comes.
#include "elem.cuh"
#include "linear_rnn.cuh"

namespace b200 {
namespace {

constexpr int OW_C = 16;                          // tokens per chunk
constexpr int OW_D = 128;                         // channels incl. padding
constexpr int OW_Q = 0, OW_K = 8192, OW_A = 16384, OW_B = OW_A + 1024, OW_SLOT = OW_B + OW_D * 4;   // bytes of a chunk's fragments
constexpr int OW_PREP_WARPS = 4;
constexpr int OW_WARPS = 8, OW_OUT_WARPS = 4, OW_THREADS = 32 * (OW_WARPS + OW_OUT_WARPS), OW_COLS = 16 * OW_WARPS;
constexpr int OW_OP = OW_COLS + 8;                // fp32 pitch of o: the rows of an accumulator store in different banks
constexpr int OW_VP = 24;                         // bf16 pitch of a warp's 16 x 16 values: 48-byte rows, conflict-free ldmatrix
constexpr int OW_STAGES = 4;

// Slots of a sequence's chunks start here: cu / 16 + b grows by at least the chunks of sequence b from b to b + 1.
__device__ __forceinline__ int64_t first_slot(const int32_t* cu, int b) { return cu[b] / OW_C + b; }

__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16(a, b);
  lo = pack_bf16(a - bf16_lo(hi), b - bf16_hi(hi));
}
__device__ __forceinline__ uint4 split_words(float a, float b, float c, float d) {   // (hi, hi, lo, lo) of two pairs
  uint4 w;
  split_pair(a, b, w.x, w.z);
  split_pair(c, d, w.y, w.w);
  return w;
}

// Raw inputs of one token: q, f' (KEYED: k, z) of four channels
template <bool KEYED>
struct Token {
  uint2 q, k;
  float4 z;
};

// Sums over the lanes of N values each (N a power of two up to 16): lane l is left with value (l >> 1) >> (4 - log2 N).
template <int N>
__device__ __forceinline__ float reduce_scatter(float (&v)[N], int lane) {
  int bit = 16;
#pragma unroll
  for (int n = N / 2; n >= 1; n >>= 1, bit >>= 1) {
    const bool up = lane & bit;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float keep = up ? v[i + n] : v[i], send = up ? v[i] : v[i + n];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
    }
  }
#pragma unroll
  for (; bit >= 1; bit >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], bit);
  return v[0];
}

// grid (slots, heads / OW_PREP_WARPS): a warp = one chunk of one head.  Issue-bound (gates, 136 products of four channels per
// lane, their sums over the lanes by halves: one shuffle per value instead of five); 128 registers a thread for 16 warps per SM.
template <bool KEYED>
__global__ void __launch_bounds__(32 * OW_PREP_WARPS, 4) outer_prep_kernel(const __grid_constant__ OuterRnnParams p, int batch) {
  __shared__ float As[OW_PREP_WARPS][OW_C][OW_C + 2];
  pdl_trigger();                                  // the walk waits for this grid before it reads the slots
  const int slot = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int b = -1;                                     // the last sequence whose slots start at or before this one
  for (int i0 = 0; i0 < batch; i0 += 32 * OW_PREP_WARPS)
    b += __syncthreads_count(i0 + tid < batch && first_slot(p.cu, i0 + tid) <= slot);
  const int head = blockIdx.y * OW_PREP_WARPS + warp;
  if (b < 0 || head >= p.heads) return;
  const int row0 = p.cu[b] + static_cast<int>(slot - first_slot(p.cu, b)) * OW_C, rows = min(OW_C, p.cu[b + 1] - row0);
  if (rows <= 0) return;
  const int ch = 4 * lane;
  const bool on = ch < p.dim;
  const __nv_bfloat16* base = static_cast<const __nv_bfloat16*>(p.x) + static_cast<int64_t>(row0) * p.stride + head * p.dim + ch;
  const float* zbase = KEYED ? p.z + static_cast<int64_t>(row0) * p.z_stride + head * p.dim + ch : nullptr;
  auto load = [&](int t) {
    Token<KEYED> x;
    x.q = x.k = make_uint2(0u, 0u), x.z = make_float4(0.f, 0.f, 0.f, 0.f);
    if (on && t < rows) {
      x.q = *reinterpret_cast<const uint2*>(base + t * p.stride + p.q_off);
      x.k = *reinterpret_cast<const uint2*>(base + t * p.stride + p.k_off);
      if constexpr (KEYED) x.z = load4(zbase + t * p.z_stride);
    }
    return x;
  };
  constexpr int AHEAD = KEYED ? 2 : 4;            // tokens requested at a time
  Token<KEYED> raw[2][AHEAD];
#pragma unroll
  for (int i = 0; i < AHEAD; ++i) raw[0][i] = load(i);
  float4 low = make_float4(0.f, 0.f, 0.f, 0.f), bias = low;
  if (on) {
    if constexpr (!KEYED) low = load4(p.lower + head * p.dim + ch);
    bias = load4(p.bias + head * p.dim + ch);
  }
  const F2 one = f2(1.f, 1.f);
  F2 run[2] = {one, one}, g[OW_C][2];             // B_t, and k_s f_(s+1) .. f_t, of channels (0, 1) and (2, 3)
  uint8_t* ws = reinterpret_cast<uint8_t*>(p.chunks) + (static_cast<int64_t>(slot) * p.heads + head) * OW_SLOT;
#pragma unroll
  for (int t = 0; t < OW_C; ++t) {
    if (t % AHEAD == 0 && t + AHEAD < OW_C) {
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) raw[(t / AHEAD + 1) & 1][i] = load(t + AHEAD + i);
    }
    const Token<KEYED> x = raw[(t / AHEAD) & 1][t % AHEAD];
    F2 q[2] = {f2(0.f, 0.f), f2(0.f, 0.f)}, f[2] = {one, one}, k[2] = {q[0], q[0]};   // padding keeps the state and reads nothing
    if (on && t < rows) {
      const float k0 = bf16_lo(x.k.x), k1 = bf16_hi(x.k.x), k2 = bf16_lo(x.k.y), k3 = bf16_hi(x.k.y);
      const float q0 = bf16_lo(x.q.x), q1 = bf16_hi(x.q.x), q2 = bf16_lo(x.q.y), q3 = bf16_hi(x.q.y);
      if constexpr (KEYED) {
        f[0] = f2(sigmoid_root<__nv_bfloat16>(x.z.x + bias.x, p.inv_tau), sigmoid_root<__nv_bfloat16>(x.z.y + bias.y, p.inv_tau));
        f[1] = f2(sigmoid_root<__nv_bfloat16>(x.z.z + bias.z, p.inv_tau), sigmoid_root<__nv_bfloat16>(x.z.w + bias.w, p.inv_tau));
        k[0] = f2(k0, k1), k[1] = f2(k2, k3);
        q[0] = f2(q0 * p.q_scale, q1 * p.q_scale), q[1] = f2(q2 * p.q_scale, q3 * p.q_scale);
      } else {
        const float f0 = low.x + (1.0f - low.x) * sigmoid_f<__nv_bfloat16>(k0 + bias.x), f1 = low.y + (1.0f - low.y) * sigmoid_f<__nv_bfloat16>(k1 + bias.y);
        const float f2_ = low.z + (1.0f - low.z) * sigmoid_f<__nv_bfloat16>(k2 + bias.z), f3 = low.w + (1.0f - low.w) * sigmoid_f<__nv_bfloat16>(k3 + bias.w);
        f[0] = f2(f0, f1), f[1] = f2(f2_, f3);
        k[0] = f2(1.0f - f0, 1.0f - f1), k[1] = f2(1.0f - f2_, 1.0f - f3);
        q[0] = f2(silu_f<__nv_bfloat16>(q0), silu_f<__nv_bfloat16>(q1)), q[1] = f2(silu_f<__nv_bfloat16>(q2), silu_f<__nv_bfloat16>(q3));
      }
    }
    // A's row t; the keys move on
    constexpr int MOST = OW_C;
    float a[MOST];
#pragma unroll
    for (int s = 0; s < MOST; ++s) {
      if (s > t) {
        a[s] = 0.f;
        continue;
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) g[s][c] = s < t ? mul2(g[s][c], f[c]) : k[c];
      const float2 y = unf2(fma2(q[1], g[s][1], mul2(q[0], g[s][0])));
      a[s] = y.x + y.y;
    }
    if (t < 4) {
      float v[4] = {a[0], a[1], a[2], a[3]};
      const float sum = reduce_scatter<4>(v, lane);
      if ((lane & 7) == 0) As[warp][t][lane >> 3] = sum;
    } else if (t < 8) {
      float v[8] = {a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7]};
      const float sum = reduce_scatter<8>(v, lane);
      if ((lane & 3) == 0) As[warp][t][lane >> 2] = sum;
    } else {
      const float sum = reduce_scatter<16>(a, lane);
      if ((lane & 1) == 0) As[warp][t][lane >> 1] = sum;
    }
    // q B: (hi, hi, lo, lo) of a lane's two channel pairs
#pragma unroll
    for (int c = 0; c < 2; ++c) run[c] = mul2(run[c], f[c]);
    const float2 u = unf2(mul2(q[0], run[0])), w = unf2(mul2(q[1], run[1]));
    *reinterpret_cast<uint4*>(ws + OW_Q + t * 512 + (lane ^ ((t & 1) * 4)) * 16) = split_words(u.x, u.y, w.x, w.y);
  }
  // K R: a channel's tokens 2 j, 2 j + 1, 2 j + 8, 2 j + 9
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    float x[OW_C];
#pragma unroll
    for (int s = 0; s < OW_C; ++s) {
      const float2 y = unf2(g[s][c >> 1]);
      x[s] = c & 1 ? y.y : y.x;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = c * 4 + j;
      *reinterpret_cast<uint4*>(ws + OW_K + i * 512 + (lane ^ (i & 7)) * 16) = split_words(x[2 * j], x[2 * j + 1], x[2 * j + 8], x[2 * j + 9]);
    }
  }
  const float2 b0 = unf2(run[0]), b1 = unf2(run[1]);
  *reinterpret_cast<float4*>(ws + OW_B + lane * 16) = make_float4(b0.x, b0.y, b1.x, b1.y);
  // A as a left operand: rows lane / 4 (+ 8), columns (lane % 4) * 2 (+ 1) (+ 8); above the diagonal nothing was left
  __syncwarp();
  uint32_t hi[4], lo[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = (lane >> 2) + (i & 1) * 8, s = (lane & 3) * 2 + (i >> 1) * 8;
    const float2 x = *reinterpret_cast<const float2*>(&As[warp][t][s]);
    split_pair(s <= t ? x.x : 0.f, s + 1 <= t ? x.y : 0.f, hi[i], lo[i]);
  }
  *reinterpret_cast<uint4*>(ws + OW_A + lane * 16) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
  *reinterpret_cast<uint4*>(ws + OW_A + 512 + lane * 16) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
}

template <bool V>
struct Flag {
  static constexpr bool value = V;
};

struct WalkSmem {
  uint8_t slot[OW_STAGES][OW_SLOT];
  __nv_bfloat16 v[OW_STAGES][OW_WARPS][OW_C * OW_VP];
  float o[2][OW_C][OW_OP];
  uint64_t full[OW_STAGES], done[2], taken[2];
};

// One CTA = one head of one sequence or segment and up to 128 value columns.  LOCAL: only the state from zero and the total
// decay of every segment.  Eight warps multiply, 16 value columns each, and bring their own values; four others take o from
// shared memory, a chunk behind: head norm, gate, stores.  Slots come by one bulk copy each, OW_STAGES ahead.
// What bounds it: the tensor pipe, 84 products per warp and chunk (8.4 cycles of a scheduler each, two warps per scheduler).  The
// state's update stands between the products of q and S, so that consecutive ones do not depend on one another, and nothing
// else is left to the multiplying warps (with norm, gate and stores in their own loop a chunk took 2.2 to 3.0 us, now 1.7; the
// pipe alone 1.4).  Half heads per CTA, two to a cluster that exchanges the norm's sums, gained on one long sequence and lost on
// batches: the exchange made the output warps the bound.
// 8 sequences of 256 to 1024 tokens, 16 heads of 128 x 128, both launches: HGRN2 336 -> 158 us, gated linear attention 461 -> 176
// against linear_rnn_chunk.cu, whose CTAs go through gates, decays, scores and products of every chunk in turn.
// grid (vdim / 128, heads, sequences * segments)
template <bool LOCAL>
__global__ void __launch_bounds__(OW_THREADS, 1) outer_walk_kernel(const __grid_constant__ OuterRnnParams p, int* err) {
  extern __shared__ __align__(128) uint8_t ow_smem[];
  WalkSmem& sm = *reinterpret_cast<WalkSmem*>(ow_smem);
  const int seq = blockIdx.z / p.segments, seg = blockIdx.z % p.segments, head = blockIdx.y, col0 = blockIdx.x * OW_COLS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int all = p.cu[seq + 1] - p.cu[seq], seg0 = seg * p.segment;
  const int row0 = p.cu[seq] + seg0, len = min(all - seg0, p.segment);
  if (len <= 0 || (LOCAL && seg0 + len == all)) {   // nothing follows a sequence's last segment
    pdl_wait();                                   // an idle CTA still orders the grid after the preparation
    return;
  }
  if (first_slot(p.cu, seq) + (all + OW_C - 1) / OW_C > p.chunk_slots) {   // more tokens than the call named: nobody prepared the end
    pdl_wait();
    if (tid == 0) atomicExch(err, 1);
    return;
  }
  const int chunks = (len + OW_C - 1) / OW_C;
  if (tid == 0) {
#pragma unroll
    for (int s = 0; s < OW_STAGES; ++s) mbar_init(&sm.full[s], 1);
#pragma unroll
    for (int b = 0; b < 2; ++b) mbar_init(&sm.done[b], OW_WARPS), mbar_init(&sm.taken[b], OW_OUT_WARPS);
    mbar_fence_init();
  }
  __syncthreads();
  if (warp >= OW_WARPS) {
    // ------------------------------------------------------------------------------------------------ copies and outputs
    const int out_warp = warp - OW_WARPS, c = col0 + 4 * lane;
    const uint8_t* slots = reinterpret_cast<const uint8_t*>(p.chunks) + ((first_slot(p.cu, seq) + seg0 / OW_C) * p.heads + head) * OW_SLOT;
    auto fetch_slot = [&](int i) {                // the parts a pass reads
      uint64_t* bar = &sm.full[i % OW_STAGES];
      constexpr int skip = LOCAL ? OW_K : 0;
      mbar_expect_tx(bar, OW_SLOT - skip);
      bulk_g2s(sm.slot[i % OW_STAGES] + skip, slots + static_cast<int64_t>(i) * p.heads * OW_SLOT + skip, OW_SLOT - skip, bar);
    };
    const bool copies = tid == 32 * OW_WARPS, on = c < p.vdim, fused_norm = p.out != nullptr;
    pdl_wait();                                   // the slots are complete
    if (copies)
      for (int i = 0; i < OW_STAGES && i < chunks; ++i) fetch_slot(i);
    float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!LOCAL && fused_norm && on) w = load4(p.norm + c);
    constexpr int ROWS = OW_C / OW_OUT_WARPS;
    const __nv_bfloat16* gate = p.gate ? static_cast<const __nv_bfloat16*>(p.gate) + row0 * p.gate_stride + head * p.vdim + c : nullptr;
    static_assert(ROWS == 4, "a warp's rows are dealt to its lanes by two bits");
    const int t0 = out_warp * ROWS;
    uint2 raw[2][ROWS] = {};                      // silu's inputs, requested a chunk ahead
    auto request = [&](int i, uint2 (&to)[ROWS]) {
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
        if (on && i * OW_C + t0 + r < len) to[r] = *reinterpret_cast<const uint2*>(gate + (i * OW_C + t0 + r) * p.gate_stride);
    };
    auto take = [&](int i, const uint2 (&silu_in)[ROWS], uint2 (&next)[ROWS]) {
      const int first = i * OW_C + t0;
      if (!LOCAL && gate && i + 1 < chunks) request(i + 1, next);
      if (!warp_wait_bounded(&sm.done[i & 1], (i >> 1) & 1)) return false;
      if (copies && i + OW_STAGES < chunks) fetch_slot(i + OW_STAGES);
      float4 y[ROWS];
      if (!LOCAL) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r) y[r] = on ? *reinterpret_cast<const float4*>(&sm.o[i & 1][t0 + r][4 * lane]) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.taken[i & 1]);
      if (LOCAL) return true;
      if (fused_norm) {
        // Sums over the warp by halves: lane bits 4 and 3 are left with the row, and a lane sees to one row's scale.  (Four sums and
        // four scales in every lane made this loop, not the products, the bound: 1.9 us a chunk.)
        float v[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) v[r] = y[r].x * y[r].x + y[r].y * y[r].y + y[r].z * y[r].z + y[r].w * y[r].w;
        const bool up16 = lane & 16, up8 = lane & 8;
        float a = (up16 ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, up16 ? v[0] : v[2], 16);
        const float b = (up16 ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, up16 ? v[1] : v[3], 16);
        a = (up8 ? b : a) + __shfl_xor_sync(0xffffffffu, up8 ? a : b, 8);
        a += __shfl_xor_sync(0xffffffffu, a, 4);
        a += __shfl_xor_sync(0xffffffffu, a, 2);
        a += __shfl_xor_sync(0xffffffffu, a, 1);
        const float my_scale = 1.0f / sqrtf(a / static_cast<float>(p.true_vdim) + p.eps);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          const float scale = __shfl_sync(0xffffffffu, my_scale, r * 8);
          float4 z = make_float4(y[r].x * scale * w.x, y[r].y * scale * w.y, y[r].z * scale * w.z, y[r].w * scale * w.w);
          if (gate) {
            z.x *= silu_f<__nv_bfloat16>(bf16_lo(silu_in[r].x)), z.y *= silu_f<__nv_bfloat16>(bf16_hi(silu_in[r].x));
            z.z *= silu_f<__nv_bfloat16>(bf16_lo(silu_in[r].y)), z.w *= silu_f<__nv_bfloat16>(bf16_hi(silu_in[r].y));
          }
          if (on && first + r < len) store4(static_cast<__nv_bfloat16*>(p.out) + (row0 + first + r) * p.out_stride + head * p.vdim + c, z);
        }
      } else {
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
          if (on && first + r < len) store4(p.o + (static_cast<int64_t>(row0 + first + r) * p.heads + head) * p.vdim + c, y[r]);
      }
      return true;
    };
    if (!LOCAL && gate) request(0, raw[0]);
    bool ok = true;
    int at = 0;                                   // the chunk waited for last
#pragma unroll 1
    for (int i = 0; i < chunks && ok; i += 2) {
      ok = take(at = i, raw[0], raw[1]);
      if (ok && i + 1 < chunks) ok = take(at = i + 1, raw[1], raw[0]);
    }
    if (!ok) {
      atomicExch(err, 1);
      // bulk copies that nobody waits for any more may still be landing in this CTA's shared memory
      if (copies)
        for (int i = at; i < at + OW_STAGES && i < chunks; ++i) mbar_wait_bounded(&sm.full[i % OW_STAGES], i / OW_STAGES & 1, 1u << 12);
    }
    return;
  }
  // ---------------------------------------------------------------------------------------------------------- products
  const int wcol = col0 + warp * 16;
  const bool warp_on = wcol < p.vdim;
  const __nv_bfloat16* values = static_cast<const __nv_bfloat16*>(p.x) + static_cast<int64_t>(row0) * p.stride + p.v_off + head * p.vdim;
  auto fetch_values = [&](int i) {                // a warp's own 16 columns, one vector per lane; zeros behind the end
    const int t = lane >> 1, c = wcol + (lane & 1) * 8;
    const bool on = i * OW_C + t < len && c < p.vdim;
    if (i < chunks)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(&sm.v[i % OW_STAGES][warp][t * OW_VP + (lane & 1) * 8])),
                   "l"(values + (on ? (i * OW_C + t) * p.stride + c : 0)), "r"(on ? 16 : 0)
                   : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < OW_STAGES; ++i) fetch_values(i);
  // S^T: value column lane / 4 (+ 8); tile n = 2 m + a holds channels 16 m + (lane % 4) * 4 + 2 a (+ 1)
  float S[OW_D / 8][4];
  const int64_t head_elems = static_cast<int64_t>(p.dim) * p.vdim;
  float* slot_state = p.state + (static_cast<int64_t>(p.slots[seq]) * p.heads + head) * head_elems;
  float* seg_state = p.seg_state + (static_cast<int64_t>(blockIdx.z) * p.heads + head) * head_elems;
  const float* from = p.segments > 1 ? seg_state : slot_state;
  const bool carry = !LOCAL && (p.segments > 1 || p.start[seq] > 0);
  const int my_col = wcol + (lane >> 2), my_ch = (lane & 3) * 4;
#pragma unroll
  for (int n = 0; n < OW_D / 8; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int d = (n >> 1) * 16 + my_ch + (n & 1) * 2 + (j & 1), c = my_col + (j >> 1) * 8;
      S[n][j] = carry && d < p.dim && c < p.vdim ? from[static_cast<int64_t>(d) * p.vdim + c] : 0.f;
    }
  float total = 1.f;
#pragma unroll 1
  for (int i = 0; i < chunks; ++i) {
    const int st = i % OW_STAGES;
    asm volatile("cp.async.wait_group %0;" ::"n"(OW_STAGES - 1) : "memory");
    __syncwarp();
    // the slot is here, and the buffer of o that chunk i - 2 used is free (so the barriers are never two phases ahead)
    const bool taken = i < 2 || mbar_wait_bounded(&sm.taken[i & 1], ((i >> 1) - 1) & 1);
    if (!warp_wait_bounded(&sm.full[st], (i / OW_STAGES) & 1, taken)) {
      atomicExch(err, 1);
      asm volatile("cp.async.wait_all;" ::: "memory");
      return;
    }
    const uint8_t* at = sm.slot[st];
    float o[2][4] = {}, x[2][4] = {};             // products of high parts; all others
    if (warp_on) {
      uint32_t vm[4];   // the chunk's values of this warp's columns: matrices (k 0-7, c 0-7), (k 0-7, c 8-15), (k 8-15, ...)
      ldmatrix_x4_trans(vm, smem_u32(&sm.v[st][warp][((lane & 7) + (lane >> 4) * 8) * OW_VP + ((lane >> 3) & 1) * 8]));
      if (!LOCAL) {
        const uint4 ah4 = *reinterpret_cast<const uint4*>(at + OW_A + lane * 16), al4 = *reinterpret_cast<const uint4*>(at + OW_A + 512 + lane * 16);
        const uint32_t ah[4] = {ah4.x, ah4.y, ah4.z, ah4.w}, al[4] = {al4.x, al4.y, al4.z, al4.w};
        mma_bf16_16816(o[0], ah, vm[0], vm[2]);
        mma_bf16_16816(o[1], ah, vm[1], vm[3]);
        mma_bf16_16816(x[0], al, vm[0], vm[2]);
        mma_bf16_16816(x[1], al, vm[1], vm[3]);
      }
      const uint8_t* q0 = at + OW_Q + (lane >> 2) * 512;
      const int flip = ((lane >> 2) & 1) * 4;
      // the update's tile (m, a), slot lane / 4 = channel 16 m + (slot / 2) * 4 + 2 a + slot % 2
      const int slot = lane >> 2, row = (slot & 1) * 4 + (lane & 3);
      auto products = [&](auto enters) {          // whether a state enters the chunk
#pragma unroll
        for (int m = 0; m < OW_D / 16; ++m) {
          float(&a)[4] = S[2 * m];
          float(&b)[4] = S[2 * m + 1];
          const float4 d = *reinterpret_cast<const float4*>(at + OW_B + (4 * m + (lane & 3)) * 16);
          const uint8_t* kr = at + OW_K + ((4 * m + (slot >> 1)) ^ row) * 16 + row * 512;
          const uint4 k0 = *reinterpret_cast<const uint4*>(kr), k1 = *reinterpret_cast<const uint4*>(kr + 8 * 512);
          if (enters.value) {
            const int unit = ((4 * m + (lane & 3)) ^ flip) * 16;
            const uint4 r0 = *reinterpret_cast<const uint4*>(q0 + unit), r1 = *reinterpret_cast<const uint4*>(q0 + 8 * 512 + unit);
            const uint32_t qh[4] = {r0.x, r1.x, r0.y, r1.y}, ql[4] = {r0.z, r1.z, r0.w, r1.w};
            uint32_t h[2][2], l[2][2];
#pragma unroll
            for (int n = 0; n < 2; ++n) {           // value columns 0-7 and 8-15 of the warp
              split_pair(a[2 * n], a[2 * n + 1], h[n][0], l[n][0]);
              split_pair(b[2 * n], b[2 * n + 1], h[n][1], l[n][1]);
            }
            a[0] *= d.x, a[1] *= d.y, a[2] *= d.x, a[3] *= d.y;
            b[0] *= d.z, b[1] *= d.w, b[2] *= d.z, b[3] *= d.w;
            mma_bf16_16816(x[0], qh, l[0][0], l[0][1]);
            mma_bf16_16816(x[1], qh, l[1][0], l[1][1]);
            mma_bf16_16816(a, vm, k0.x, k0.y);
            mma_bf16_16816(b, vm, k1.x, k1.y);
            mma_bf16_16816(o[0], qh, h[0][0], h[0][1]);
            mma_bf16_16816(o[1], qh, h[1][0], h[1][1]);
            mma_bf16_16816(x[0], ql, h[0][0], h[0][1]);
            mma_bf16_16816(x[1], ql, h[1][0], h[1][1]);
          } else {
            a[0] *= d.x, a[1] *= d.y, a[2] *= d.x, a[3] *= d.y;
            b[0] *= d.z, b[1] *= d.w, b[2] *= d.z, b[3] *= d.w;
            mma_bf16_16816(a, vm, k0.x, k0.y);
            mma_bf16_16816(b, vm, k1.x, k1.y);
          }
          mma_bf16_16816(a, vm, k0.z, k0.w);
          mma_bf16_16816(b, vm, k1.z, k1.w);
        }
      };
      if (!LOCAL && (carry || i > 0)) products(Flag<true>());
      else products(Flag<false>());
    }
    if (LOCAL && tid < OW_D) total *= *reinterpret_cast<const float*>(at + OW_B + tid * 4);
    fetch_values(i + OW_STAGES);                  // the warp has read its stage of values
    if (!LOCAL) {
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int half = 0; half < 2; ++half)
          *reinterpret_cast<float2*>(&sm.o[i & 1][(lane >> 2) + half * 8][warp * 16 + n * 8 + (lane & 3) * 2]) =
              make_float2(o[n][2 * half] + x[n][2 * half], o[n][2 * half + 1] + x[n][2 * half + 1]);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.done[i & 1]);
  }
  pdl_wait();                                     // the launches before this one are done: their states may be overwritten
  if (!LOCAL && seg0 + len < all) return;         // only the last segment leaves the sequence's state behind
  float* to = LOCAL ? seg_state : slot_state;
#pragma unroll
  for (int n = 0; n < OW_D / 8; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int d = (n >> 1) * 16 + my_ch + (n & 1) * 2 + (j & 1), c = my_col + (j >> 1) * 8;
      if (d < p.dim && c < p.vdim) to[static_cast<int64_t>(d) * p.vdim + c] = S[n][j];
    }
  if (LOCAL && blockIdx.x == 0 && tid < p.dim) p.seg_decay[(static_cast<int64_t>(blockIdx.z) * p.heads + head) * p.dim + tid] = total;
}

int64_t slots_of(int64_t tokens, int64_t batch) { return tokens / OW_C + batch; }

template <bool LOCAL>
int launch_pass(const OuterRnnParams& p, dim3 grid, bool early, int* err, cudaStream_t st) {
  constexpr int smem = sizeof(WalkSmem);
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    if (cudaFuncSetAttribute(outer_walk_kernel<LOCAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
      return fail(ERR_RUNTIME, "outer_rnn: cannot raise dynamic shared memory to %d", smem);
    configured[dev] = true;
  }
  if (launch_pdl(early, outer_walk_kernel<LOCAL>, grid, dim3(OW_THREADS), smem, st, p, err) != cudaSuccess)
    return fail(ERR_LAUNCH, "outer_rnn: %s", cudaGetErrorString(cudaGetLastError()));
  return OK;
}

template <bool KEYED>
int launch_walk(OuterRnnParams p, int n, int tokens, cudaStream_t st) {
  int* err = wait_timeout_flag();
  if (!err) return fail(ERR_RUNTIME, "outer_rnn: no error flag");
  p.chunk_slots = static_cast<int>(slots_of(tokens, n));
  const dim3 prep(static_cast<unsigned>(p.chunk_slots), (p.heads + OW_PREP_WARPS - 1) / OW_PREP_WARPS);
  outer_prep_kernel<KEYED><<<prep, 32 * OW_PREP_WARPS, 0, st>>>(p, n);
  const dim3 grid((p.vdim + OW_COLS - 1) / OW_COLS, p.heads, n * p.segments);
  if (p.segments > 1) {
    const int rc = launch_pass<true>(p, grid, true, err, st);
    if (rc != OK) return rc;
    outer_rnn_fold_launch(p, n, st);
  }
  const int rc = launch_pass<false>(p, grid, p.segments == 1, err, st);
  return rc != OK ? rc : check_launch("outer_rnn (walk)");
}

}  // namespace

bool outer_rnn_walk_supports(const OuterRnnParams& p) {
  return p.chunks && p.dim > 64 && p.dim <= OW_D && p.dim % 8 == 0 && p.vdim % 8 == 0 && aligned16(p.bias) && (!p.lower || aligned16(p.lower));
}
int outer_rnn_walk_launch(const OuterRnnParams& p, RnnKind kind, int n, int tokens, cudaStream_t st) {
  return kind == RNN_KEYED ? launch_walk<true>(p, n, tokens, st) : launch_walk<false>(p, n, tokens, st);
}

}  // namespace b200

using namespace b200;

// 1120 bytes per token and head: at most 1 GiB, a small part of the card's memory.
extern "C" int64_t b200_outer_walk_workspace_bytes(int32_t tokens, int32_t batch, int32_t heads, int32_t dim, int32_t vdim) {
  if (tokens <= 0 || batch <= 0 || dim <= 64 || dim > OW_D || dim % 8 != 0 || vdim % 8 != 0) return 0;
  const int64_t bytes = slots_of(tokens, batch) * heads * OW_SLOT;
  return bytes <= (int64_t{1} << 30) ? bytes : 0;
}
