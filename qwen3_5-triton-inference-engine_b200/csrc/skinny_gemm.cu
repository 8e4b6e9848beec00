// Weight-streaming GEMM for decode batches:  Y[M, N] = X[M, K] . W[N, K]^T  with M <= 32 rows (one token per
// sequence), bf16 in / bf16 out, fp32 accumulation.  Replaces triton_kernels/gemm_2d.py for the decode-step projections
// whose input width is the model's hidden size; the reference's own note is that these GEMVs are about half of a
// decode step (README-EN.md:116).
//
// The product is HBM-bound on W (M is tiny), so the kernel is built like the decode-attention kernels: X is staged once
// per CTA in shared memory (a tensor-map box per 128 columns), every warp streams rows of W through a private ring of 4 KiB tiles
// (tensor-map TMA, 128-byte swizzle -> conflict-free ldmatrix, one mbarrier per tile, no cluster multicast), and
// multiplies with mma.sync m16n8k16 taking the W rows as the MMA M dimension and the batch as N (M <= 32 is far too
// thin for a tcgen05 tile).  CTAs walk the row blocks persistently, so X is read once per CTA however large N is.
// Every wait is bounded.
//
// Two forms.  Plain: a warp's tile is 16 consecutive rows of W (one box {64 k, 16 rows, 2 k-blocks}), a CTA covers 64
// outputs with four row groups of two warps each (the even and the odd k tiles).  SwiGLU (W = [gate rows | up rows], the fused gate/up projection followed by
// triton_kernels/swiglu.py): a warp's tile is 8 gate rows stacked on the 8 matching up rows (two boxes of 8 rows), so the
// accumulator fragment of a thread holds gate_j (row r) and up_j (row r + 8) of the same output j and the activation is
// applied in registers; a CTA covers 32 outputs.
//
// The residual add and RMSNorm between a projection back to the hidden size and the next one need no launch of their own: the
// pair-K form that produces the rows adds the residual and writes, next to the sum s, the rows s (1 + gain) and the sum of squares of every 16
// columns; the product behind it takes those rows as X and multiplies its sums by the row's 1 / rms, which is complete long before
// the weights are through.  Decode step of the 24-layer 0.8B model: one sequence 634 -> 608 us, 8 sequences 747 -> 703, 32 917 -> 885.
#include "b200_attn.h"
#include "umma.cuh"

#include <mutex>

namespace b200 {

constexpr int SG_WARPS = 4;
constexpr int SG_THREADS = SG_WARPS * 32;
constexpr int SG_ROWS = 16 * SG_WARPS;   // outputs per CTA step, plain form (8 * SG_WARPS in the SwiGLU form)
constexpr int SG_TILE_K = 128;           // k elements per tile: two swizzled blocks of [16 rows][64 k] bf16
constexpr int SG_TILE_BYTES = 2 * 16 * 128;
constexpr int SG_RING = 8;                        // tiles in flight per warp
constexpr int SG_RING_BYTES = SG_RING * SG_TILE_BYTES;
constexpr int SG_KSPLIT = 2;                      // K = 1280 or less: warps per row group, alternating k tiles
constexpr int SG_STD_WARPS = SG_WARPS * SG_KSPLIT;
constexpr int SG_STD_THREADS = SG_STD_WARPS * 32;
constexpr int SG_STD_RING = SG_RING / SG_KSPLIT;  // the same bytes in flight per CTA
constexpr int SG_MAX_M = 32;
constexpr int SG_MAX_K = 1280;           // X staging: 32 rows of it next to 128 KiB of weight rings (skinny_smem)

struct SkinnyGemmParams {
  const __nv_bfloat16* x;  // [M, K]
  __nv_bfloat16* y;        // [M, N]
  int64_t x_stride, y_stride;
  int* err;
  int m, n, k, row_blocks, overlap, up_row0;  // n: outputs; up_row0: first W row of the `up` half (SwiGLU form)
  const float* squares;    // normed form: [M, K / 16] sums of squares of 16 columns each; null: X as it is
  float eps;
  int true_k;              // columns that the mean counts (the others are zeros)
  // arg-max form: ids[b] = argmax_n y[b, n] instead of y (keys / counter: zero-filled workspace, left zero)
  int64_t* ids;
  unsigned long long* keys;
  int* counter;
};

// Which m16n8k16 products a step of 16 k takes for NT groups of eight batch rows, and the sums they go to.  A warp's k steps are a
// chain: with fewer than four groups the steps take turns among the four accumulators, joined at the end by `join_steps`.
// One step costs eight cycles of a scheduler per group, and two warps share one: 31 rows of zeros behind a single one were most of 1.8 us
// of a 6.3 us launch.
template <int NT>
struct StepProducts;
template <>
struct StepProducts<4> {
  // lane address: row = (lane & 7) + 8 * (lane >> 4) of sixteen, k half = (lane >> 3) & 1
  static __device__ __forceinline__ uint32_t lane_offset(int lane) {
    return static_cast<uint32_t>(((lane & 7) + ((lane >> 4) << 3)) * 128 + (((lane >> 3) & 1) ^ (lane & 7)) * 16);
  }
  template <int KS>
  static __device__ __forceinline__ void run(float (&acc)[4][4], const uint32_t (&a)[4], uint32_t (&b)[8], uint32_t xk) {
    uint32_t b01[4], b23[4];
    ldmatrix_x4(b01, xk);                   // batch rows 0-15: (b0, b1) of n8 tiles 0 and 1
    ldmatrix_x4(b23, xk + 16 * 128);        // batch rows 16-31
    mma_bf16_16816(acc[0], a, b01[0], b01[1]);
    mma_bf16_16816(acc[1], a, b01[2], b01[3]);
    mma_bf16_16816(acc[2], a, b23[0], b23[1]);
    mma_bf16_16816(acc[3], a, b23[2], b23[3]);
  }
};
template <>
struct StepProducts<2> {
  static __device__ __forceinline__ uint32_t lane_offset(int lane) { return StepProducts<4>::lane_offset(lane); }
  template <int KS>
  static __device__ __forceinline__ void run(float (&acc)[4][4], const uint32_t (&a)[4], uint32_t (&b)[8], uint32_t xk) {
    uint32_t b01[4];
    ldmatrix_x4(b01, xk);
    mma_bf16_16816(acc[(KS & 1) * 2], a, b01[0], b01[1]);
    mma_bf16_16816(acc[(KS & 1) * 2 + 1], a, b01[2], b01[3]);
  }
};
template <>
struct StepProducts<1> {
  // eight rows, four k groups of eight: one load serves two steps
  static __device__ __forceinline__ uint32_t lane_offset(int lane) { return static_cast<uint32_t>((lane & 7) * 128 + ((lane >> 3) ^ (lane & 7)) * 16); }
  template <int KS>
  static __device__ __forceinline__ void run(float (&acc)[4][4], const uint32_t (&a)[4], uint32_t (&b)[8], uint32_t xk) {
    uint32_t (&b4)[4] = *reinterpret_cast<uint32_t (*)[4]>(b);
    if constexpr ((KS & 1) == 0) ldmatrix_x4(b4, xk);
    mma_bf16_16816(acc[KS & 3], a, b[(KS & 1) * 2], b[(KS & 1) * 2 + 1]);
  }
};
template <int NT>
__device__ __forceinline__ void join_steps(float (&acc)[4][4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if constexpr (NT == 1) acc[0][j] = (acc[0][j] + acc[1][j]) + (acc[2][j] + acc[3][j]);
    if constexpr (NT == 2) {
      acc[0][j] += acc[2][j];
      acc[1][j] += acc[3][j];
    }
  }
}
// The eight steps of a tile of 128 k: A (W tile) by ldmatrix from `tile` + offset(step), X from xj[step & 3] + `xt` on: two blocks of
// [8 NT rows][64 k] with the 128-byte swizzle, where a step's 32 bytes are two bits of the lane's address to turn over.
template <int NT, int KS, typename Offset>
__device__ __forceinline__ void tile_steps(float (&acc)[4][4], uint32_t (&b)[8], uint32_t tile, const uint32_t (&xj)[4], uint32_t xt, const Offset& offset) {
  if constexpr (KS < SG_TILE_K / 16) {
    uint32_t a[4];
    ldmatrix_x4(a, tile + offset(KS));
    StepProducts<NT>::template run<KS>(acc, a, b, xj[KS & 3] + xt + (KS >> 2) * (NT * 8 * 128));
    tile_steps<NT, KS + 1>(acc, b, tile, xj, xt, offset);
  }
}
constexpr int skinny_smem(int nt, int k) {  // rings, output staging, odd-tile sums, X
  return SG_WARPS * SG_RING_BYTES + nt * 8 * SG_ROWS * 2 + nt * 4 * SG_WARPS * 32 * 4 + nt * 8 * k * 2 + 2048;
}

// NT: groups of eight batch rows that are staged and multiplied (M <= 8, 16 or 32 rows)
template <bool SWIGLU, bool ARGMAX, int NT>
__global__ void __launch_bounds__(SG_STD_THREADS, 1)
skinny_gemm_kernel(const __grid_constant__ SkinnyGemmParams p, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  constexpr int SLOT_BYTES = SG_TILE_BYTES;
  constexpr int RING = SG_STD_RING;
  constexpr int OUT = SWIGLU ? 8 * SG_WARPS : SG_ROWS;  // outputs per CTA step
  constexpr int ROWS = NT * 8;
  __shared__ uint64_t bars[SG_STD_WARPS][RING];
  __shared__ uint64_t bar_x[SG_MAX_K / SG_TILE_K];  // one per k tile
  __shared__ __align__(8) float scale[ROWS];                   // normed form: 1 / rms of the rows
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // warps wr and wr + 4 share the rows of group wr and take the even / the odd k tiles: a warp's k steps are a chain of
  // dependent ldmatrix + MMA, so two short chains per row group finish in half the time of one long one
  const int wr = warp & (SG_WARPS - 1), kh = warp / SG_WARPS;
  uint8_t* ring = smem + warp * (RING * SLOT_BYTES);
  uint8_t* stage = smem + SG_WARPS * SG_RING_BYTES;                    // [ROWS][OUT] bf16 output staging, <= 4 KiB
  float* part = reinterpret_cast<float*>(stage + ROWS * SG_ROWS * 2);  // [4 NT][4 groups x 32 lanes]: odd-tile sums
  constexpr int X_TILE = ROWS * SG_TILE_K * 2;
  // X, tile by tile; the swizzle counts from 1024-byte boundaries
  uint8_t* xs = smem + (SG_WARPS * SG_RING_BYTES + ROWS * SG_ROWS * 2 + 4 * NT * SG_WARPS * 32 * 4 + 1023) / 1024 * 1024;
  const int k_tiles = p.k / SG_TILE_K;

  if (lane == 0) {
    for (int s = 0; s < RING; ++s) mbar_init(&bars[warp][s], 1);
    if (warp == 0)
      for (int i = 0; i < SG_MAX_K / SG_TILE_K; ++i) mbar_init(&bar_x[i], 1);
    mbar_fence_init();
  }
  // my tiles: row block rb = blockIdx.x, + gridDim.x, ...; tile index t counts (row block, k tile) pairs
  const int my_blocks = (p.row_blocks - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
  const int my_kt = (k_tiles - kh + SG_KSPLIT - 1) / SG_KSPLIT;  // k tiles kh, kh + 2, ... of every row block
  const int total_tiles = my_blocks * my_kt;
  __syncwarp();
  auto issue = [&](int t) {
    const int rb = blockIdx.x + (t / my_kt) * gridDim.x, kt = kh + SG_KSPLIT * (t % my_kt);
    const int slot = t % RING;
    mbar_expect_tx(&bars[warp][slot], SLOT_BYTES);
    if (SWIGLU) {  // map_w has 8-row boxes: gate rows to the first half of the tile, up rows to the second
      tma_load_3d(ring + slot * SLOT_BYTES, &map_w, 0, rb * OUT + wr * 8, kt * 2, &bars[warp][slot]);
      tma_load_3d(ring + slot * SLOT_BYTES + SG_TILE_BYTES / 2, &map_w, 0, p.up_row0 + rb * OUT + wr * 8, kt * 2,
                  &bars[warp][slot]);
    } else {
      tma_load_3d(ring + slot * SLOT_BYTES, &map_w, 0, rb * OUT + wr * 16, kt * 2, &bars[warp][slot]);
    }
  };
  // X by tensor-map boxes of a k tile each, whose products start when it is there; rows beyond M arrive as zeros.  A copy takes some 60
  // cycles of the thread that asks for it, whatever its size, so every warp asks for some.  Decode step of 8 / 16 / 32 sequences: rows by
  // loads of all threads 703 / 882 / 1047 us, a copy per row - / - / 985, boxes from one thread 645 / 717 / 888, from all warps 634 / 709 / 872
  // (one sequence: 608, -, 614, 597).
  auto stage_x = [&]() {
    for (int kt = warp; kt < k_tiles; kt += SG_STD_WARPS) {
      mbar_expect_tx(&bar_x[kt], X_TILE);
      tma_load_3d(xs + kt * X_TILE, &map_x, 0, 0, kt * 2, &bar_x[kt]);
    }
  };
  // Started early, the weights are requested while the predecessor runs and X after it.  In plain stream order X goes
  // first: requested behind 128 KiB of weight tiles it would arrive behind them.
  const bool early = (p.overlap & OVERLAP_START) != 0;
  if (p.overlap & OVERLAP_TRIGGER) pdl_trigger();
  __syncthreads();  // bar_x is initialised for everybody
  if (!early && lane == 0) stage_x();
  if (lane == 0) {
    for (int t = 0; t < RING && t < total_tiles; ++t) issue(t);  // weights: independent of the predecessor
  }
  pdl_wait();  // X is the predecessor's output
  // normed form: eight threads per row, asked for now and first looked at behind the products
  constexpr int SQUARES = SG_MAX_K / 16 / 8;
  const bool normed = !ARGMAX && p.squares != nullptr;   // a positive factor per row moves no arg-max (and cost the LM head of 32 rows 2 of 91 us)
  float sq[SQUARES];
#pragma unroll
  for (int i = 0; i < SQUARES; ++i)
    sq[i] = normed && (tid >> 3) < p.m && i * 8 + (tid & 7) < (p.k >> 4) ? p.squares[(tid >> 3) * (p.k >> 4) + i * 8 + (tid & 7)] : 0.f;
  if (early && lane == 0) stage_x();
  bool ok = true;

  const uint32_t xs_base = smem_u32(xs);
  // ldmatrix lane address of A (W tile): row = lane % 16, chunk parity = lane / 16
  const int a_row = lane & 15, a_par = lane >> 4;
  const uint32_t xs_lane = xs_base + StepProducts<NT>::lane_offset(lane);
  const uint32_t xj[4] = {xs_lane, xs_lane ^ 32, xs_lane ^ 64, xs_lane ^ 96};
  const auto a_offset = [&](int ks) -> uint32_t {
    // plain: [k-block][16 rows][128 B]; SwiGLU: [gate | up][k-block][8 rows][128 B]; 16-byte chunks XOR-swizzled by row
    return (SWIGLU ? (a_row >> 3) * (SG_TILE_BYTES / 2) + (ks >> 2) * (8 * 128) + (a_row & 7) * 128 : (ks >> 2) * (16 * 128) + a_row * 128) +
           ((((ks & 3) * 2 + a_par) ^ (a_row & 7)) << 4);
  };
  // arg-max form: this thread's running best over its rows, per batch column (nt * 2 + (j & 1))
  float best_v[2 * NT];
  uint32_t best_i[2 * NT];
#pragma unroll
  for (int c = 0; c < 2 * NT; ++c) {
    best_v[c] = -INFINITY;
    best_i[c] = 0xffffffffu;
  }
  int t = 0;
  for (int blk = 0; blk < my_blocks; ++blk) {  // a failed wait clears `ok`; the loop then only keeps its barriers
    const int rb = blockIdx.x + blk * gridDim.x;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    for (int kt = kh; kt < k_tiles && ok; kt += SG_KSPLIT, ++t) {
      const int slot = t % RING;
      if (!mbar_wait_bounded(&bars[warp][slot], (t / RING) & 1)) {
        ok = false;
        break;
      }
      if (blk == 0 && !mbar_wait_bounded(&bar_x[kt], 0)) {
        ok = false;
        break;
      }
      uint32_t b[8];
      tile_steps<NT, 0>(acc, b, smem_u32(ring + slot * SLOT_BYTES), xj, kt * X_TILE, a_offset);
      __syncwarp();  // every lane has read the tile: its slot can take the tile RING ahead
      if (lane == 0 && t + RING < total_tiles) issue(t + RING);
    }
    join_steps<NT>(acc);
    // the odd-tile warps hand their sums to the even-tile warps of the same row group
    if (kh == 1) {
#pragma unroll
      for (int i = 0; i < 4 * NT; ++i) part[i * (SG_WARPS * 32) + wr * 32 + lane] = acc[i >> 2][i & 3];
    }
    if (normed && blk == 0) {
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < SQUARES; ++i) ss += sq[i];
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if ((tid & 7) == 0 && (tid >> 3) < ROWS) scale[tid >> 3] = rsqrtf(ss / static_cast<float>(p.true_k) + p.eps);
    }
    __syncthreads();  // (also: the previous block's staging has been written out)
    // acc[nt]: rows (tile row = lane/4, +8), cols (batch = nt*8 + (lane%4)*2, +1)  ->  stage[batch][output] -> Y
    if (kh == 0) {
#pragma unroll
      for (int i = 0; i < 4 * NT; ++i) acc[i >> 2][i & 3] += part[i * (SG_WARPS * 32) + wr * 32 + lane];
      if (normed) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          const float2 r = *reinterpret_cast<const float2*>(scale + nt * 8 + (lane & 3) * 2);
          acc[nt][0] *= r.x, acc[nt][1] *= r.y, acc[nt][2] *= r.x, acc[nt][3] *= r.y;
        }
      }
    }
    if (ARGMAX) {
      if (kh == 0) {
        // rows ascend with the row block and, inside it, from fragment row r to r + 8: strict > keeps the lowest index
        const uint32_t n_lo = static_cast<uint32_t>(rb * OUT + wr * 16 + (lane >> 2));
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int c = nt * 2 + (j & 1);
            const uint32_t n = n_lo + (j >= 2 ? 8u : 0u);
            if (n < static_cast<uint32_t>(p.n) && (acc[nt][j] > best_v[c] || best_i[c] == 0xffffffffu)) {
              best_v[c] = acc[nt][j];
              best_i[c] = n;
            }
          }
      }
      __syncthreads();  // `part` may be rewritten by the next row block
      continue;
    }
    if (kh == 0) {
      __nv_bfloat16* st = reinterpret_cast<__nv_bfloat16*>(stage);
      const int bc = (lane & 3) * 2;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        if (SWIGLU) {
          // rows r and r + 8 of the tile are gate_j and up_j; the projection is a bf16 tensor in the reference
          const int j = wr * 8 + (lane >> 2);
          const float g0 = round_bf16(acc[nt][0]), g1 = round_bf16(acc[nt][1]);
          const float u0 = round_bf16(acc[nt][2]), u1 = round_bf16(acc[nt][3]);
          st[(nt * 8 + bc) * OUT + j] = __float2bfloat16_rn(g0 / (1.0f + expf(-g0)) * u0);
          st[(nt * 8 + bc + 1) * OUT + j] = __float2bfloat16_rn(g1 / (1.0f + expf(-g1)) * u1);
        } else {
          const int nr = wr * 16 + (lane >> 2);
          st[(nt * 8 + bc) * OUT + nr] = __float2bfloat16_rn(acc[nt][0]);
          st[(nt * 8 + bc + 1) * OUT + nr] = __float2bfloat16_rn(acc[nt][1]);
          st[(nt * 8 + bc) * OUT + nr + 8] = __float2bfloat16_rn(acc[nt][2]);
          st[(nt * 8 + bc + 1) * OUT + nr + 8] = __float2bfloat16_rn(acc[nt][3]);
        }
      }
    }
    __syncthreads();
    for (int i = tid; i < ROWS * (OUT / 8); i += SG_STD_THREADS) {
      const int r = i / (OUT / 8), c = i % (OUT / 8);
      const int n0 = rb * OUT + c * 8;
      if (r < p.m && n0 < p.n)  // N is a multiple of 8: a 16-byte chunk is inside or outside as a whole
        *reinterpret_cast<uint4*>(p.y + static_cast<int64_t>(r) * p.y_stride + n0) =
            *reinterpret_cast<const uint4*>(stage + (r * OUT + c * 8) * 2);
    }
  }
  if (ARGMAX) {
    // lanes that share lane % 4 hold the same batch columns: fold them, then the four row groups, then the CTAs
    unsigned long long* keybuf = reinterpret_cast<unsigned long long*>(part);  // [4 row groups][32 batch]
    if (kh == 0) {
#pragma unroll
      for (int c = 0; c < 2 * NT; ++c) {
        unsigned long long key = best_i[c] == 0xffffffffu ? 0ull : argmax_key(best_v[c], best_i[c]);
#pragma unroll
        for (int o = 4; o <= 16; o <<= 1) {
          const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
          key = other > key ? other : key;
        }
        if (lane < 4) keybuf[wr * SG_MAX_M + (c >> 1) * 8 + lane * 2 + (c & 1)] = key;
      }
    }
    __syncthreads();
    if (warp == 0) {
      if (lane < p.m && ok) {
        unsigned long long key = keybuf[lane];
#pragma unroll
        for (int w = 1; w < SG_WARPS; ++w) key = keybuf[w * SG_MAX_M + lane] > key ? keybuf[w * SG_MAX_M + lane] : key;
        atomicMax(p.keys + lane, key);
      }
      __threadfence();
      __syncwarp();
      int last = 0;
      if (lane == 0) last = (atomicAdd(p.counter, 1) == static_cast<int>(gridDim.x) - 1);
      last = __shfl_sync(0xffffffffu, last, 0);
      if (last) {  // every CTA's keys are in: unpack the ids and leave the workspace zero for the next launch
        __threadfence();
        if (lane < p.m) {
          const unsigned long long top = atomicExch(p.keys + lane, 0ull);
          p.ids[lane] = static_cast<int64_t>(0xffffffffu - static_cast<uint32_t>(top & 0xffffffffull));
        }
        if (lane == 0) *p.counter = 0;
      }
    }
  }
  if (!ok) {
    if (lane == 0) atomicExch(p.err, 1);
    // let this warp's copies in flight land before the shared memory goes away
    for (int s = 0; s < RING; ++s) mbar_wait_bounded(&bars[warp][s], 0, 1u << 12);
    for (int kt = 0; kt < k_tiles; ++kt) mbar_wait_bounded(&bar_x[kt], 0, 1u << 12);
  }
}

// ------------------------------------------------------------------------------------------------ wide-K form
// Projections back to the hidden size (out / o / down projection: N = hidden, K = 2048 .. 3584 and more) have few
// output rows and long ones.  A CTA owns 16 outputs (one MMA M tile) and its four warps split K: warp w streams the
// 4 KiB tiles kt = w, w + 4, ... of those 16 rows, accumulates its own [16 x 32] product and the four partial sums meet
// in shared memory (fixed order, so the result is deterministic).  X no longer fits next to the rings, so it is staged
// in chunks of at most 1024 k, double-buffered: the last warp to leave a chunk (a counter in shared memory, nobody
// waits) requests the chunk after the next into the buffer that just became free.
constexpr int WK_RING = 5;                // W tiles in flight per warp
constexpr int WK_CHUNK_MAX = 1024;        // k elements of X per staged chunk
constexpr int WK_ROWS = 16;               // outputs per CTA step
constexpr int WK_MAX_K = 16384;
constexpr int WK_X_PITCH_MAX = WK_CHUNK_MAX * 2 + 16;
constexpr int WK_SMEM = SG_WARPS * WK_RING * SG_TILE_BYTES + SG_WARPS * WK_ROWS * SG_MAX_M * 4 +
                        2 * SG_MAX_M * WK_X_PITCH_MAX + 1024;
static_assert(WK_SMEM <= 227 * 1024, "weight rings + two X chunks must fit the 227 KiB a CTA may use");

struct WideKParams {
  const __nv_bfloat16* x;  // [M, K]
  __nv_bfloat16* y;        // [M, N]
  int64_t x_stride, y_stride;
  int* err;
  int m, n, k, row_blocks, overlap, chunk_k, n_chunks;
  // pair-K form with the residual added: y = s = residual + X W^T, scaled = s (1 + gain), squares[m][row block] = sums of s^2; or null
  const __nv_bfloat16 *residual, *gain;
  int64_t res_stride;
  __nv_bfloat16* scaled;   // [M, N] contiguous
  float* squares;
  // ... or with S hyper-connected streams [M, S, N] in place of the residual: x_t <- sum_s mix[s, t] x_s + out[t] y with y = earlier parts + X W^T,
  // s = sum_t in[t] x_t, scaled = s gain gains[n]
  float* streams;
  const float *joint, *gains;   // [mix S*S | out S | in S | gain], [N] or null
  const __nv_bfloat16* parts;   // [n_parts][M, N] contiguous
  int s, n_parts;
};
constexpr int JOINT_STREAMS = 4;

__global__ void __launch_bounds__(SG_THREADS, 1)
skinny_gemm_widek_kernel(const __grid_constant__ WideKParams p, const __grid_constant__ CUtensorMap map_w) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ uint64_t bars[SG_WARPS][WK_RING];
  __shared__ uint64_t bar_x[2];
  __shared__ int x_left[2];  // warps that have left the chunk in buffer 0 / 1 (counts up, never reset)
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint8_t* ring = smem + warp * WK_RING * SG_TILE_BYTES;
  float* red = reinterpret_cast<float*>(smem + SG_WARPS * WK_RING * SG_TILE_BYTES);   // [4 warps][32 batch][16 rows]
  uint8_t* xs = reinterpret_cast<uint8_t*>(red) + SG_WARPS * WK_ROWS * SG_MAX_M * 4;  // [2][32][x_pitch]
  const int x_pitch = p.chunk_k * 2 + 16;
  const int x_buf_bytes = SG_MAX_M * x_pitch;
  const int k_tiles = p.k / SG_TILE_K, chunk_tiles = p.chunk_k / SG_TILE_K;

  if (tid == 0) {
    for (int w = 0; w < SG_WARPS; ++w)
      for (int s = 0; s < WK_RING; ++s) mbar_init(&bars[w][s], 1);
    mbar_init(&bar_x[0], 1);
    mbar_init(&bar_x[1], 1);
    x_left[0] = x_left[1] = 0;
    mbar_fence_init();
  }
  const int my_blocks = (p.row_blocks - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
  const int my_tiles = k_tiles > warp ? (k_tiles - warp + SG_WARPS - 1) / SG_WARPS : 0;  // per row block, this warp
  const int total_tiles = my_blocks * my_tiles;
  const int total_chunks = my_blocks * p.n_chunks;
  __syncthreads();
  auto issue = [&](int t) {  // lane 0: tile t of this warp = (row block t / my_tiles, k tile warp + 4 * (t % my_tiles))
    const int rb = blockIdx.x + (t / my_tiles) * gridDim.x, kt = warp + SG_WARPS * (t % my_tiles);
    const int slot = t % WK_RING;
    mbar_expect_tx(&bars[warp][slot], SG_TILE_BYTES);
    tma_load_3d(ring + slot * SG_TILE_BYTES, &map_w, 0, rb * WK_ROWS, kt * 2, &bars[warp][slot]);
  };
  // chunk q of this CTA's chunk stream (row block q / n_chunks, k range (q % n_chunks) * chunk_k ...) -> buffer q & 1
  auto stage_x = [&](int q) {  // a whole warp
    const int buf = q & 1, c = q % p.n_chunks;
    if (lane == 0) mbar_expect_tx(&bar_x[buf], static_cast<uint32_t>(p.m) * p.chunk_k * 2);
    __syncwarp();
    if (lane < p.m)
      bulk_g2s(xs + buf * x_buf_bytes + lane * x_pitch, p.x + static_cast<int64_t>(lane) * p.x_stride + c * p.chunk_k,
               p.chunk_k * 2, &bar_x[buf]);
  };
  if (p.overlap & OVERLAP_TRIGGER) pdl_trigger();
  if (lane == 0) {
    for (int t = 0; t < WK_RING && t < total_tiles; ++t) issue(t);  // weights: independent of the predecessor
  }
  pdl_wait();  // X is the predecessor's output
  for (int i = tid; i < 2 * (SG_MAX_M - p.m) * (p.chunk_k >> 3); i += SG_THREADS) {  // rows beyond M are zero
    const int per_buf = (SG_MAX_M - p.m) * (p.chunk_k >> 3);
    const int buf = i / per_buf, j = i % per_buf;
    const int r = p.m + j / (p.chunk_k >> 3), c = j % (p.chunk_k >> 3);
    *reinterpret_cast<uint4*>(xs + buf * x_buf_bytes + r * x_pitch + c * 16) = make_uint4(0, 0, 0, 0);
  }
  if (warp == 0) {
    stage_x(0);
    if (total_chunks > 1) stage_x(1);
  }
  __syncthreads();  // the zero rows are in place

  const int a_row = lane & 15, a_par = lane >> 4;
  const uint32_t b_lane = static_cast<uint32_t>(((lane & 7) + ((lane >> 4) << 3)) * x_pitch + ((lane >> 3) & 1) * 16);
  bool ok = true;
  int t = 0;
  // leave chunk q: the last of the four warps to do so requests chunk q + 2 into the buffer that is now free
  auto leave_chunk = [&](int q) {
    int last = 0;
    if (lane == 0) last = ((atomicAdd(&x_left[q & 1], 1) & (SG_WARPS - 1)) == SG_WARPS - 1);
    last = __shfl_sync(0xffffffffu, last, 0);
    if (last && q + 2 < total_chunks) stage_x(q + 2);
  };
  for (int blk = 0; blk < my_blocks; ++blk) {
    const int rb = blockIdx.x + blk * gridDim.x;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    int cur = -1;  // chunk (within the row block) whose X this warp is reading
    for (int kt = warp; kt < k_tiles; kt += SG_WARPS, ++t) {
      const int c = kt / chunk_tiles;
      while (cur < c) {  // move on to the chunk of this tile, leaving the ones in between
        if (cur >= 0) leave_chunk(blk * p.n_chunks + cur);
        ++cur;
      }
      const int q = blk * p.n_chunks + c;
      if (ok && !mbar_wait_bounded(&bar_x[q & 1], (q >> 1) & 1)) ok = false;
      const int slot = t % WK_RING;
      if (ok && !mbar_wait_bounded(&bars[warp][slot], (t / WK_RING) & 1)) ok = false;
      if (ok) {
        const uint32_t tile = smem_u32(ring + slot * SG_TILE_BYTES);
        const uint32_t xk0 = smem_u32(xs + (q & 1) * x_buf_bytes) + b_lane + ((kt - c * chunk_tiles) * SG_TILE_K) * 2;
#pragma unroll
        for (int ks = 0; ks < SG_TILE_K / 16; ++ks) {
          uint32_t a[4], b01[4], b23[4];
          const uint32_t a_off = (ks >> 2) * (16 * 128) + a_row * 128 + ((((ks & 3) * 2 + a_par) ^ (a_row & 7)) << 4);
          ldmatrix_x4(b01, xk0 + ks * 32);
          ldmatrix_x4(b23, xk0 + ks * 32 + 16 * x_pitch);
          ldmatrix_x4(a, tile + a_off);
          mma_bf16_16816(acc[0], a, b01[0], b01[1]);
          mma_bf16_16816(acc[1], a, b01[2], b01[3]);
          mma_bf16_16816(acc[2], a, b23[0], b23[1]);
          mma_bf16_16816(acc[3], a, b23[2], b23[3]);
        }
      }
      __syncwarp();  // every lane has read the tile: its slot can take the tile WK_RING ahead
      if (ok && lane == 0 && t + WK_RING < total_tiles) issue(t + WK_RING);
    }
    while (cur < p.n_chunks) {  // leave the remaining chunks of this row block (also those this warp had no tile in)
      if (cur >= 0) leave_chunk(blk * p.n_chunks + cur);
      ++cur;
    }
    // ---- the four partial [16 x 32] sums meet in shared memory: red[warp][batch][row]
    {
      float* mine = red + warp * (WK_ROWS * SG_MAX_M);
      const int r0 = lane >> 2, bc = (lane & 3) * 2;
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        mine[(nt * 8 + bc) * WK_ROWS + r0] = acc[nt][0];
        mine[(nt * 8 + bc + 1) * WK_ROWS + r0] = acc[nt][1];
        mine[(nt * 8 + bc) * WK_ROWS + r0 + 8] = acc[nt][2];
        mine[(nt * 8 + bc + 1) * WK_ROWS + r0 + 8] = acc[nt][3];
      }
    }
    __syncthreads();
    {
      // thread -> batch row tid / 4, outputs (tid % 4) * 4 .. + 4: one 8-byte store
      const int b = tid >> 2, r = (tid & 3) * 4;
      float o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int idx = b * WK_ROWS + r + j;
        o[j] = ((red[idx] + red[WK_ROWS * SG_MAX_M + idx]) + red[2 * WK_ROWS * SG_MAX_M + idx]) +
               red[3 * WK_ROWS * SG_MAX_M + idx];
      }
      const int n0 = rb * WK_ROWS + r;
      if (b < p.m && n0 < p.n)  // N is a multiple of 8 and r of 4: the four outputs are inside or outside together
        *reinterpret_cast<uint2*>(p.y + static_cast<int64_t>(b) * p.y_stride + n0) =
            make_uint2(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]));
    }
    __syncthreads();  // red is free for the next row block
  }
  if (!ok) {
    if (lane == 0) atomicExch(p.err, 1);
    // let this warp's copies in flight land before the shared memory goes away
    for (int s = 0; s < WK_RING; ++s) mbar_wait_bounded(&bars[warp][s], 0, 1u << 12);
    if (warp == 0) {
      mbar_wait_bounded(&bar_x[0], 0, 1u << 12);
      mbar_wait_bounded(&bar_x[1], 0, 1u << 12);
    }
  }
}

// ------------------------------------------------------------------------------------------------ pair-K form
// The same 16-outputs-per-step decomposition for K <= 4096, on a cluster of two CTAs that take one half of K each: twice
// as many SMs stream W, a CTA stages only its half of X -- once, whole, so there is no chunk pipeline -- and the two
// partial [16 x 32] sums meet through distributed shared memory (rank 1 stores its sum into rank 0's shared memory,
// one cluster barrier, rank 0 adds, rounds and writes).  No cluster multicast is used; every CTA loads its own tiles.
constexpr int PK_RING = 4;                 // W tiles in flight per warp: all of a row block (a decode step of one sequence 597 us with three, 587 with four)
constexpr int PK_MAX_K = 4096;
constexpr int pairk_smem(int nt, int k) {  // rings, sums of the warps and the peer, half of X
  return SG_WARPS * PK_RING * SG_TILE_BYTES + (SG_WARPS + 1) * WK_ROWS * nt * 8 * 4 + nt * 8 * k + 2048;
}
static_assert(pairk_smem(4, PK_MAX_K) <= 227 * 1024, "weight rings + half of X must fit the 227 KiB a CTA may use");

// END: what becomes of the product: 0 the output, 1 joined with a residual, 2 with hyper-connected streams (one kernel that decided when it
// ran cost a decode step of 32 sequences 4 us)
template <int NT, int END>
__global__ void __launch_bounds__(SG_THREADS, 1)
skinny_gemm_pairk_kernel(const __grid_constant__ WideKParams p, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  constexpr int ROWS = NT * 8;
  __shared__ uint64_t bars[SG_WARPS][PK_RING];
  __shared__ uint64_t bar_x[PK_MAX_K / 2 / SG_TILE_K];  // one per k tile
  __shared__ float joint[JOINT_STREAMS * JOINT_STREAMS + 2 * JOINT_STREAMS + 1];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  uint8_t* ring = smem + warp * PK_RING * SG_TILE_BYTES;
  float* red = reinterpret_cast<float*>(smem + SG_WARPS * PK_RING * SG_TILE_BYTES);  // [4 warps + peer][ROWS][16]
  float* peer = red + SG_WARPS * WK_ROWS * ROWS;                                 // written by rank 1 into rank 0
  constexpr int X_TILE = ROWS * SG_TILE_K * 2;
  // this CTA's half of X, tile by tile; the swizzle counts from 1024-byte boundaries
  uint8_t* xs = smem + (SG_WARPS * PK_RING * SG_TILE_BYTES + (SG_WARPS + 1) * WK_ROWS * ROWS * 4 + 1023) / 1024 * 1024;
  const int half_k = p.k >> 1;
  const int half_tiles = half_k / SG_TILE_K;

  if (tid == 0) {
    for (int w = 0; w < SG_WARPS; ++w)
      for (int s = 0; s < PK_RING; ++s) mbar_init(&bars[w][s], 1);
    for (int i = 0; i < PK_MAX_K / 2 / SG_TILE_K; ++i) mbar_init(&bar_x[i], 1);
    mbar_fence_init();
  }
  const int my_blocks = (p.row_blocks - pair + pairs - 1) / pairs;
  const int my_tiles = half_tiles > warp ? (half_tiles - warp + SG_WARPS - 1) / SG_WARPS : 0;  // per row block, this warp
  const int total_tiles = my_blocks * my_tiles;
  __syncthreads();
  cluster_started();
  auto issue = [&](int t) {  // lane 0: tile t of this warp
    const int rb = pair + (t / my_tiles) * pairs, kt = static_cast<int>(rank) * half_tiles + warp + SG_WARPS * (t % my_tiles);
    const int slot = t % PK_RING;
    mbar_expect_tx(&bars[warp][slot], SG_TILE_BYTES);
    tma_load_3d(ring + slot * SG_TILE_BYTES, &map_w, 0, rb * WK_ROWS, kt * 2, &bars[warp][slot]);
  };
  if (p.overlap & OVERLAP_TRIGGER) pdl_trigger();
  if (lane == 0) {
    for (int t = 0; t < PK_RING && t < total_tiles; ++t) issue(t);  // weights: independent of the predecessor
  }
  // thread -> batch row tid / 4, outputs (tid % 4) * 4 .. + 4 of a row block (N is a multiple of 8 and r of 4: inside or outside together)
  constexpr bool joins = END > 0, hyper = END == 2;
  const int b = tid >> 2, r = (tid & 3) * 4;
  const auto writes = [&](int n0) { return rank == 0 && b < p.m && n0 < p.n; };
  uint2 res = {}, gain = {};
  float4 old[JOINT_STREAMS], gains = make_float4(1.f, 1.f, 1.f, 1.f);
  if (joins && !hyper && writes(pair * WK_ROWS + r)) gain = *reinterpret_cast<const uint2*>(p.gain + pair * WK_ROWS + r);
  if (hyper && tid < p.s * p.s + 2 * p.s + 1) joint[tid] = p.joint[tid];
  pdl_wait();  // X is the predecessor's output
  if (lane == 0) {
    for (int kl = warp; kl < half_tiles; kl += SG_WARPS) {
      mbar_expect_tx(&bar_x[kl], X_TILE);
      tma_load_3d(xs + kl * X_TILE, &map_x, 0, 0, (static_cast<int>(rank) * half_tiles + kl) * 2, &bar_x[kl]);
    }
  }
  // what the row is joined with, on its way under the products
  const auto fetch = [&](int n0) {
    if (!joins || !writes(n0)) return;
    if (!hyper) {
      res = *reinterpret_cast<const uint2*>(p.residual + b * p.res_stride + n0);
      return;
    }
#pragma unroll
    for (int i = 0; i < JOINT_STREAMS; ++i)
      if (i < p.s) old[i] = *reinterpret_cast<const float4*>(p.streams + (static_cast<int64_t>(b) * p.s + i) * p.n + n0);
    if (p.gains != nullptr) gains = *reinterpret_cast<const float4*>(p.gains + n0);
  };
  fetch(pair * WK_ROWS + r);
  __syncthreads();
  cluster_all_started();  // here, where X is on its way, and not in front of the store to the peer, where everybody waits for it
  bool ok = true;

  const int a_row = lane & 15, a_par = lane >> 4;
  const uint32_t xs_base = smem_u32(xs) + StepProducts<NT>::lane_offset(lane);
  const uint32_t xj[4] = {xs_base, xs_base ^ 32, xs_base ^ 64, xs_base ^ 96};
  const auto a_offset = [&](int ks) -> uint32_t { return (ks >> 2) * (16 * 128) + a_row * 128 + ((((ks & 3) * 2 + a_par) ^ (a_row & 7)) << 4); };
  const uint32_t peer_remote = cluster_map(smem_u32(peer), 0);
  int t = 0;
  for (int blk = 0; blk < my_blocks; ++blk) {
    const int rb = pair + blk * pairs;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    const int n0 = rb * WK_ROWS + r;
    if (blk > 0) {
      fetch(n0);
      if (joins && !hyper && writes(n0)) gain = *reinterpret_cast<const uint2*>(p.gain + n0);
    }
    for (int kl = warp; kl < half_tiles; kl += SG_WARPS, ++t) {
      const int slot = t % PK_RING;
      if (ok && !mbar_wait_bounded(&bars[warp][slot], (t / PK_RING) & 1)) ok = false;
      if (blk == 0 && ok && !mbar_wait_bounded(&bar_x[kl], 0)) ok = false;
      if (ok) {
        uint32_t b[8];
        tile_steps<NT, 0>(acc, b, smem_u32(ring + slot * SG_TILE_BYTES), xj, kl * X_TILE, a_offset);
      }
      __syncwarp();  // every lane has read the tile: its slot can take the tile PK_RING ahead
      if (ok && lane == 0 && t + PK_RING < total_tiles) issue(t + PK_RING);
    }
    // ---- the warps' partial [16 x 32] sums meet in shared memory: red[warp][batch][row]
    join_steps<NT>(acc);
    {
      float* mine = red + warp * (WK_ROWS * ROWS);
      const int r0 = lane >> 2, bc = (lane & 3) * 2;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        mine[(nt * 8 + bc) * WK_ROWS + r0] = acc[nt][0];
        mine[(nt * 8 + bc + 1) * WK_ROWS + r0] = acc[nt][1];
        mine[(nt * 8 + bc) * WK_ROWS + r0 + 8] = acc[nt][2];
        mine[(nt * 8 + bc + 1) * WK_ROWS + r0 + 8] = acc[nt][3];
      }
    }
    __syncthreads();
    const bool mine = NT == 4 || b < ROWS;
    float o[4] = {};
    if (mine) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int idx = b * WK_ROWS + r + j;
        o[j] = ((red[idx] + red[WK_ROWS * ROWS + idx]) + red[2 * WK_ROWS * ROWS + idx]) + red[3 * WK_ROWS * ROWS + idx];
      }
      if (rank == 1) st_cluster_f32x4(peer_remote + (b * WK_ROWS + r) * 4, o[0], o[1], o[2], o[3]);
    }
    cluster_sync();  // rank 1's sum is in rank 0's shared memory; red is free again in both CTAs
    if (rank == 0 && mine) {
      const float4 other = *reinterpret_cast<const float4*>(peer + b * WK_ROWS + r);
      uint2 y = make_uint2(pack_bf16(o[0] + other.x, o[1] + other.y), pack_bf16(o[2] + other.z, o[3] + other.w));
      if constexpr (hyper) {
        float v[4] = {bf16_lo(y.x), bf16_hi(y.x), bf16_lo(y.y), bf16_hi(y.y)}, u[4] = {};
        if (writes(n0)) {
          if (p.n_parts > 0) {                          // the parts in their order, this one last
            float sum[4] = {};
            for (int i = 0; i < p.n_parts; ++i) {
              const uint2 part = *reinterpret_cast<const uint2*>(p.parts + (static_cast<int64_t>(i) * p.m + b) * p.n + n0);
              sum[0] += bf16_lo(part.x), sum[1] += bf16_hi(part.x), sum[2] += bf16_lo(part.y), sum[3] += bf16_hi(part.y);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] += sum[j];
          }
          const float *out = joint + p.s * p.s, *in = out + p.s;
#pragma unroll
          for (int st = 0; st < JOINT_STREAMS; ++st)
            if (st < p.s) {
              float a[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) a[j] = out[st] * v[j];
#pragma unroll
              for (int i = 0; i < JOINT_STREAMS; ++i)
                if (i < p.s) {
                  const float m = joint[i * p.s + st];
                  a[0] = fmaf(m, old[i].x, a[0]), a[1] = fmaf(m, old[i].y, a[1]), a[2] = fmaf(m, old[i].z, a[2]), a[3] = fmaf(m, old[i].w, a[3]);
                }
              *reinterpret_cast<float4*>(p.streams + (static_cast<int64_t>(b) * p.s + st) * p.n + n0) = make_float4(a[0], a[1], a[2], a[3]);
#pragma unroll
              for (int j = 0; j < 4; ++j) u[j] = fmaf(in[st], a[j], u[j]);
            }
          const float g = in[p.s];
          *reinterpret_cast<uint2*>(p.scaled + static_cast<int64_t>(b) * p.n + n0) =
              make_uint2(pack_bf16(u[0] * g * gains.x, u[1] * g * gains.y), pack_bf16(u[2] * g * gains.z, u[3] * g * gains.w));
        }
        float ss = u[0] * u[0] + u[1] * u[1] + u[2] * u[2] + u[3] * u[3];
        ss += __shfl_xor_sync(0xffffffffu, ss, 1);
        ss += __shfl_xor_sync(0xffffffffu, ss, 2);
        if (r == 0 && b < p.m) p.squares[b * p.row_blocks + rb] = ss;
      } else if constexpr (joins) {
        // product and sum are bf16 tensors in the reference
        const float v0 = round_bf16(bf16_lo(y.x) + bf16_lo(res.x)), v1 = round_bf16(bf16_hi(y.x) + bf16_hi(res.x));
        const float v2 = round_bf16(bf16_lo(y.y) + bf16_lo(res.y)), v3 = round_bf16(bf16_hi(y.y) + bf16_hi(res.y));
        y = make_uint2(pack_bf16(v0, v1), pack_bf16(v2, v3));
        if (writes(n0))
          *reinterpret_cast<uint2*>(p.scaled + static_cast<int64_t>(b) * p.n + n0) =
              make_uint2(pack_bf16(v0 * (1.f + bf16_lo(gain.x)), v1 * (1.f + bf16_hi(gain.x))),
                         pack_bf16(v2 * (1.f + bf16_lo(gain.y)), v3 * (1.f + bf16_hi(gain.y))));
        float ss = writes(n0) ? fmaf(v0, v0, fmaf(v1, v1, fmaf(v2, v2, v3 * v3))) : 0.f;
        ss += __shfl_xor_sync(0xffffffffu, ss, 1);
        ss += __shfl_xor_sync(0xffffffffu, ss, 2);
        if (r == 0 && b < p.m) p.squares[b * p.row_blocks + rb] = ss;
      }
      if (!hyper && writes(n0)) *reinterpret_cast<uint2*>(p.y + static_cast<int64_t>(b) * p.y_stride + n0) = y;
    }
    if (blk + 1 < my_blocks) cluster_sync();  // rank 0 has read `peer` before rank 1 writes the next sum
  }
  if (!ok) {
    if (lane == 0) atomicExch(p.err, 1);
    // let this warp's copies in flight land before the shared memory goes away
    for (int s = 0; s < PK_RING; ++s) mbar_wait_bounded(&bars[warp][s], 0, 1u << 12);
    for (int kl = 0; kl < half_tiles; ++kl) mbar_wait_bounded(&bar_x[kl], 0, 1u << 12);
  }
}

// Shared by all host threads: searched and filled under a mutex, the map is copied out.
static bool cache_weight_map(const void* base, int64_t n, int64_t k, int64_t stride, int box_rows, CUtensorMap* out) {
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  struct Entry {
    const void* base;
    int64_t n, k, stride;
    int dev, box_rows;
    CUtensorMap map;
  };
  constexpr int N = 128;  // a model has a fixed set of weight matrices
  static Entry entries[N];
  static int used = 0, next = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  for (int i = 0; i < used; ++i)
    if (entries[i].base == base && entries[i].n == n && entries[i].k == k && entries[i].stride == stride && entries[i].dev == dev &&
        entries[i].box_rows == box_rows) {
      *out = entries[i].map;
      return true;
    }
  Entry& e = entries[next];
  e.base = nullptr;  // not a valid entry while it is being rewritten
  if (!encode_tile_map(&e.map, base, static_cast<uint64_t>(n), static_cast<uint64_t>(k), static_cast<uint64_t>(stride) * 2, box_rows, 2))
    return false;
  e.base = base;
  e.n = n;
  e.k = k;
  e.stride = stride;
  e.dev = dev;
  e.box_rows = box_rows;
  next = (next + 1) % N;
  if (used < N) ++used;
  *out = e.map;
  return true;
}

}  // namespace b200

using namespace b200;

// X [m, k] as boxes of `rows` rows and 128 k
static bool encode_x_map(CUtensorMap* map, const void* x, int m, int k, int64_t stride, int rows) {
  return encode_tile_map(map, x, static_cast<uint64_t>(m), static_cast<uint64_t>(k), static_cast<uint64_t>(m > 1 ? stride : k) * 2, rows, 2);
}

template <bool SWIGLU, bool ARGMAX, int NT>
static int launch_skinny_rows(SkinnyGemmParams p, const CUtensorMap& map, cudaStream_t stream, const char* what) {
  CUtensorMap map_x = {};
  if (!encode_x_map(&map_x, p.x, p.m, p.k, p.x_stride, NT * 8)) return fail(ERR_RUNTIME, "%s: cannot encode the tensor map of x", what);
  constexpr int smem_max = skinny_smem(NT, SG_MAX_K);
  static_assert(smem_max <= 227 * 1024, "weight rings + X staging must fit the 227 KiB a CTA may use");
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    if (cudaFuncSetAttribute(skinny_gemm_kernel<SWIGLU, ARGMAX, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max) !=
        cudaSuccess)
      return fail(ERR_RUNTIME, "%s: cannot raise dynamic shared memory to %d", what, smem_max);
    configured[dev] = true;
  }
  const int sms = sm_count();
  if (launch_pdl((p.overlap & OVERLAP_START) != 0, skinny_gemm_kernel<SWIGLU, ARGMAX, NT>, dim3(p.row_blocks < sms ? p.row_blocks : sms),
                 dim3(SG_STD_THREADS), skinny_smem(NT, p.k), stream, p, map, map_x) != cudaSuccess)
    return fail(ERR_LAUNCH, "%s: %s", what, cudaGetErrorString(cudaGetLastError()));
  return check_launch(what);
}

template <bool SWIGLU, bool ARGMAX = false>
static int launch_skinny(SkinnyGemmParams p, const void* weight, int64_t w_stride, int w_rows, cudaStream_t stream, const char* what) {
  CUtensorMap map;
  if (!cache_weight_map(weight, w_rows, p.k, w_stride, SWIGLU ? 8 : 16, &map)) return fail(ERR_RUNTIME, "%s: cannot encode the weight tensor map", what);
  p.err = wait_timeout_flag();
  if (!p.err) return fail(ERR_RUNTIME, "%s: no error flag", what);
  constexpr int out_per_cta = SWIGLU ? 8 * SG_WARPS : SG_ROWS;
  p.row_blocks = (p.n + out_per_cta - 1) / out_per_cta;
  // as few groups of eight rows as hold the batch
  if (p.m <= 8) return launch_skinny_rows<SWIGLU, ARGMAX, 1>(p, map, stream, what);
  if (p.m <= 16) return launch_skinny_rows<SWIGLU, ARGMAX, 2>(p, map, stream, what);
  return launch_skinny_rows<SWIGLU, ARGMAX, 4>(p, map, stream, what);
}

// Chunking of K for the wide-K form: the fewest equal chunks of whole 128-k tiles that are at most WK_CHUNK_MAX long.
static bool widek_chunks(int k, int* chunk_k, int* n_chunks) {
  if (k <= 0 || k % SG_TILE_K != 0 || k > WK_MAX_K) return false;
  const int n = (k + WK_CHUNK_MAX - 1) / WK_CHUNK_MAX;
  if (k % (n * SG_TILE_K) != 0) return false;
  *chunk_k = k / n;
  *n_chunks = n;
  return true;
}

static int launch_widek(WideKParams p, const void* weight, int64_t w_stride, cudaStream_t stream) {
  const char* what = "skinny_gemm";
  CUtensorMap map;
  if (!cache_weight_map(weight, p.n, p.k, w_stride, 16, &map)) return fail(ERR_RUNTIME, "%s: cannot encode the weight tensor map", what);
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    if (cudaFuncSetAttribute(skinny_gemm_widek_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, WK_SMEM) != cudaSuccess)
      return fail(ERR_RUNTIME, "%s: cannot raise dynamic shared memory to %d", what, WK_SMEM);
    configured[dev] = true;
  }
  p.err = wait_timeout_flag();
  if (!p.err) return fail(ERR_RUNTIME, "%s: no error flag", what);
  p.row_blocks = (p.n + WK_ROWS - 1) / WK_ROWS;
  int grid = p.row_blocks;
  const int sms = sm_count();
  if (grid > sms) grid = sms;
  const int dyn = SG_WARPS * WK_RING * SG_TILE_BYTES + SG_WARPS * WK_ROWS * SG_MAX_M * 4 +
                  2 * SG_MAX_M * (p.chunk_k * 2 + 16) + 1024;
  if (launch_pdl((p.overlap & OVERLAP_START) != 0, skinny_gemm_widek_kernel, dim3(grid), dim3(SG_THREADS), dyn, stream, p,
                 map) != cudaSuccess)
    return fail(ERR_LAUNCH, "%s: %s", what, cudaGetErrorString(cudaGetLastError()));
  return check_launch(what);
}

template <int NT, int END>
static int launch_pairk_rows(WideKParams p, const CUtensorMap& map, cudaStream_t stream) {
  const char* what = "skinny_gemm";
  CUtensorMap map_x = {};
  if (!encode_x_map(&map_x, p.x, p.m, p.k, p.x_stride, NT * 8)) return fail(ERR_RUNTIME, "%s: cannot encode the tensor map of x", what);
  constexpr int smem_max = pairk_smem(NT, PK_MAX_K);
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    if (cudaFuncSetAttribute(skinny_gemm_pairk_kernel<NT, END>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max) != cudaSuccess)
      return fail(ERR_RUNTIME, "%s: cannot raise dynamic shared memory to %d", what, smem_max);
    configured[dev] = true;
  }
  const int sms = sm_count(), pairs = p.row_blocks < sms / 2 ? p.row_blocks : sms / 2;
  if (launch_pdl_cluster((p.overlap & OVERLAP_START) != 0, 2, skinny_gemm_pairk_kernel<NT, END>, dim3(2 * pairs), dim3(SG_THREADS),
                         pairk_smem(NT, p.k), stream, p, map, map_x) != cudaSuccess)
    return fail(ERR_LAUNCH, "%s: %s", what, cudaGetErrorString(cudaGetLastError()));
  return check_launch(what);
}

template <int END>
static int launch_pairk(WideKParams p, const void* weight, int64_t w_stride, cudaStream_t stream) {
  const char* what = "skinny_gemm";
  CUtensorMap map;
  if (!cache_weight_map(weight, p.n, p.k, w_stride, 16, &map)) return fail(ERR_RUNTIME, "%s: cannot encode the weight tensor map", what);
  p.err = wait_timeout_flag();
  if (!p.err) return fail(ERR_RUNTIME, "%s: no error flag", what);
  p.row_blocks = (p.n + WK_ROWS - 1) / WK_ROWS;
  if (p.m <= 8) return launch_pairk_rows<1, END>(p, map, stream);
  if (p.m <= 16) return launch_pairk_rows<2, END>(p, map, stream);
  return launch_pairk_rows<4, END>(p, map, stream);
}

static int check_skinny_shape(const char* what, int m, int n, int k) {
  B200_REQUIRE(m > 0 && m <= SG_MAX_M, "%s: M must be in [1, %d] (got %d)", what, SG_MAX_M, m);
  B200_REQUIRE(n > 0 && n % 8 == 0 && k >= SG_TILE_K && k % SG_TILE_K == 0 && k <= SG_MAX_K,
               "%s: N must be a multiple of 8, K a multiple of %d up to %d (got N=%d K=%d)", what, SG_TILE_K, SG_MAX_K, n,
               k);
  return OK;
}

extern "C" int b200_skinny_gemm_join(const void* x, int64_t x_stride, const void* weight, const void* residual, int64_t res_stride,
                                     const void* gain, void* sum, void* scaled, float* squares, int32_t m, int32_t n, int32_t k,
                                     int32_t overlap, b200_stream_t stream) {
  B200_REQUIRE(m > 0 && m <= SG_MAX_M && n > 0 && n % WK_ROWS == 0 && k > SG_MAX_K && k <= PK_MAX_K && k % (2 * SG_TILE_K) == 0,
               "skinny_gemm_join: M must be in [1, %d], N a multiple of %d, K in (%d, %d] a multiple of %d (got M=%d N=%d K=%d)", SG_MAX_M,
               WK_ROWS, SG_MAX_K, PK_MAX_K, 2 * SG_TILE_K, m, n, k);
  B200_REQUIRE(aligned16(x) && aligned16(weight) && aligned16(residual) && aligned16(gain) && aligned16(sum) && aligned16(scaled) &&
                   squares != nullptr && x_stride % 8 == 0 && res_stride % 8 == 0,
               "skinny_gemm_join: pointers must be 16-byte aligned, row strides multiples of 8 elements");
  WideKParams p = {};
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.y = static_cast<__nv_bfloat16*>(sum);
  p.x_stride = x_stride;
  p.y_stride = n;
  p.m = m;
  p.n = n;
  p.k = k;
  p.overlap = overlap;
  p.residual = static_cast<const __nv_bfloat16*>(residual);
  p.res_stride = res_stride;
  p.gain = static_cast<const __nv_bfloat16*>(gain);
  p.scaled = static_cast<__nv_bfloat16*>(scaled);
  p.squares = squares;
  return launch_pairk<1>(p, weight, k, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int b200_skinny_gemm_hyper_join(const void* x, int64_t x_stride, const void* weight, int64_t w_stride, float* streams, const float* joint,
                                           const float* gains, const void* parts, int32_t n_parts, void* scaled, float* squares, int32_t m,
                                           int32_t n, int32_t k, int32_t s, int32_t overlap, b200_stream_t stream) {
  B200_REQUIRE(m > 0 && m <= SG_MAX_M && n > 0 && n % WK_ROWS == 0 && k > SG_MAX_K && k <= PK_MAX_K && k % (2 * SG_TILE_K) == 0,
               "skinny_gemm_hyper_join: M must be in [1, %d], N a multiple of %d, K in (%d, %d] a multiple of %d (got M=%d N=%d K=%d)", SG_MAX_M,
               WK_ROWS, SG_MAX_K, PK_MAX_K, 2 * SG_TILE_K, m, n, k);
  B200_REQUIRE(s > 0 && s <= JOINT_STREAMS && n_parts >= 0 && (n_parts == 0 || aligned16(parts)), "skinny_gemm_hyper_join: 1 to %d streams (got %d)",
               JOINT_STREAMS, s);
  B200_REQUIRE(aligned16(x) && aligned16(weight) && aligned16(streams) && aligned16(scaled) && joint != nullptr && squares != nullptr &&
                   (gains == nullptr || aligned16(gains)) && x_stride % 8 == 0 && w_stride >= k && w_stride % 8 == 0,
               "skinny_gemm_hyper_join: pointers must be 16-byte aligned, row strides multiples of 8 elements");
  WideKParams p = {};
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.x_stride = x_stride;
  p.m = m;
  p.n = n;
  p.k = k;
  p.overlap = overlap;
  p.scaled = static_cast<__nv_bfloat16*>(scaled);
  p.squares = squares;
  p.streams = streams;
  p.joint = joint;
  p.gains = gains;
  p.parts = static_cast<const __nv_bfloat16*>(parts);
  p.s = s;
  p.n_parts = n_parts;
  return launch_pairk<2>(p, weight, w_stride, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int b200_skinny_gemm_part(const void* x, int64_t x_stride, const void* weight, int64_t w_stride, void* y,
                                     int64_t y_stride, int32_t m, int32_t n, int32_t k, int32_t overlap, b200_stream_t stream) {
  B200_REQUIRE(w_stride >= k && w_stride % 8 == 0, "skinny_gemm: weight rows must be whole 16-byte groups apart");
  B200_REQUIRE(aligned16(x) && aligned16(weight) && aligned16(y) && x_stride % 8 == 0 && y_stride % 8 == 0,
               "skinny_gemm: pointers must be 16-byte aligned, row strides multiples of 8 elements");
  if (k > SG_MAX_K) {  // long rows: K split over the warps of a CTA, X staged in chunks
    WideKParams wp = {};
    B200_REQUIRE(m > 0 && m <= SG_MAX_M && n > 0 && n % 8 == 0 && widek_chunks(k, &wp.chunk_k, &wp.n_chunks),
                 "skinny_gemm: M must be in [1, %d], N a multiple of 8, K > %d a multiple of 128 that splits into equal "
                 "chunks of whole tiles of at most %d (got M=%d N=%d K=%d)", SG_MAX_M, SG_MAX_K, WK_CHUNK_MAX, m, n, k);
    wp.x = static_cast<const __nv_bfloat16*>(x);
    wp.y = static_cast<__nv_bfloat16*>(y);
    wp.x_stride = x_stride;
    wp.y_stride = y_stride;
    wp.m = m;
    wp.n = n;
    wp.k = k;
    wp.overlap = overlap;
    if (k <= PK_MAX_K && k % (2 * SG_TILE_K) == 0) return launch_pairk<0>(wp, weight, w_stride, reinterpret_cast<cudaStream_t>(stream));
    return launch_widek(wp, weight, w_stride, reinterpret_cast<cudaStream_t>(stream));
  }
  int rc = check_skinny_shape("skinny_gemm", m, n, k);
  if (rc != OK) return rc;
  SkinnyGemmParams p = {};
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.y = static_cast<__nv_bfloat16*>(y);
  p.x_stride = x_stride;
  p.y_stride = y_stride;
  p.m = m;
  p.n = n;
  p.k = k;
  p.overlap = overlap;
  return launch_skinny<false>(p, weight, w_stride, n, reinterpret_cast<cudaStream_t>(stream), "skinny_gemm");
}

extern "C" int b200_skinny_gemm(const void* x, int64_t x_stride, const void* weight, void* y, int64_t y_stride, int32_t m,
                                int32_t n, int32_t k, int32_t overlap, b200_stream_t stream) {
  return b200_skinny_gemm_part(x, x_stride, weight, k, y, y_stride, m, n, k, overlap, stream);
}

extern "C" int b200_skinny_gemm_swiglu(const void* x, int64_t x_stride, const void* weight, void* y, int64_t y_stride,
                                       int32_t m, int32_t intermediate, int32_t k, int32_t overlap,
                                       b200_stream_t stream) {
  int rc = check_skinny_shape("skinny_gemm_swiglu", m, intermediate, k);
  if (rc != OK) return rc;
  B200_REQUIRE(aligned16(x) && aligned16(weight) && aligned16(y) && x_stride % 8 == 0 && y_stride % 8 == 0,
               "skinny_gemm_swiglu: pointers must be 16-byte aligned, row strides multiples of 8 elements");
  SkinnyGemmParams p = {};
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.y = static_cast<__nv_bfloat16*>(y);
  p.x_stride = x_stride;
  p.y_stride = y_stride;
  p.m = m;
  p.n = intermediate;
  p.k = k;
  p.overlap = overlap;
  p.up_row0 = intermediate;
  return launch_skinny<true>(p, weight, k, 2 * intermediate, reinterpret_cast<cudaStream_t>(stream), "skinny_gemm_swiglu");
}

extern "C" int b200_skinny_gemm_normed(const void* x, const float* squares, const void* weight, void* y, int64_t y_stride, int32_t m,
                                       int32_t n, int32_t k, int32_t true_k, float eps, int32_t swiglu, int32_t overlap,
                                       b200_stream_t stream) {
  int rc = check_skinny_shape("skinny_gemm_normed", m, n, k);
  if (rc != OK) return rc;
  B200_REQUIRE(true_k > 0 && true_k <= k, "skinny_gemm_normed: the mean over %d of %d columns", true_k, k);
  B200_REQUIRE(aligned16(x) && aligned16(weight) && aligned16(y) && squares != nullptr && y_stride % 8 == 0,
               "skinny_gemm_normed: pointers must be 16-byte aligned, the row stride of y a multiple of 8 elements");
  SkinnyGemmParams p = {};
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.y = static_cast<__nv_bfloat16*>(y);
  p.x_stride = k;
  p.y_stride = y_stride;
  p.m = m;
  p.n = n;
  p.k = k;
  p.overlap = overlap;
  p.squares = squares;
  p.eps = eps;
  p.true_k = true_k;
  p.up_row0 = n;
  if (swiglu) return launch_skinny<true>(p, weight, k, 2 * n, reinterpret_cast<cudaStream_t>(stream), "skinny_gemm_normed");
  return launch_skinny<false>(p, weight, k, n, reinterpret_cast<cudaStream_t>(stream), "skinny_gemm_normed");
}

extern "C" int b200_lm_head_argmax(const void* x, int64_t x_stride, const void* weight, int64_t* ids, void* workspace,
                                   int32_t m, int32_t n, int32_t k, int32_t overlap, b200_stream_t stream) {
  int rc = check_skinny_shape("lm_head_argmax", m, n, k);
  if (rc != OK) return rc;
  B200_REQUIRE(aligned16(x) && aligned16(weight) && x_stride % 8 == 0 && ids != nullptr && workspace != nullptr &&
                   (reinterpret_cast<uintptr_t>(workspace) % 8 == 0),
               "lm_head_argmax: x / weight must be 16-byte aligned, the x row stride a multiple of 8, the workspace "
               "8-byte aligned");
  SkinnyGemmParams p = {};
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.x_stride = x_stride;
  p.m = m;
  p.n = n;
  p.k = k;
  p.overlap = overlap;
  p.ids = ids;
  p.keys = static_cast<unsigned long long*>(workspace);  // the layout of b200_argmax_rows: 1024 keys, then counters
  p.counter = reinterpret_cast<int*>(p.keys + 1024);
  return launch_skinny<false, true>(p, weight, k, n, reinterpret_cast<cudaStream_t>(stream), "lm_head_argmax");
}
