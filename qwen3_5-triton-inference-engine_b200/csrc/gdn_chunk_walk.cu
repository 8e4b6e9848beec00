// Gated-DeltaNet chunk-64 prefill of a packed batch in two launches: what a chunk needs of itself alone, all chunks at once,
// and then a walk over every sequence's chunks with the state in registers.  Per chunk (G = cumsum(g) inside it, S the state
// that enters, b = beta; triton_kernels/gdn_recurrent_prefill.py:248-396, :404-537, :563-690 as one function):
//   prep   L[t,i] = b_t e^(G_t - G_i) <k_t,k_i> (i < t),  P = (I + L)^-1 diag(b),  A[t,i] = e^(G_t - G_i) <q_t,k_i> (i <= t)
//   walk   R = v - e^G (k S),  delta = P R,  o = e^G (q S) + A delta,  S <- e^(G_63) S + k^T (e^(G_63 - G) delta)
// The walk runs transposed, with the 16 value columns of a warp as the rows of m16n8k16: S^T [16 x 128] stays in accumulators,
// and an accumulator pair of one product is the left operand of the next (S -> k S, q S; R -> delta; delta -> A delta, S), so
// no value leaves the registers between products and warps never wait for one another inside a chunk.  P and A arrive as
// right-operand fragments: a lane's two registers of an 8 x 16 tile, high and low parts, are 16 consecutive bytes.
// The workspace is at most 1 GiB: where all slots would take more, the two launches go through a window of them at a time, and
// the states wait in device memory in between (fp32, so that the results are the same bits).
// Precision: q, k, v are exact bf16 operands; fp32 operands (S, R, delta, P, A) are bf16 pairs hi + lo with the products
// hi hi + hi lo + lo hi (hi + lo against an exact one).
#include "b200_attn.h"
#include "common.cuh"
#include "gdn_inverse.cuh"

namespace b200 {
namespace {

constexpr int GW_PITCH = GDN_D + 8;                   // bf16 pitch of [64][128] tiles: 272-byte rows, conflict-free ldmatrix
constexpr int GW_TILE = CHUNK * GW_PITCH;             // elements
constexpr int GW_FRAGS = 20;                          // 8 x 16 tiles of a lower triangular 64 x 64 matrix
constexpr int GW_MAT_BYTES = GW_FRAGS * 512;          // ... as fragments: 32 lanes x (hi, hi, lo, lo)
constexpr double GW_LOG2E = 1.4426950408889634;       // decays are powers of two: G is kept in units of log 2
constexpr int GW_GATE_FLOATS = 2 * CHUNK;             // e^G | e^(G_63 - G)
constexpr int GW_SLOT_BYTES = 2 * GW_MAT_BYTES + GW_GATE_FLOATS * 4;   // P | A | gates of one chunk and head

// First fragment of the 8-row tile n; its 16-column tiles 0 .. n / 2 follow one another.
__host__ __device__ constexpr int frag_row(int n) { return (n >> 1) * ((n >> 1) + 1) + (n & 1) * ((n >> 1) + 1); }

struct GdnWalkParams {
  const __nv_bfloat16 *q, *k, *v;
  int64_t q_t, q_h, k_t, k_h, v_t, v_h;
  const float *beta, *g;
  int64_t be_t, be_h, g_t, g_h;
  const int32_t* cu;
  uint8_t* ws;            // [slots of a window, heads, GW_SLOT_BYTES]
  float* state;           // [batch, heads, 128, 128]
  __nv_bfloat16* out;
  int64_t o_t, o_h;
  int heads, batch, items, slots;
  int from, to;           // the window's slots
  int *next, *err;        // counter of the walk's items, behind the slots; the flag of waits that ran out
};
template <int N>
struct Const {
  static constexpr int value = N;
};

// Workspace slots of a sequence's chunks start here: cu / 64 + b grows by at least the chunks of sequence b from b to b + 1,
// so no prefix sum over the batch is needed.
__device__ __forceinline__ int first_slot(const int32_t* cu, int b) { return cu[b] / CHUNK + b; }

__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16(a, b);
  lo = pack_bf16(a - bf16_lo(hi), b - bf16_hi(hi));
}
// 16 bytes global -> shared without registers; zeros, and nothing read, when `on` is false
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(on ? 16 : 0) : "memory");
}

// `cols` bf16 columns of 64 rows of one head, rows from `rows` on as zeros
template <int THREADS>
__device__ __forceinline__ void fetch_rows(uint32_t dst, int pitch, const __nv_bfloat16* src, int64_t stride_t, int rows, int cols, int tid) {
  const int vecs = cols / 8;
  for (int i = tid; i < CHUNK * vecs; i += THREADS) {
    const int r = i / vecs, c = (i % vecs) * 8;
    cp_async16(dst + (r * pitch + c) * 2, src + (r < rows ? r : 0) * stride_t + c, r < rows);
  }
}

// ---------------------------------------------------------------------------------------------------------------- prep
constexpr int GP_THREADS = 256;
// k tile, later P | q tile, later L | merge scratch | G (two floats), beta | G of the first 32 tokens
constexpr int GP_SCRATCH = 2 * GW_TILE * 2;
constexpr int GP_SC = GP_SCRATCH + INV_SCRATCH_FLOATS * 4;
constexpr int GP_SMEM = GP_SC + 3 * CHUNK * 4 + 8;
static_assert(CHUNK * INV_LP * 4 <= GW_TILE * 2, "L and P lie over the q and k tiles");

// grid (slots, heads).  A latency chain of loads, scores, a 64 x 64 triangular inverse on the CUDA cores and stores: four CTAs
// per SM hide it from one another (40 KB of shared memory and 64 registers a thread each).
__global__ void __launch_bounds__(GP_THREADS, 4) gdn_walk_prep_kernel(const __grid_constant__ GdnWalkParams p) {
  extern __shared__ __align__(16) uint8_t smem[];
  pdl_trigger();          // the walk may take over SMs as the last CTAs of this grid finish
  const int slot = p.from + blockIdx.x, h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int b = -1;             // the last sequence whose slots start at or before this one
  for (int i0 = 0; i0 < p.batch; i0 += GP_THREADS) b += __syncthreads_count(i0 + tid < p.batch && first_slot(p.cu, i0 + tid) <= slot);
  if (blockIdx.x == 0 && h == 0 && tid == 0) {
    *p.next = 0;
    if (first_slot(p.cu, p.batch) > p.slots) atomicExch(p.err, 1);   // more tokens than the call named
  }
  if (b < 0) return;
  const int t0 = p.cu[b] + (slot - first_slot(p.cu, b)) * CHUNK, rows = min(CHUNK, p.cu[b + 1] - t0);
  if (rows <= 0) return;
  __nv_bfloat16* kb = reinterpret_cast<__nv_bfloat16*>(smem);
  __nv_bfloat16* qb = kb + GW_TILE;
  float* Pm = reinterpret_cast<float*>(smem);
  float* Lm = reinterpret_cast<float*>(smem + GW_TILE * 2);
  float2* gs = reinterpret_cast<float2*>(smem + GP_SC); // G, and what its rounding left: decays between far tokens keep their digits
  float* bs = reinterpret_cast<float*>(gs + CHUNK);     // beta
  double* first = reinterpret_cast<double*>(bs + CHUNK);
  fetch_rows<GP_THREADS>(smem_u32(kb), GW_PITCH, p.k + t0 * p.k_t + h * p.k_h, p.k_t, rows, GDN_D, tid);
  fetch_rows<GP_THREADS>(smem_u32(qb), GW_PITCH, p.q + t0 * p.q_t + h * p.q_h, p.q_t, rows, GDN_D, tid);
  double G = 0.0;
  if (tid < CHUNK) {
    const int64_t t = t0 + tid;
    const bool on = tid < rows;
    G = on ? static_cast<double>(p.g[t * p.g_t + h * p.g_h]) : 0.0;
    bs[tid] = on ? p.beta[t * p.be_t + h * p.be_h] : 0.f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double x = __shfl_up_sync(0xffffffffu, G, o);
      if (lane >= o) G += x;
    }
    if (tid == 31) *first = G;
  }
  cp_async_wait_all();
  __syncthreads();
  if (tid < CHUNK) {
    if (tid >= 32) G += *first;
    G *= GW_LOG2E;
    const float hi = static_cast<float>(G);
    gs[tid] = make_float2(hi, static_cast<float>(G - hi));
  }
  uint8_t* ws = p.ws + (static_cast<int64_t>(blockIdx.x) * p.heads + h) * GW_SLOT_BYTES;
  // ---- scores: warp = (16 rows, 32 columns); columns past the diagonal block are skipped
  const int mt = warp & 3, nh = warp >> 2, gr = lane >> 2, c2 = (lane & 3) * 2;
  float sk[4][4] = {}, sq[4][4] = {};
  if (nh * 32 <= mt * 16 + 15) {
    const uint32_t ka = smem_u32(kb) + ((mt * 16 + (lane & 15)) * GW_PITCH + (lane >> 4) * 8) * 2, qa = ka + GW_TILE * 2;
    const uint32_t kn = smem_u32(kb) + ((nh * 32 + (lane >> 4) * 8 + (lane & 7)) * GW_PITCH + ((lane >> 3) & 1) * 8) * 2;
#pragma unroll
    for (int ks = 0; ks < GDN_D / 16; ++ks) {
      uint32_t a[4], x[4];
      ldmatrix_x4(a, ka + ks * 32);
      ldmatrix_x4(x, qa + ks * 32);
#pragma unroll
      for (int np = 0; np < 2; ++np) {
        if (nh * 32 + np * 16 > mt * 16) continue;
        uint32_t w[4];
        ldmatrix_x4(w, kn + np * 16 * GW_PITCH * 2 + ks * 32);
        mma_bf16_16816(sk[2 * np], a, w[0], w[1]);
        mma_bf16_16816(sk[2 * np + 1], a, w[2], w[3]);
        mma_bf16_16816(sq[2 * np], x, w[0], w[1]);
        mma_bf16_16816(sq[2 * np + 1], x, w[2], w[3]);
      }
    }
  }
  __syncthreads();                                      // the tiles have been read; G is there
  if (tid < CHUNK) {
    const float2 g = gs[tid], end = gs[CHUNK - 1];
    float* gates = reinterpret_cast<float*>(ws + 2 * GW_MAT_BYTES);
    gates[tid] = exp2f(g.x + g.y);
    gates[CHUNK + tid] = exp2f((end.x - g.x) + (end.y - g.y));
  }
#pragma unroll
  for (int np = 0; np < 2; ++np) {
    const int i0 = nh * 32 + np * 16;                   // 16 columns: one k step of the fragments
    if (i0 > mt * 16) continue;
#pragma unroll
    for (int half = 0; half < 2; ++half) {              // rows gr and gr + 8
      const int t = mt * 16 + half * 8 + gr;
      const float2 Gt = gs[t];
      const float bt = bs[t];
      uint4 w;
      float a[4], l[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int n = 2 * np + (e >> 1), i = i0 + (e >> 1) * 8 + c2 + (e & 1);
        const float2 Gi = gs[i];
        const float d = i <= t ? ex2_fast((Gt.x - Gi.x) + (Gt.y - Gi.y)) : 0.f;
        l[e] = i < t ? bt * d * sk[n][half * 2 + (e & 1)] : 0.f;
        a[e] = d * (i <= t ? sq[n][half * 2 + (e & 1)] : 0.f);
      }
      *reinterpret_cast<float2*>(Lm + t * INV_LP + i0 + c2) = make_float2(l[0], l[1]);
      *reinterpret_cast<float2*>(Lm + t * INV_LP + i0 + 8 + c2) = make_float2(l[2], l[3]);
      split_pair(a[0], a[1], w.x, w.z);
      split_pair(a[2], a[3], w.y, w.w);
      *reinterpret_cast<uint4*>(ws + GW_MAT_BYTES + (frag_row(2 * mt + half) + i0 / 16) * 512 + lane * 16) = w;
    }
  }
  __syncthreads();
  if (tid < 128) blocked_inverse64(Lm, Pm, reinterpret_cast<float*>(smem + GP_SCRATCH), tid);
  __syncthreads();
  // ---- P = inverse diag(beta) as fragments; blocks above the diagonal hold leftovers and are masked
  for (int f = warp; f < GW_FRAGS; f += GP_THREADS / 32) {
    int n = 0;
    while (n < 7 && frag_row(n + 1) <= f) ++n;
    const int t = n * 8 + gr, i = (f - frag_row(n)) * 16 + c2;
    const float2 x = *reinterpret_cast<const float2*>(Pm + t * INV_LP + i), y = *reinterpret_cast<const float2*>(Pm + t * INV_LP + i + 8);
    uint4 w;
    split_pair(i <= t ? x.x * bs[i] : 0.f, i + 1 <= t ? x.y * bs[i + 1] : 0.f, w.x, w.z);
    split_pair(i + 8 <= t ? y.x * bs[i + 8] : 0.f, i + 9 <= t ? y.y * bs[i + 9] : 0.f, w.y, w.w);
    *reinterpret_cast<uint4*>(ws + f * 512 + lane * 16) = w;
  }
}

// ---------------------------------------------------------------------------------------------------------------- walk
constexpr int GW_STAGES = 2;
constexpr int GW_COPY_WARPS = 4;                        // a whole warpgroup, so that it can hand registers over

// Shared memory of a CTA with COLS value columns: stages of k | q | v tiles and a slot of the workspace, then what a stage holds
// (item or -1, first token, rows, flags: last (1) and first (2) chunk of a sequence; of a window 1 and 4), its barriers, and a word between the copy warps.
template <int COLS>
struct WalkSmem {
  static constexpr int VP = COLS + 8;                   // bf16 pitch of the value tile
  static constexpr int K = 0, Q = GW_TILE * 2, V = 2 * Q, P = V + CHUNK * VP * 2, STAGE = P + GW_SLOT_BYTES;
  static constexpr int INFO = GW_STAGES * STAGE, BARS = INFO + GW_STAGES * 16, HANDOVER = BARS + GW_STAGES * 16, BYTES = HANDOVER + 16;
};

// The copy warps: items = (sequence, head, COLS value columns), the first by block index, the others from a counter; chunks go
// into the next stage that `empty` releases, across items.  WINDOWS: only the chunks of this launch's window.
template <int COLS, bool WINDOWS>
__device__ __forceinline__ void copy_chunks(const GdnWalkParams& p, uint8_t* smem, int ct) {
  using L = WalkSmem<COLS>;
  constexpr int SPLIT = GDN_D / COLS, THREADS = 32 * GW_COPY_WARPS;
  uint64_t *full = reinterpret_cast<uint64_t*>(smem + L::BARS), *empty = full + GW_STAGES;
  int* handover = reinterpret_cast<int*>(smem + L::HANDOVER);
  int stage = 0;
  uint32_t parity = 1;
  bool waited = false, ok = true;                       // a thread whose wait ran out copies nothing more, and completes no stage
  for (int item = blockIdx.x;;) {
    int h = 0, col = 0, start = 0, len = 0, slot0 = 0;
    const bool more = item < p.items;
    if (more) {
      const int bh = item / SPLIT, b = bh / p.heads;
      h = bh % p.heads, col = item % SPLIT * COLS;
      start = p.cu[b], len = p.cu[b + 1] - start, slot0 = first_slot(p.cu, b);
    }
    int begin = 0, end = len;
    bool some = true;
    if (WINDOWS && more) {
      const int chunks = (len + CHUNK - 1) / CHUNK;
      begin = min(max(p.from - slot0, 0), chunks) * CHUNK, end = min(len, min(p.to - slot0, chunks) * CHUNK);
      some = len > 0 ? begin < end : p.from <= slot0 && slot0 < p.to;
    }
    for (int t0 = begin; some && (t0 == begin || t0 < end); t0 += CHUNK) {   // an empty sequence passes once: its state is zero
      ok = ok && mbar_wait_bounded(&empty[stage], parity);
      uint8_t* to = smem + stage * L::STAGE;
      const int rows = ok ? min(CHUNK, len - t0) : 0;
      if (rows > 0) {
        const int64_t t = start + t0;
        fetch_rows<THREADS>(smem_u32(to) + L::K, GW_PITCH, p.k + t * p.k_t + h * p.k_h, p.k_t, rows, GDN_D, ct);
        fetch_rows<THREADS>(smem_u32(to) + L::Q, GW_PITCH, p.q + t * p.q_t + h * p.q_h, p.q_t, rows, GDN_D, ct);
        fetch_rows<THREADS>(smem_u32(to) + L::V, L::VP, p.v + t * p.v_t + h * p.v_h + col, p.v_t, rows, COLS, ct);
      }
      if (!waited) pdl_wait();                          // the prepared matrices and the counter are complete
      waited = true;
      if (ct == 0 && ok) {
        // a batch of more tokens than the call named: nobody prepared this sequence's end, and its state and output stay as they are
        const bool fits = !more || slot0 + (len + CHUNK - 1) / CHUNK <= p.slots;
        *reinterpret_cast<int4*>(smem + L::INFO + stage * 16) =
            make_int4(more ? item : -1, start + t0, fits ? rows : 0,
                      fits ? (t0 + CHUNK >= end ? 1 : 0) | (t0 == 0 ? 2 : 0) | (WINDOWS && t0 > 0 && t0 == begin ? 4 : 0) : 0);
        if (fits && rows > 0) {
          mbar_expect_tx(&full[stage], GW_SLOT_BYTES);
          bulk_g2s(to + L::P, p.ws + (static_cast<int64_t>(slot0 + t0 / CHUNK - (WINDOWS ? p.from : 0)) * p.heads + h) * GW_SLOT_BYTES, GW_SLOT_BYTES, &full[stage]);
        } else {
          mbar_arrive(&full[stage]);
        }
      }
      if (ok) asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full[stage])) : "memory");
      if (++stage == GW_STAGES) stage = 0, parity ^= 1;
    }
    if (!more) break;
    if (WINDOWS && !waited) pdl_wait();                 // the counter is complete, also where the first item has nothing here
    if (WINDOWS) waited = true;
    __syncwarp();
    if (ct == 0 && ok) *handover = gridDim.x + atomicAdd(p.next, 1);
    ok = named_barrier_all(1, THREADS, ok);             // they go on or give up as one
    if (!ok) break;
    item = *handover;
    named_barrier(1, THREADS);
  }
  cp_async_wait_all();
  if (!ok) {
    atomicExch(p.err, 1);
    // bulk copies that nobody waits for any more may still be landing in this CTA's shared memory: either phase of a stage
    if (ct == 0)
      for (int i = 0; i < 2 * GW_STAGES; ++i) mbar_wait_bounded(&full[i >> 1], i & 1, 1u << 12);
  }
}
template <int COLS>
__device__ __forceinline__ void init_stages(uint8_t* smem, int consumers) {
  uint64_t *full = reinterpret_cast<uint64_t*>(smem + WalkSmem<COLS>::BARS), *empty = full + GW_STAGES;
  for (int s = 0; s < GW_STAGES; ++s) {
    mbar_init(&full[s], 32 * GW_COPY_WARPS + 1);        // every copy thread's part, and the bytes of the bulk copy
    mbar_init(&empty[s], consumers);
  }
}

// Left-operand fragments of 16 columns of an accumulator row block, as a bf16 pair
__device__ __forceinline__ void split_frag(const float (&x)[4], const float (&y)[4], uint32_t (&hi)[4], uint32_t (&lo)[4]) {
  split_pair(x[0], x[1], hi[0], lo[0]);
  split_pair(x[2], x[3], hi[1], lo[1]);
  split_pair(y[0], y[1], hi[2], lo[2]);
  split_pair(y[2], y[3], hi[3], lo[3]);
}
// acc[n] += (hi + lo) (w.xy + w.zw) without lo w.zw, for the row tiles 2 KS <= n < N of a triangular matrix.  Four tiles at a
// time, product by product: an accumulator's next product comes four instructions later, which covers the tensor pipe's latency.
template <int KS, int N>
__device__ __forceinline__ void triangular(float (&acc)[N][4], const uint32_t (&hi)[4], const uint32_t (&lo)[4], const uint8_t* frags, int lane) {
  uint4 w[N];
#pragma unroll
  for (int n = 2 * KS; n < N; ++n) w[n] = *reinterpret_cast<const uint4*>(frags + (frag_row(n) + KS) * 512 + lane * 16);
#pragma unroll
  for (int n0 = 2 * KS; n0 < N; n0 += 4) {
#pragma unroll
    for (int n = n0; n < n0 + 4 && n < N; ++n) mma_bf16_16816(acc[n], hi, w[n].x, w[n].y);
#pragma unroll
    for (int n = n0; n < n0 + 4 && n < N; ++n) mma_bf16_16816(acc[n], lo, w[n].x, w[n].y);
#pragma unroll
    for (int n = n0; n < n0 + 4 && n < N; ++n) mma_bf16_16816(acc[n], hi, w[n].z, w[n].w);
  }
}

// One chunk of up to 16 * TILES tokens: S^T [16 x 128] in accumulators (value column lane / 4 (+ 8), key dims
// 8 n + (lane % 4) * 2 (+ 1)) moves on, o^T replaces the warp's columns of the value tile.
template <int WARPS, int TILES>
__device__ __forceinline__ void walk_chunk(float (&S)[GDN_D / 8][4], const uint8_t* st, bool carry, int warp, int lane) {
  using L = WalkSmem<16 * WARPS>;
  constexpr int N = 2 * TILES;                          // 8-token tiles
  const int c2 = (lane & 3) * 2;
  const uint32_t at = smem_u32(st);
  const uint32_t nk_off = (((lane >> 4) * 8 + (lane & 7)) * GW_PITCH + ((lane >> 3) & 1) * 8) * 2;   // [n][k] tiles: k and q rows
  const uint32_t kn_off = ((((lane >> 3) & 1) * 8 + (lane & 7)) * GW_PITCH + (lane >> 4) * 8) * 2;   // [k][n], transposing
  const uint32_t v_off = (((lane >> 4) * 8 + (lane & 7)) * L::VP + warp * 16 + ((lane >> 3) & 1) * 8) * 2;
  const uint8_t *fp = st + L::P, *fa = fp + GW_MAT_BYTES;
  const float* eg = reinterpret_cast<const float*>(fa + GW_MAT_BYTES);
  // ---- (k S)^T and (q S)^T; nothing to do for a sequence's first chunk
  float M[N][4] = {}, O[N][4] = {};
  if (carry) {
    uint32_t hi[2][4], lo[2][4], w[2][4], x[2][4];      // this step's and the next one's
    auto load = [&](int i) {                            // step i: 16 tokens of 16 key dims
      ldmatrix_x4(w[i & 1], at + L::K + nk_off + ((i % TILES) * 16 * GW_PITCH + (i / TILES) * 16) * 2);
      ldmatrix_x4(x[i & 1], at + L::Q + nk_off + ((i % TILES) * 16 * GW_PITCH + (i / TILES) * 16) * 2);
    };
    load(0);
    split_frag(S[0], S[1], hi[0], lo[0]);
#pragma unroll
    for (int i = 0; i < 8 * TILES; ++i) {
      const int ks = i / TILES, n = (i % TILES) * 2, a = ks & 1, c = i & 1;
      if (i + 1 < 8 * TILES) load(i + 1);
      if (i % TILES == TILES / 2 && ks + 1 < GDN_D / 16) split_frag(S[2 * ks + 2], S[2 * ks + 3], hi[a ^ 1], lo[a ^ 1]);
      mma_bf16_16816(M[n], hi[a], w[c][0], w[c][1]);
      mma_bf16_16816(M[n + 1], hi[a], w[c][2], w[c][3]);
      mma_bf16_16816(O[n], hi[a], x[c][0], x[c][1]);
      mma_bf16_16816(O[n + 1], hi[a], x[c][2], x[c][3]);
      mma_bf16_16816(M[n], lo[a], w[c][0], w[c][1]);
      mma_bf16_16816(M[n + 1], lo[a], w[c][2], w[c][3]);
      mma_bf16_16816(O[n], lo[a], x[c][0], x[c][1]);
      mma_bf16_16816(O[n + 1], lo[a], x[c][2], x[c][3]);
    }
  }
  // ---- R^T = v^T - e^G (k S)^T; e^G (q S)^T
#pragma unroll
  for (int n = 0; n < N; n += 2) {
    uint32_t v[4];
    ldmatrix_x4_trans(v, at + L::V + v_off + n * 8 * L::VP * 2);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float2 e = *reinterpret_cast<const float2*>(eg + (n + i) * 8 + c2);
      M[n + i][0] = fmaf(-e.x, M[n + i][0], bf16_lo(v[2 * i]));
      M[n + i][1] = fmaf(-e.y, M[n + i][1], bf16_hi(v[2 * i]));
      M[n + i][2] = fmaf(-e.x, M[n + i][2], bf16_lo(v[2 * i + 1]));
      M[n + i][3] = fmaf(-e.y, M[n + i][3], bf16_hi(v[2 * i + 1]));
      O[n + i][0] *= e.x, O[n + i][1] *= e.y, O[n + i][2] *= e.x, O[n + i][3] *= e.y;
    }
  }
  const float keep = eg[CHUNK - 1];
#pragma unroll
  for (int n = 0; n < GDN_D / 8; ++n) S[n][0] *= keep, S[n][1] *= keep, S[n][2] *= keep, S[n][3] *= keep;
  // ---- delta^T = R^T P^T by 16 tokens; as soon as 16 are complete they go into
  //      o^T += delta^T A^T and S^T += (e^(G_63 - G) delta)^T k, one step behind
  float D[N][4] = {};
  auto delta = [&](auto step) {
    constexpr int KS = decltype(step)::value;
    if constexpr (KS < TILES) {
      uint32_t hi[4], lo[4];
      split_frag(M[2 * KS], M[2 * KS + 1], hi, lo);
      triangular<KS, N>(D, hi, lo, fp, lane);
    }
  };
  auto use = [&](auto step) {
    constexpr int KS = decltype(step)::value;
    if constexpr (KS < TILES) {
      uint32_t hi[4], lo[4], eh[4], el[4], w[2][4], z[2][4];
      auto load = [&](int i) {                          // 16 tokens of 32 key dims
        ldmatrix_x4_trans(w[i & 1], at + L::K + kn_off + (KS * 16 * GW_PITCH + i * 32) * 2);
        ldmatrix_x4_trans(z[i & 1], at + L::K + kn_off + (KS * 16 * GW_PITCH + i * 32 + 16) * 2);
      };
      load(0);
      split_frag(D[2 * KS], D[2 * KS + 1], hi, lo);
      const float2 ra = *reinterpret_cast<const float2*>(eg + CHUNK + KS * 16 + c2);
      const float2 rb = *reinterpret_cast<const float2*>(eg + CHUNK + KS * 16 + 8 + c2);
      float x[4] = {D[2 * KS][0] * ra.x, D[2 * KS][1] * ra.y, D[2 * KS][2] * ra.x, D[2 * KS][3] * ra.y};
      float y[4] = {D[2 * KS + 1][0] * rb.x, D[2 * KS + 1][1] * rb.y, D[2 * KS + 1][2] * rb.x, D[2 * KS + 1][3] * rb.y};
      split_frag(x, y, eh, el);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int n = 4 * i, c = i & 1;
        if (i < 3) load(i + 1);
        mma_bf16_16816(S[n], eh, w[c][0], w[c][1]);
        mma_bf16_16816(S[n + 1], eh, w[c][2], w[c][3]);
        mma_bf16_16816(S[n + 2], eh, z[c][0], z[c][1]);
        mma_bf16_16816(S[n + 3], eh, z[c][2], z[c][3]);
        mma_bf16_16816(S[n], el, w[c][0], w[c][1]);
        mma_bf16_16816(S[n + 1], el, w[c][2], w[c][3]);
        mma_bf16_16816(S[n + 2], el, z[c][0], z[c][1]);
        mma_bf16_16816(S[n + 3], el, z[c][2], z[c][3]);
      }
      triangular<KS, N>(O, hi, lo, fa, lane);
    }
  };
  delta(Const<0>());
  delta(Const<1>());
  use(Const<0>());
  delta(Const<2>());
  use(Const<1>());
  delta(Const<3>());
  use(Const<2>());
  use(Const<3>());
#pragma unroll
  for (int n = 0; n < N; n += 2)
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(at + L::V + v_off + n * 8 * L::VP * 2),
                 "r"(pack_bf16(O[n][0], O[n][1])), "r"(pack_bf16(O[n][2], O[n][3])), "r"(pack_bf16(O[n + 1][0], O[n + 1][1])),
                 "r"(pack_bf16(O[n + 1][2], O[n + 1][3]))
                 : "memory");
}

// A warp = 16 value columns of one head, alone with its 16 x 128 state; the tensor pipe bounds it (504 products of 2048
// multiply-adds per full chunk).  32 x 128 tokens, 16 heads: 50 us, the pipe active 58 % of the time on average and 67 % on the
// busiest SM, where every second chunk is a sequence's first and waits for its loads.
template <int WARPS, bool WINDOWS>
__global__ void __launch_bounds__(32 * (WARPS + GW_COPY_WARPS), 1) gdn_walk_kernel(const __grid_constant__ GdnWalkParams p) {
  using L = WalkSmem<16 * WARPS>;
  constexpr int SPLIT = 8 / WARPS;
  extern __shared__ __align__(16) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint64_t *full = reinterpret_cast<uint64_t*>(smem + L::BARS), *empty = full + GW_STAGES;
  if (tid == 0) {
    init_stages<16 * WARPS>(smem, WARPS);
    mbar_fence_init();
  }
  __syncthreads();
  if (warp >= WARPS) {
    // 8 + 4 warps start with 168 registers each (3 x 168 = 504 per column of warpgroups): 40 + 2 x 232 of them
    if constexpr (WARPS == 8) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    copy_chunks<16 * WARPS, WINDOWS>(p, smem, tid - 32 * WARPS);
    return;
  }
  if constexpr (WARPS == 8) asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
  // S^T: value column lane / 4 (+ 8) of the warp's 16, key dims 8 n + (lane % 4) * 2 (+ 1)
  float S[GDN_D / 8][4];
#pragma unroll
  for (int n = 0; n < GDN_D / 8; ++n) S[n][0] = S[n][1] = S[n][2] = S[n][3] = 0.f;
  const int gr = lane >> 2, c2 = (lane & 3) * 2;
  int stage = 0;
  uint32_t parity = 0;
  for (;;) {
    if (!warp_wait_bounded(&full[stage], parity)) {
      if (lane == 0) atomicExch(p.err, 1);
      return;
    }
    const int4 info = *reinterpret_cast<const int4*>(smem + L::INFO + stage * 16);
    if (info.x < 0) return;
    const int bh = info.x / SPLIT, h = bh % p.heads, col = info.x % SPLIT * 16 * WARPS + warp * 16;
    if (WINDOWS && (info.w & 4)) {                      // what the window before left
      const float* from = p.state + static_cast<int64_t>(bh) * GDN_D * GDN_D + col;
#pragma unroll
      for (int n = 0; n < GDN_D / 8; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) S[n][j] = from[(n * 8 + c2 + (j & 1)) * GDN_D + gr + (j >> 1) * 8];
    }
    if (info.z > 0) {
      const uint8_t* st = smem + stage * L::STAGE;
      const bool carry = !(info.w & 2);
      // a sequence's last chunk pays for 16, 32 or 64 tokens
      if (info.z > 32) walk_chunk<WARPS, 4>(S, st, carry, warp, lane);
      else if (info.z > 16) walk_chunk<WARPS, 2>(S, st, carry, warp, lane);
      else walk_chunk<WARPS, 1>(S, st, carry, warp, lane);
      // 32 bytes per token go out
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = i * 16 + (lane >> 1), c = (lane & 1) * 8;
        if (t < info.z)
          *reinterpret_cast<uint4*>(p.out + (static_cast<int64_t>(info.y) + t) * p.o_t + h * p.o_h + col + c) =
              *reinterpret_cast<const uint4*>(st + L::V + (t * L::VP + warp * 16 + c) * 2);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[stage]);
    if (++stage == GW_STAGES) stage = 0, parity ^= 1;
    if (info.w & 1) {
      float* to = p.state + static_cast<int64_t>(bh) * GDN_D * GDN_D + col;
#pragma unroll
      for (int n = 0; n < GDN_D / 8; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          to[(n * 8 + c2 + (j & 1)) * GDN_D + gr + (j >> 1) * 8] = S[n][j];
          S[n][j] = 0.f;
        }
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------- teams
// Few heads leave the warps above alone on their schedulers, where the chain of a chunk's products sets the time (3.4 us per
// chunk).  Here four warps share 16 value columns: a warp computes 16 of the chunk's tokens in k S, q S, delta and o, and keeps
// 32 of the state's key dims; S, R and delta go round as left-operand fragments in shared memory, a lane's four registers being
// 16 consecutive bytes, so that nothing is rearranged.  Three meetings per chunk, each through an mbarrier.  What nobody waits for, the
// output q S + A delta, comes behind the last one; or, with one team per CTA, four more warps compute it one chunk behind (APART),
// which takes it off the chain that the chunks are: one sequence of 2048 tokens 80.7 -> 77.8 us (with prep), of 8192 298 -> 286; without any
// output it would be 73 and 268.  S and delta then have two places and two barriers each, by turns: the team in front may be a chunk ahead, and
// must not come round to a place, or a phase, that is still waited for.  Not kept: bulk copies of rows instead of 16-byte pieces (60 cycles
// each, 216 us), three stages (no change), the output's first read behind R (79), rolled products (79 to 82).
template <int TEAMS>
struct TeamSmem {
  using L = WalkSmem<16 * TEAMS>;
  static constexpr bool APART = TEAMS == 1;
  static constexpr int PLACES = APART ? 2 : 1;
  static constexpr int S = 0, S_STEP = 8 * 1024, R = S + PLACES * S_STEP, E = R + 4 * 1024, D = E + 4 * 1024, D_STEP = 4 * 1024;   // hi, lo: 512 bytes each
  static constexpr int EX = (L::BYTES + 127) / 128 * 128, EX_BYTES = D + PLACES * D_STEP, BARS = EX + TEAMS * EX_BYTES, BYTES = BARS + TEAMS * 64;
  static constexpr int BAR_S = 0, BAR_R = 2, BAR_D = 3, BAR_OUT = 5;   // two each where there are two places, but for R
  static constexpr int WARPS = (APART ? 8 : 4) * TEAMS, THREADS = 32 * (WARPS + GW_COPY_WARPS);
  // place, barrier and phase of the n-th state, delta or output
  static __device__ __forceinline__ int place(uint32_t n) { return APART ? n & 1 : 0; }
  static __device__ __forceinline__ int bar_of(int first, uint32_t n) { return first + place(n); }
  static __device__ __forceinline__ uint32_t phase_of(uint32_t n) { return APART ? (n >> 1) & 1 : n & 1; }
};

__device__ __forceinline__ void put_frag(uint8_t* to, const uint32_t (&hi)[4], const uint32_t (&lo)[4], int lane) {
  *reinterpret_cast<uint4*>(to + lane * 16) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
  *reinterpret_cast<uint4*>(to + 512 + lane * 16) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
}
__device__ __forceinline__ void get_frag(const uint8_t* from, uint32_t (&hi)[4], uint32_t (&lo)[4], int lane) {
  const uint4 a = *reinterpret_cast<const uint4*>(from + lane * 16), b = *reinterpret_cast<const uint4*>(from + 512 + lane * 16);
  hi[0] = a.x, hi[1] = a.y, hi[2] = a.z, hi[3] = a.w;
  lo[0] = b.x, lo[1] = b.y, lo[2] = b.z, lo[3] = b.w;
}
// The three products of a pair of left operands with the pairs of two row tiles, each into sums of its own
__device__ __forceinline__ void pair_products(float (&s)[2][3][4], const uint32_t (&hi)[4], const uint32_t (&lo)[4], const uint4& a, const uint4& b) {
  mma_bf16_16816(s[0][0], hi, a.x, a.y);
  mma_bf16_16816(s[1][0], hi, b.x, b.y);
  mma_bf16_16816(s[0][1], lo, a.x, a.y);
  mma_bf16_16816(s[1][1], lo, b.x, b.y);
  mma_bf16_16816(s[0][2], hi, a.z, a.w);
  mma_bf16_16816(s[1][2], hi, b.z, b.w);
}

// Wait among the warps of a team, which are a few hundred cycles apart at most: polls that do not put the warp to sleep.  Lanes
// that give up stay with their warp, which leaves as one before the next chunk.
__device__ __forceinline__ bool team_wait(uint64_t* bar, uint32_t parity) {
  for (int i = 0; i < (1 << 22); ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// o^T of a warp's 16 tokens: e^G (q S)^T, and A delta from its own fragments (dh, dl) and those of the tokens before, at `d`
__device__ __forceinline__ void query_state(float (&O)[2][4], const uint32_t (&sh)[8][4], const uint32_t (&sl)[8][4], uint32_t q, const float* eg, int c2) {
  float m[2][2][4] = {};
#pragma unroll
  for (int ks = 0; ks < 8; ++ks) {
    uint32_t b[4];
    ldmatrix_x4(b, q + ks * 32);
    mma_bf16_16816(m[0][0], sh[ks], b[0], b[1]);
    mma_bf16_16816(m[1][0], sh[ks], b[2], b[3]);
    mma_bf16_16816(m[0][1], sl[ks], b[0], b[1]);
    mma_bf16_16816(m[1][1], sl[ks], b[2], b[3]);
  }
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    const float2 e = *reinterpret_cast<const float2*>(eg + n * 8 + c2);
#pragma unroll
    for (int j = 0; j < 4; ++j) O[n][j] = (m[n][0][j] + m[n][1][j]) * ((j & 1) ? e.y : e.x);
  }
}
__device__ __forceinline__ void add_within(float (&O)[2][4], const uint32_t (&dh)[4], const uint32_t (&dl)[4], const uint8_t* d, const uint8_t* fa, int w, int lane) {
  float x[2][3][4] = {};
  pair_products(x, dh, dl, *reinterpret_cast<const uint4*>(fa + (frag_row(2 * w) + w) * 512 + lane * 16),
                *reinterpret_cast<const uint4*>(fa + (frag_row(2 * w + 1) + w) * 512 + lane * 16));
#pragma unroll
  for (int ks = 0; ks < 3; ++ks) {
    if (ks >= w) break;
    uint32_t xh[4], xl[4];
    get_frag(d + ks * 1024, xh, xl, lane);
    pair_products(x, xh, xl, *reinterpret_cast<const uint4*>(fa + (frag_row(2 * w) + ks) * 512 + lane * 16),
                  *reinterpret_cast<const uint4*>(fa + (frag_row(2 * w + 1) + ks) * 512 + lane * 16));
  }
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j) O[n][j] += x[n][0][j] + x[n][1][j] + x[n][2][j];
}
// ... through the own rows of the value tile, 32 bytes per token
__device__ __forceinline__ void store_tokens(const float (&O)[2][4], uint32_t tile, const uint8_t* rows, int pitch, __nv_bfloat16* out, int64_t o_t, int tokens, int lane) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(tile), "r"(pack_bf16(O[0][0], O[0][1])),
               "r"(pack_bf16(O[0][2], O[0][3])), "r"(pack_bf16(O[1][0], O[1][1])), "r"(pack_bf16(O[1][2], O[1][3]))
               : "memory");
  __syncwarp();
  const int t = lane >> 1, c = (lane & 1) * 8;
  if (t < tokens) *reinterpret_cast<uint4*>(out + t * o_t + c) = *reinterpret_cast<const uint4*>(rows + (t * pitch + c) * 2);
}

// The output warps have done with every chunk before this one: their places may be written again, their phases are over
template <typename T>
__device__ __forceinline__ bool outputs_done(uint64_t* bars, uint32_t& outputs, uint32_t chunks, bool ok) {
  if constexpr (T::APART)
    for (; outputs < chunks; ++outputs) ok = ok && team_wait(&bars[T::bar_of(T::BAR_OUT, outputs)], T::phase_of(outputs));
  return ok;
}

// The four warps of the output (APART): what the chunk's other team publishes, one chunk behind it
template <int TEAMS, bool WINDOWS>
__device__ __forceinline__ void output_chunks(const GdnWalkParams& p, uint8_t* smem, int tid) {
  using L = WalkSmem<16 * TEAMS>;
  using T = TeamSmem<TEAMS>;
  constexpr int SPLIT = 8 / TEAMS;
  const int lane = tid & 31, w = (tid >> 5) & 3;
  uint64_t *full = reinterpret_cast<uint64_t*>(smem + L::BARS), *empty = full + GW_STAGES;
  const uint8_t* ex = smem + T::EX;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + T::BARS);
  uint32_t states = 0, chunks = 0, full_parity = 0;     // states taken over and chunks begun so far
  const int c2 = (lane & 3) * 2;
  const uint32_t nk_off = ((w * 16 + (lane >> 4) * 8 + (lane & 7)) * GW_PITCH + ((lane >> 3) & 1) * 8) * 2;
  const uint32_t v_off = ((w * 16 + (lane >> 4) * 8 + (lane & 7)) * L::VP + ((lane >> 3) & 1) * 8) * 2;
  const int v_rows = L::V + w * 16 * L::VP * 2;
  int stage = 0, bh = 0, h = 0, col = 0;
  bool ok = true;
  for (;;) {
    ok = warp_wait_bounded(&full[stage], full_parity, ok);
    if (!ok) break;
    const int4 info = *reinterpret_cast<const int4*>(smem + L::INFO + stage * 16);
    if (info.x < 0) return;
    if (info.w & (WINDOWS ? 6 : 2)) bh = info.x / SPLIT, h = bh % p.heads, col = info.x % SPLIT * 16;
    if (info.z > 0) {
      const uint8_t* st = smem + stage * L::STAGE;
      const uint8_t* fa = st + L::P + GW_MAT_BYTES;
      const float* eg = reinterpret_cast<const float*>(fa + GW_MAT_BYTES) + w * 16;
      const bool mine = info.z > 16 * w;
      float O[2][4] = {};
      if (!(info.w & 2)) {
        ok = ok && team_wait(&bars[T::bar_of(T::BAR_S, states)], T::phase_of(states));
        if (mine) {
          uint32_t sh[8][4], sl[8][4];
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) get_frag(ex + T::S + T::place(states) * T::S_STEP + ks * 1024, sh[ks], sl[ks], lane);
          query_state(O, sh, sl, smem_u32(st) + L::Q + nk_off, eg, c2);
        }
        ++states;
      }
      ok = ok && team_wait(&bars[T::bar_of(T::BAR_D, chunks)], T::phase_of(chunks));
      if (mine) {
        const uint8_t* d = ex + T::D + T::place(chunks) * T::D_STEP;
        uint32_t dh[4], dl[4];
        get_frag(d + w * 1024, dh, dl, lane);
        add_within(O, dh, dl, d, fa, w, lane);
        store_tokens(O, smem_u32(st) + L::V + v_off, st + v_rows, L::VP, p.out + (static_cast<int64_t>(info.y) + w * 16) * p.o_t + h * p.o_h + col,
                     p.o_t, ok ? info.z - w * 16 : 0, lane);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[T::bar_of(T::BAR_OUT, chunks)]);
      ++chunks;
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[stage]);
    if (++stage == GW_STAGES) stage = 0, full_parity ^= 1;
  }
  if (lane == 0) atomicExch(p.err, 1);
}

template <int TEAMS, bool WINDOWS>
__global__ void __launch_bounds__(TeamSmem<TEAMS>::THREADS, 1) gdn_walk_team_kernel(const __grid_constant__ GdnWalkParams p) {
  using L = WalkSmem<16 * TEAMS>;
  using T = TeamSmem<TEAMS>;
  constexpr int SPLIT = 8 / TEAMS;
  extern __shared__ __align__(16) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, w = (tid >> 5) & 3;
  uint64_t *full = reinterpret_cast<uint64_t*>(smem + L::BARS), *empty = full + GW_STAGES;
  if (tid == 0) {
    init_stages<16 * TEAMS>(smem, T::WARPS);
    for (int i = 0; i < TEAMS * 8; ++i) mbar_init(reinterpret_cast<uint64_t*>(smem + T::BARS) + i, 4);
    mbar_fence_init();
  }
  __syncthreads();
  if (tid >= 128 * TEAMS) {
    if (tid >= 32 * T::WARPS) copy_chunks<16 * TEAMS, WINDOWS>(p, smem, tid - 32 * T::WARPS);
    else if constexpr (T::APART) output_chunks<TEAMS, WINDOWS>(p, smem, tid);
    return;
  }
  const int team = tid >> 7;
  uint8_t* ex = smem + T::EX + team * T::EX_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + T::BARS) + team * 8;
  uint32_t states = 0, chunks = 0, outputs = 0, full_parity = 0;   // states taken over, chunks begun, outputs waited for, so far
  auto arrive = [&](int i) {
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars[i]);
  };
  const int gr = lane >> 2, c2 = (lane & 3) * 2;
  const uint32_t nk_off = ((w * 16 + (lane >> 4) * 8 + (lane & 7)) * GW_PITCH + ((lane >> 3) & 1) * 8) * 2;
  const uint32_t v_off = ((w * 16 + (lane >> 4) * 8 + (lane & 7)) * L::VP + team * 16 + ((lane >> 3) & 1) * 8) * 2;
  const int v_rows = L::V + (w * 16 * L::VP + team * 16) * 2;
  int stage = 0, bh = 0, h = 0, col = 0;
  bool ok = true;
  // S^T: value column lane / 4 (+ 8) of the team's 16, key dims 32 w + 8 n + (lane % 4) * 2 (+ 1)
  float S[4][4] = {};
  const uint32_t kn_off = ((((lane >> 3) & 1) * 8 + (lane & 7)) * GW_PITCH + w * 32 + (lane >> 4) * 8) * 2;
  uint32_t published = 0;
  auto publish = [&]() {
    uint8_t* to = ex + T::S + T::place(published) * T::S_STEP + 2 * w * 1024;
    uint32_t hi[4], lo[4];
    split_frag(S[0], S[1], hi, lo);
    put_frag(to, hi, lo, lane);
    split_frag(S[2], S[3], hi, lo);
    put_frag(to + 1024, hi, lo, lane);
    arrive(T::bar_of(T::BAR_S, published));
    ++published;
  };
  for (;;) {
    ok = warp_wait_bounded(&full[stage], full_parity, ok);
    if (!ok) break;
    const int4 info = *reinterpret_cast<const int4*>(smem + L::INFO + stage * 16);
    if (info.x < 0) return;
    if (info.w & (WINDOWS ? 6 : 2)) bh = info.x / SPLIT, h = bh % p.heads, col = info.x % SPLIT * 16 * TEAMS + team * 16;
    if (WINDOWS && (info.w & 4)) {                      // what the window before left
      const float* from = p.state + static_cast<int64_t>(bh) * GDN_D * GDN_D + w * 32 * GDN_D + col;
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) S[n][j] = from[(n * 8 + c2 + (j & 1)) * GDN_D + gr + (j >> 1) * 8];
      ok = outputs_done<T>(bars, outputs, chunks, ok);
      publish();
    }
    if (info.z > 0) {
      const uint8_t* st = smem + stage * L::STAGE;
      const uint32_t at = smem_u32(st);
      const uint8_t *fp = st + L::P, *fa = fp + GW_MAT_BYTES;
      const float* eg = reinterpret_cast<const float*>(fa + GW_MAT_BYTES);
      const bool mine = info.z > 16 * w, carry = !(info.w & 2), last = info.w & 1;
      const int groups = (info.z + 15) >> 4;
      uint32_t rh[4], rl[4], sh[8][4], sl[8][4];
      float O[2][4] = {}, D[2][4] = {};
      if (carry) {
        ok = ok && team_wait(&bars[T::bar_of(T::BAR_S, states)], T::phase_of(states));
        ++states;
      }
      if (mine) {
        // ---- k S of the own tokens, R
        float m[2][2][4] = {};
        if (carry) {
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) get_frag(ex + T::S + T::place(states - 1) * T::S_STEP + ks * 1024, sh[ks], sl[ks], lane);
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) {
            uint32_t b[4];
            ldmatrix_x4(b, at + L::K + nk_off + ks * 32);
            mma_bf16_16816(m[0][0], sh[ks], b[0], b[1]);
            mma_bf16_16816(m[1][0], sh[ks], b[2], b[3]);
            mma_bf16_16816(m[0][1], sl[ks], b[0], b[1]);
            mma_bf16_16816(m[1][1], sl[ks], b[2], b[3]);
          }
        }
        uint32_t v[4];
        ldmatrix_x4_trans(v, at + L::V + v_off);
        float R[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const float2 e = *reinterpret_cast<const float2*>(eg + w * 16 + n * 8 + c2);
          R[n][0] = fmaf(-e.x, m[n][0][0] + m[n][1][0], bf16_lo(v[2 * n]));
          R[n][1] = fmaf(-e.y, m[n][0][1] + m[n][1][1], bf16_hi(v[2 * n]));
          R[n][2] = fmaf(-e.x, m[n][0][2] + m[n][1][2], bf16_lo(v[2 * n + 1]));
          R[n][3] = fmaf(-e.y, m[n][0][3] + m[n][1][3], bf16_hi(v[2 * n + 1]));
        }
        split_frag(R[0], R[1], rh, rl);
        put_frag(ex + T::R + w * 1024, rh, rl, lane);
      }
      arrive(T::BAR_R);
      const float keep = eg[CHUNK - 1];
#pragma unroll
      for (int n = 0; n < 4; ++n) S[n][0] *= keep, S[n][1] *= keep, S[n][2] *= keep, S[n][3] *= keep;
      float s[2][3][4] = {};
      if (mine)                                         // the own tokens' part of delta
        pair_products(s, rh, rl, *reinterpret_cast<const uint4*>(fp + (frag_row(2 * w) + w) * 512 + lane * 16),
                      *reinterpret_cast<const uint4*>(fp + (frag_row(2 * w + 1) + w) * 512 + lane * 16));
      ok = ok && team_wait(&bars[T::BAR_R], chunks & 1);
      uint8_t* d = ex + T::D + T::place(chunks) * T::D_STEP;
      uint32_t dh[4], dl[4], eh[4], el[4];
      if (mine) {
#pragma unroll
        for (int ks = 0; ks < 3; ++ks) {
          if (ks >= w) break;
          uint32_t xh[4], xl[4];
          get_frag(ex + T::R + ks * 1024, xh, xl, lane);
          pair_products(s, xh, xl, *reinterpret_cast<const uint4*>(fp + (frag_row(2 * w) + ks) * 512 + lane * 16),
                        *reinterpret_cast<const uint4*>(fp + (frag_row(2 * w + 1) + ks) * 512 + lane * 16));
        }
        float x[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const float2 r = *reinterpret_cast<const float2*>(eg + CHUNK + w * 16 + n * 8 + c2);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            D[n][j] = s[n][0][j] + s[n][1][j] + s[n][2][j];
            x[n][j] = D[n][j] * ((j & 1) ? r.y : r.x);
          }
        }
        split_frag(x[0], x[1], eh, el);
        put_frag(ex + T::E + w * 1024, eh, el, lane);
        split_frag(D[0], D[1], dh, dl);
        put_frag(d + w * 1024, dh, dl, lane);
      }
      arrive(T::bar_of(T::BAR_D, chunks));
      ok = ok && team_wait(&bars[T::bar_of(T::BAR_D, chunks)], T::phase_of(chunks));
      // ---- the own key dims of the state
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        if (ks >= groups) break;
        uint32_t xh[4], xl[4], a[4], b[4];
        get_frag(ex + T::E + ks * 1024, xh, xl, lane);
        ldmatrix_x4_trans(a, at + L::K + kn_off + ks * 16 * GW_PITCH * 2);
        ldmatrix_x4_trans(b, at + L::K + kn_off + ks * 16 * GW_PITCH * 2 + 32);
        mma_bf16_16816(S[0], xh, a[0], a[1]);
        mma_bf16_16816(S[1], xh, a[2], a[3]);
        mma_bf16_16816(S[2], xh, b[0], b[1]);
        mma_bf16_16816(S[3], xh, b[2], b[3]);
        mma_bf16_16816(S[0], xl, a[0], a[1]);
        mma_bf16_16816(S[1], xl, a[2], a[3]);
        mma_bf16_16816(S[2], xl, b[0], b[1]);
        mma_bf16_16816(S[3], xl, b[2], b[3]);
      }
      ok = outputs_done<T>(bars, outputs, chunks, ok);
      if (!last) publish();
      ++chunks;
      if (!T::APART && mine) {                          // the output, where nobody waits for it any more
        if (carry) query_state(O, sh, sl, at + L::Q + nk_off, eg + w * 16, c2);
        add_within(O, dh, dl, d, fa, w, lane);
        store_tokens(O, at + L::V + v_off, st + v_rows, L::VP, p.out + (static_cast<int64_t>(info.y) + w * 16) * p.o_t + h * p.o_h + col, p.o_t,
                     ok ? info.z - w * 16 : 0, lane);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[stage]);
    if (++stage == GW_STAGES) stage = 0, full_parity ^= 1;
    if ((info.w & 1) && ok) {
      float* to = p.state + static_cast<int64_t>(bh) * GDN_D * GDN_D + w * 32 * GDN_D + col;
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          to[(n * 8 + c2 + (j & 1)) * GDN_D + gr + (j >> 1) * 8] = S[n][j];
          S[n][j] = 0.f;
        }
    }
  }
  if (lane == 0) atomicExch(p.err, 1);
}

int64_t walk_slots(int batch, int total_tokens) { return static_cast<int64_t>(total_tokens) / CHUNK + batch; }
// Slots of a window: at most 1 GiB of them, as in the other walks (51 thousand chunks of a head, 3.3 million tokens).
int64_t window_slots(int batch, int total_tokens, int heads) {
  const int64_t slots = walk_slots(batch, total_tokens), most = (int64_t{1} << 30) / (static_cast<int64_t>(heads) * GW_SLOT_BYTES);
  return slots <= most ? slots : most > 0 ? most : 1;
}

// `items_per_head` CTAs' worth of work per head and sequence, at most one CTA per SM
int launch_walk(void (*kernel)(GdnWalkParams), int threads, int smem, int items_per_head, GdnWalkParams p, cudaStream_t st) {
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return fail(ERR_RUNTIME, "gdn_chunked_prefill_walk: cannot raise dynamic shared memory to %d", smem);
  p.items = p.batch * p.heads * items_per_head;
  const cudaError_t err = launch_pdl(true, kernel, dim3(p.items < sm_count() ? p.items : sm_count()), dim3(threads), smem, st, p);
  if (err != cudaSuccess) return fail(ERR_LAUNCH, "gdn_chunked_prefill_walk: %s", cudaGetErrorString(err));
  return check_launch("gdn_chunked_prefill_walk");
}

// The two launches of a window
template <bool WINDOWS>
int prep_and_walk(const GdnWalkParams& p, cudaStream_t st) {
  gdn_walk_prep_kernel<<<dim3(p.to - p.from, p.heads), GP_THREADS, GP_SMEM, st>>>(p);
  if (const int rc = check_launch("gdn_chunked_prefill_walk (prep)")) return rc;
  const int pairs = p.heads * p.batch, sms = sm_count();
  constexpr int copy = 32 * GW_COPY_WARPS;
  // What fills the device: four warps per 16 value columns while that leaves SMs free (one sequence of 2048 tokens: 77 us against
  // 122 on half-head CTAs and 199 on whole heads), two such teams per CTA (2 x 1000..3000: 114 against 135 and 215), half a head
  // per CTA (4 x 2048: 148 against 214 in teams and 225 on whole heads), whole heads (8 x 1024: 133 against 148).
  if (pairs * 8 <= sms) return launch_walk(gdn_walk_team_kernel<1, WINDOWS>, TeamSmem<1>::THREADS, TeamSmem<1>::BYTES, 8, p, st);
  if (pairs * 4 <= sms) return launch_walk(gdn_walk_team_kernel<2, WINDOWS>, TeamSmem<2>::THREADS, TeamSmem<2>::BYTES, 4, p, st);
  if (pairs * 2 <= sms) return launch_walk(gdn_walk_kernel<4, WINDOWS>, 128 + copy, WalkSmem<64>::BYTES, 2, p, st);
  return launch_walk(gdn_walk_kernel<8, WINDOWS>, 256 + copy, WalkSmem<128>::BYTES, 1, p, st);
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" int64_t b200_gdn_chunked_prefill_walk_workspace_bytes(int32_t batch, int32_t total_tokens, int32_t num_heads) {
  return window_slots(batch, total_tokens, num_heads) * num_heads * GW_SLOT_BYTES + 16;
}

extern "C" int b200_gdn_chunked_prefill_walk(const void* q, int64_t q_stride_t, int64_t q_stride_h, const void* k, int64_t k_stride_t,
                                             int64_t k_stride_h, const void* v, int64_t v_stride_t, int64_t v_stride_h, const float* beta,
                                             int64_t beta_stride_t, int64_t beta_stride_h, const float* g, int64_t g_stride_t,
                                             int64_t g_stride_h, const int32_t* cu_seqlens, int32_t batch, int32_t total_tokens,
                                             void* workspace, float* state, void* out, int64_t out_stride_t, int64_t out_stride_h,
                                             int32_t num_heads, int32_t key_dim, int32_t value_dim, b200_stream_t stream) {
  B200_REQUIRE(batch > 0 && batch <= 65535 && total_tokens > 0 && num_heads > 0 && num_heads <= 65535,
               "gdn_chunked_prefill_walk: bad shape");
  B200_REQUIRE(static_cast<int64_t>(batch) * num_heads < (1 << 28), "gdn_chunked_prefill_walk: too many heads and sequences");
  B200_REQUIRE(key_dim == GDN_D && value_dim == GDN_D, "gdn_chunked_prefill_walk: key/value dim must be %d (got %d/%d)", GDN_D, key_dim,
               value_dim);
  B200_REQUIRE(cu_seqlens != nullptr && workspace != nullptr && aligned16(workspace),
               "gdn_chunked_prefill_walk: cu_seqlens and a 16-byte aligned workspace are required");
  B200_REQUIRE(aligned16(out) && aligned16(state) && out_stride_t % 8 == 0 && out_stride_h % 8 == 0,
               "gdn_chunked_prefill_walk: out and state must be 16-byte aligned, out strides multiples of 8 elements");
  B200_REQUIRE(aligned16(q) && aligned16(k) && aligned16(v) && q_stride_t % 8 == 0 && k_stride_t % 8 == 0 && v_stride_t % 8 == 0 &&
                   q_stride_h % 8 == 0 && k_stride_h % 8 == 0 && v_stride_h % 8 == 0,
               "gdn_chunked_prefill_walk: q/k/v must be 16-byte aligned with token and head strides that are multiples of 8 elements");
  GdnWalkParams p;
  p.q = static_cast<const __nv_bfloat16*>(q), p.q_t = q_stride_t, p.q_h = q_stride_h;
  p.k = static_cast<const __nv_bfloat16*>(k), p.k_t = k_stride_t, p.k_h = k_stride_h;
  p.v = static_cast<const __nv_bfloat16*>(v), p.v_t = v_stride_t, p.v_h = v_stride_h;
  p.beta = beta, p.be_t = beta_stride_t, p.be_h = beta_stride_h;
  p.g = g, p.g_t = g_stride_t, p.g_h = g_stride_h;
  p.cu = cu_seqlens, p.ws = static_cast<uint8_t*>(workspace), p.state = state;
  p.out = static_cast<__nv_bfloat16*>(out), p.o_t = out_stride_t, p.o_h = out_stride_h;
  p.heads = num_heads, p.batch = batch, p.slots = static_cast<int>(walk_slots(batch, total_tokens));
  const int window = static_cast<int>(window_slots(batch, total_tokens, num_heads));
  p.next = reinterpret_cast<int*>(p.ws + static_cast<int64_t>(window) * num_heads * GW_SLOT_BYTES);
  p.err = wait_timeout_flag();
  if (!p.err) return fail(ERR_RUNTIME, "gdn_chunked_prefill_walk: no error flag");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (window == p.slots) {
    p.from = 0, p.to = p.slots;
    return prep_and_walk<false>(p, st);
  }
  for (p.from = 0; p.from < p.slots; p.from = p.to) {
    p.to = p.slots - p.from < window ? p.slots : p.from + window;
    if (const int rc = prep_and_walk<true>(p, st)) return rc;
  }
  return OK;
}
