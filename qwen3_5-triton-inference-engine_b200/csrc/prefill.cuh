// Prefill attention: what its two kernels share.  prefill_umma.cu: pairs of CTAs that work through a list of items; prefill_short.cu: one CTA to
// every block of 32 query tokens, for calls that are over in one wave.
#pragma once
#include "b200_attn.h"
#include "umma.cuh"

namespace b200 {

constexpr int PU_BQ = 32;                           // query tokens per CTA
constexpr int PU_TKV = 128;                         // tokens of a K/V tile
constexpr uint32_t PU_TMEM_COLS = 512;              // S0 [0,128) S1 [128,256) (P over their first 64) O [256,512)
constexpr float PU_TAU = 8.0f;                      // lazy-rescale threshold (log2 domain)

struct PrefillUmmaParams {
  int num_kv_heads, batch, max_seqlen, group;  // group: sequences whose items are dealt together (pairs)
  __nv_bfloat16* out;
  int64_t out_t, out_h;
  const int32_t* cu_seqlens;
  int* err;
  float scale_log2;
  // fused form only: rotary embedding of q in shared memory, sigmoid gate in the epilogue
  const __nv_bfloat16* gate;
  int64_t gate_t;
  const void* position_ids;
  int ids_are_int64;
  const float* inv_freq;
};

struct PrefillTensors {  // [tokens, heads, 256] each, strides in elements
  const void *q, *k, *v;
  int64_t q_t, q_h, k_t, k_h, v_t, v_h;
  int tokens, num_kv_heads;
};

// q as {64 cols, 4 heads of a group, groups, tokens, 4 column blocks}; one load = 32 tokens of one group
inline bool encode_prefill_q(CUtensorMap* map, const PrefillTensors& t) {
  const uint64_t dims[5] = {64, GROUP, static_cast<uint64_t>(t.num_kv_heads), static_cast<uint64_t>(t.tokens), HEAD_DIM / 64};
  const uint64_t strides[4] = {static_cast<uint64_t>(t.q_h) * 2, static_cast<uint64_t>(t.q_h) * 2 * GROUP, static_cast<uint64_t>(t.q_t) * 2, 128};
  const uint32_t box[5] = {64, GROUP, 1, PU_BQ, HEAD_DIM / 64};
  return encode_map_bf16_sw128(map, t.q, 5, dims, strides, box);
}
// k or v as {64 cols, tokens, 4 column blocks, kv heads}; one load = `tokens` tokens, `blocks` column blocks of one head
inline bool encode_prefill_kv(CUtensorMap* map, const PrefillTensors& t, const void* base, int64_t stride_t, int64_t stride_h, uint32_t tokens,
                              uint32_t blocks) {
  const uint64_t dims[4] = {64, static_cast<uint64_t>(t.tokens), HEAD_DIM / 64, static_cast<uint64_t>(t.num_kv_heads)};
  const uint64_t strides[3] = {static_cast<uint64_t>(stride_t) * 2, 128, static_cast<uint64_t>(stride_h) * 2};
  const uint32_t box[4] = {64, tokens, blocks, 1};
  return encode_map_bf16_sw128(map, base, 4, dims, strides, box);
}

// Whether a call is the one-CTA kernel's, and its launch (everything in `p` but `group` set).
bool prefill_takes_short(bool fused, int batch, int total_tokens, int max_seqlen, int num_kv_heads);
int launch_prefill_short(bool fused, const PrefillTensors& t, const PrefillUmmaParams& p, cudaStream_t stream, const char* what);

}  // namespace b200
