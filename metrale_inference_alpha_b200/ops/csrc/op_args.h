// Argument blocks of the row, rotation and attention launchers: one definition shared by the kernel files, by the native callers
// (dense_layer.cu) and mirrored field for field by the ctypes binding (ops/_native.py).
#pragma once
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>

struct MbRowArgs {
  int M, K, in_mode, out_mode;
  const void* x;
  long long x_ld;
  const void* residual;
  void* residual_out;
  const void* w;
  int w_plus_one;
  float eps;
  const void* gate;
  long long gate_ld;
  int head_dim, gate_head_stride, gate_head_off, group;
  const float* xf32;
  void* out;
  long long out_ld;
  void* out_bf16;
  long long out_bf16_ld;
  float* scale;
  int scale_ld;
  void* sf;
  int sf_k64;
  float static_gs;
  const int* row_index;
  const void* gather;
  int gather_wide;
  long long gather_rows;
  void* gather_out;
  uint32_t* status;
};

struct MbRopeKvArgs {
  int M, Hq, Hkv, D, rot;
  const void* qkv;
  long long qkv_ld;
  int q_head_stride, k_off, v_off;
  const int* positions;
  const long long* slots;
  const void* q_norm_w;
  const void* k_norm_w;
  int norm_plus_one;
  float eps;
  const float* cos_tab;
  const float* sin_tab;
  int max_pos;
  void* q_out;
  void* k_cache;
  void* v_cache;
  int cache_fp8;
  const float* k_scale;
  const float* v_scale;
  long long num_slots;
  uint32_t* status;
  float* amax;             // optional [2] running max |k|, |v| of the written rows
  int early;               // the kernel in front wrote qkv and nothing else that is read here, and launches its dependents early
};

struct MbAttnArgs {
  const void* q;
  const void* k_cache;
  const void* v_cache;
  const int* block_table;
  int max_blocks;
  const int* q_start;
  const int* q_len;
  const int* ctx_len;
  int num_seqs, max_q_len, max_ctx;
  int Hq, Hkv, D, block_size;
  long long num_blocks;
  float scale;
  int cache_fp8;
  const float* k_scale;
  const float* v_scale;
  void* out;
  void* ws;                // split-KV partials
  size_t ws_bytes;
  int total_rows;          // query rows (for workspace sizing)
  int part_tokens;         // 0 = default 512
  int window;
  int force_mode;          // 0 auto, 1 split-KV, 2 split-Q
  uint32_t* status;
  void* outq;              // optional NVFP4 output (split-KV path only; MB_ERR_UNSUPPORTED otherwise)
  int ldq;
  void* outq_sf;
  int outq_sf_k64;
  float outq_gs;
  // separate value head size and softmax variants (all zero = values as wide as keys, plain softmax)
  int DV;                  // padded value row of the cache (0 = D); bf16 caches
  int dv;                  // value columns stored per head (0 = DV)
  long long out_ld;        // elements between output rows (0 = Hq * dv)
  float out_scale;         // 0 = 1
  int sink, split_p;
  const float* sink_w;     // [Hq] sink scores (null: 0), with sink
  int keep;                // with window: first tokens that stay visible
  const void* gate;        // logits of sigmoid gates on the output (bf16), or null
  long long gate_ld;
  int gate_mode;           // 1 one per head, 2 one per element
  float softcap;           // 0: off; scores become softcap tanh(score / softcap)
  const float* turn_cos;   // [turn_max, dv / 2] or null: every output row is turned back by its position
  const float* turn_sin;
  int turn_max;
  int part_fixed;          // partition size that the caller insists on for the plain decode kernel too (0 = its own)
  int sm_count;
  int early;               // see AttnDecodeArgs
};

struct MbAttnTcArgs {
  const void* q;
  const void* k_cache;
  const void* v_cache;
  const int* block_table;
  const int* q_start;
  const int* q_len;
  const int* ctx_len;
  const float* k_scale;
  const float* v_scale;
  void* out;
  uint32_t* status;
  long long num_blocks;
  int max_blocks, num_seqs, max_q_len, Hq, Hkv, D, block_size, cache_fp8;
  float scale;
  int v_mn;      // 1: V staged as stored and read as an MN-major operand (no transposition)
  long long out_ld;    // elements between output rows (0 = Hq * D)
  float out_scale;     // 0 = 1
  int sink, split_p;
  const float* sink_w; // [Hq] sink scores (null: 0), with sink
  int window, keep;    // 0 = no window; the first `keep` tokens stay visible
  const void* gate;    // logits of sigmoid gates on the output (bf16), or null
  long long gate_ld;
  int gate_mode;       // 1 one per head, 2 one per element
  float softcap;       // 0: off
  const float* turn_cos;   // [turn_max, D / 2] or null: every output row is turned back by its position
  const float* turn_sin;
  int turn_max;
  void* outq;          // plain attention at head dim 128 only: the output as NVFP4 instead of `out`, see MbGemmArgs
  int ldq;
  void* outq_sf;
  int outq_sf_k64;
  float outq_gs;
};

extern "C" {
int mb_row_op(const MbRowArgs* a, cudaStream_t stream);
int mb_qk_norm_rope_kvwrite(const MbRopeKvArgs* a, cudaStream_t stream);
int mb_paged_attention(const MbAttnArgs* a, cudaStream_t stream);
size_t mb_attn_ws_need(const MbAttnArgs* a);
int mb_attn_prefill_tc(const MbAttnTcArgs* a, cudaStream_t stream);
}
