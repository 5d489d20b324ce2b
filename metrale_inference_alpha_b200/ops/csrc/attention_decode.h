// Decode / verify attention of attention_decode.cu, called by mb_paged_attention for the calls that it serves.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>

struct AttnDecodeArgs {
  const __nv_bfloat16* q;     // [rows, Hq, D]
  const void* k_cache;        // [blocks, block, Hkv, D] bf16 or e4m3
  const void* v_cache;
  const int* block_table;
  int max_blocks;
  const int* q_start;
  const int* q_len;
  const int* ctx_len;
  int num_seqs, max_q_len, max_ctx, Hq, Hkv, D, block_size, fp8;
  long long num_blocks;
  float scale;
  const float* k_scale;
  const float* v_scale;
  __nv_bfloat16* out;         // [rows, out_ld]: head h at columns h * D
  long long out_ld;
  uint8_t* outq;              // instead of `out`: NVFP4 with a calibrated global scale, as in MbGemmArgs
  int ldq;
  uint8_t* outq_sf;
  int outq_sf_k64;
  float outq_gs;
  void* ws;
  size_t ws_bytes;
  int total_rows, part_tokens;   // part_tokens 0 = default
  int sm_count;
  // the kernel in front wrote q and the cache's rows of this step's tokens (the last q_len of every context) and nothing else that is
  // read here, and launches its dependents early
  int early;
  uint32_t* status;
};

// CTAs of a launch that an SM holds, and the shared memory of each (D 128 or 256; rows = tokens x heads of a group)
extern "C" int mb_attn_decode_per_sm(int D, int fp8, int rows, int num_seqs, size_t* smem);
bool mb_attn_decode_serves(const AttnDecodeArgs& a);
size_t mb_attn_decode_ws(const AttnDecodeArgs& a);
int mb_attn_decode(const AttnDecodeArgs& a, cudaStream_t stream);
