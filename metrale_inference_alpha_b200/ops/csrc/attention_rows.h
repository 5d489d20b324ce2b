// Prefill attention of attention_rows.cu, called by mb_attn_prefill_tc for the calls that it serves.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>

struct AttnRowsParams {
  const __nv_bfloat16* q;    // [rows, Hq, 128]
  const void* k_cache;       // [blocks, block, Hkv, 128] bf16 or e4m3
  const void* v_cache;
  const int* block_table;
  int max_blocks;
  const int* q_start;
  const int* q_len;
  const int* ctx_len;
  int Hq, Hkv, block_size;
  long long num_blocks;
  float scale;
  const float* k_scale;
  const float* v_scale;
  __nv_bfloat16* out;        // [rows, out_ld]: head h at columns h * 128
  long long out_ld;
  uint8_t* outq;             // instead of `out`: NVFP4 with a calibrated global scale, as in MbGemmArgs
  int ldq;
  uint8_t* outq_sf;
  int outq_sf_k64;
  float outq_gs;
  uint32_t* status;
};

int mb_attn_rows(const AttnRowsParams& p, int max_q_len, int num_seqs, bool fp8, cudaStream_t stream);
// the same at head dim 256, bf16 cache and output (attention_rows256.cu)
int mb_attn_rows256(const AttnRowsParams& p, int max_q_len, int num_seqs, cudaStream_t stream);
