// The GEMM of many token rows (gemm_rows.cu), called by mb_gemm once it has checked the arguments.
#pragma once
#include "gemm_args.h"

// Ranges of K that a GEMM of one tile per CTA (gemm_tcgen05.cu) is cut into when the caller names no number.
extern "C" int mb_gemm_auto_splits(int tiles, int num_kb, int sms, bool clusters);
// Whether gemm_rows.cu serves this call.
bool mb_gemm_rows_serves(const MbGemmArgs* a);
// `tn`: mb_gemm's token tile, for grouped calls the most rows of an entry of the work list
int mb_gemm_rows(const MbGemmArgs* a, int tn, cudaStream_t stream);
// fp8 blocks over a work list of entries of at most `rows` (16, 32 or 64) rows each (gemm_few.cu)
bool mb_gemm_few_serves(const MbGemmArgs* a, int rows);
int mb_gemm_few(const MbGemmArgs* a, int rows, cudaStream_t stream);
