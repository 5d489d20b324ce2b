// The GEMM of many token rows (gemm_rows.cu), called by mb_gemm once it has checked the arguments.
#pragma once
#include "gemm_args.h"

// Whether gemm_rows.cu serves this call. `splits_forced`: the caller asked for a split-K count.
bool mb_gemm_rows_serves(const MbGemmArgs* a);
// `tn`: mb_gemm's token tile, for grouped calls the most rows of an entry of the work list
int mb_gemm_rows(const MbGemmArgs* a, int tn, cudaStream_t stream);
