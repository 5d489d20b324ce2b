// Grouped expert GEMM of few token rows an expert (decode, short prompts), fp8 with 128 x 128 weight scales, sm_100a:
//     out[r, n] = sum over k blocks of a_scale[kb, r] * w_scale[e, n / 128, kb] * (X[r, kb] . W[e, n, kb])
// for the entries (expert e, first row, rows) of a work list, each of at most TN = 16, 32 or 64 rows.
//
// Bound by the stream of the weights: an entry reads its expert's whole matrix for a row or two. The 128-row tiles of gemm_rows.cu
// carry every k block of an entry through 128 x 128 sums of which one or two rows are real, and a tile ends in an epilogue that
// nothing runs under. Here the weights are the UMMA "A" operand (128 features) and the entry's rows the "B" operand, so a sum
// is TN columns; eight of them lie in TMEM, four for each of two groups of epilogue warps that take the tiles in turn, so that one
// group's waits (the work list, the scales, the stores) run under the other's sums and the copies never pause. (Eight sums shared by
// both would not do: a group waits for its own tiles' alone, and a barrier's parity does not tell it whether the phase in between
// has been.) Persistent, one CTA per SM, all of shared memory for stages.
// Measured against the 128-row tiles (us, 256 experts, 8 of them a token, 1024 x 2048 / 2048 x 512): entries of 16 rows, 1 token 10.9 -> 9.0 /
// 11.6 -> 9.9, 16 tokens 49 -> 39 / 33 -> 22, 512 tokens 186 -> 98 / 121 -> 66; of 32, 1024 tokens 203 -> 111 / 133 -> 74; of 64, 2047
// tokens 196 -> 141 / 123 -> 111.
#include "common.cuh"
#include "gemm_rows.h"
#include "tensormap.h"

namespace {

struct FewParams {
  int num_kb, n_tiles, items, n_per_expert;
  long long ldo;
  void* out;
  int out_f32;
  const float* w_scale;      // [experts * n_per_expert / 128, k blocks]
  const float* a_scale;      // [k blocks, a_ld]
  int a_ld;
  const int* tile_expert;
  const int* tile_row0;
  const int* tile_nrows;
  uint32_t* status;
};

constexpr int kFewThreads = 320;   // producer warp, MMA warp, two groups of four epilogue warps
constexpr int kChunk = 16;         // k blocks whose scales are staged together

template <int TN>
struct FewCfg {
  static constexpr int kABytes = 128 * 128, kBBytes = TN * 128, kStageBytes = kABytes + kBBytes;
  static constexpr int kScaleBytes = 2 * kChunk * TN * 4;
  static constexpr int kStagesRaw = (216 * 1024 - kScaleBytes) / kStageBytes;
  static constexpr int kStages = kStagesRaw > 12 ? 12 : kStagesRaw;
  static constexpr int kAccs = 4;                            // of a group
  static constexpr int kTmemCols = 2 * kAccs * TN;
  static constexpr int kSmem = kStages * kStageBytes + kScaleBytes + 1024;
};

template <int TN>
__global__ void __launch_bounds__(kFewThreads, 1)
gemm_few_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const FewParams p) {
  using C = FewCfg<TN>;
  constexpr int kStages = C::kStages, kAccs = C::kAccs;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* s_scale = reinterpret_cast<float*>(smem + kStages * C::kStageBytes);    // [group][k block of the chunk][row]
  __shared__ __align__(8) uint64_t full_bar[kStages];
  __shared__ __align__(8) uint64_t empty_bar[kStages];
  __shared__ __align__(8) uint64_t acc_full[2 * kAccs];
  __shared__ __align__(8) uint64_t acc_empty[2 * kAccs];
  __shared__ uint32_t tmem_base_s;
  const int warp = threadIdx.x >> 5, nkb = p.num_kb;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mb::mbar_init(&full_bar[s], 1);
      mb::mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2 * kAccs; ++i) {
      mb::mbar_init(&acc_full[i], 1);
      mb::mbar_init(&acc_empty[i], 4);
    }
    mb::mbar_fence_init();
    mb::tma_prefetch_desc(&tmW);
    mb::tma_prefetch_desc(&tmX);
  }
  if (warp == 1) mb::tmem_alloc(&tmem_base_s, C::kTmemCols);
  mb::tc_fence_before();
  __syncthreads();
  mb::tc_fence_after();
  const uint32_t tmem = tmem_base_s;
  mb::pdl_launch_dependents();
  // The work list, the rows and their scales come from preceding kernels, which may write them while this CTA is up: ordinary loads.
  mb::pdl_wait();

  // item i: entry i / n_tiles, features (i % n_tiles) * 128; entries without rows are passed over by every role alike
  if (warp == 0) {
    if (mb::elect_one()) {
      int g = 0;
      bool ok = true;
      for (int i = blockIdx.x; i < p.items && ok; i += gridDim.x) {
        const int mt = i / p.n_tiles, e = p.tile_expert[mt], row0 = p.tile_row0[mt];
        if (e < 0) continue;
        const int w_row0 = e * p.n_per_expert + (i - mt * p.n_tiles) * 128;
        for (int kb = 0; kb < nkb; ++kb, ++g) {
          const int s = g % kStages;
          ok = mb::mbar_wait(&empty_bar[s], ((g / kStages) & 1) ^ 1, p.status, MB_ST_TIMEOUT_TMA);
          if (!ok) break;
          uint8_t* st = smem + s * C::kStageBytes;
          mb::mbar_expect_tx(&full_bar[s], C::kStageBytes);
          mb::tma_load_2d(st, &tmW, &full_bar[s], kb * 128, w_row0);
          mb::tma_load_2d(st + C::kABytes, &tmX, &full_bar[s], kb * 128, row0);
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (mb::elect_one()) {
      constexpr uint32_t idesc = mb::umma_idesc(0, 0, 128, TN);
      int g = 0, turn = 0, mine[2] = {0, 0};                 // k blocks so far: all, and of either group's tiles
      bool ok = true;
      for (int i = blockIdx.x; i < p.items && ok; i += gridDim.x) {
        if (p.tile_expert[i / p.n_tiles] < 0) continue;
        const int group = turn++ & 1;
        int a = group ? mine[1] : mine[0];
        for (int kb = 0; kb < nkb; ++kb, ++g, ++a) {
          const int s = g % kStages, buf = group * kAccs + a % kAccs;
          ok = mb::mbar_wait(&acc_empty[buf], ((a / kAccs) & 1) ^ 1, p.status, MB_ST_TIMEOUT_MMA) &&
               mb::mbar_wait(&full_bar[s], (g / kStages) & 1, p.status, MB_ST_TIMEOUT_MMA);
          if (!ok) break;
          mb::tc_fence_after();
          const uint32_t a_base = mb::smem_u32(smem + s * C::kStageBytes), b_base = a_base + C::kABytes;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            mb::umma_f8f6f4(tmem + buf * TN, mb::umma_desc_sw128(a_base + j * 32), mb::umma_desc_sw128(b_base + j * 32), idesc, j != 0);
          mb::tc_commit(&empty_bar[s]);
          mb::tc_commit(&acc_full[buf]);
        }
        if (group) mine[1] = a;
        else mine[0] = a;
      }
    }
    __syncwarp();
  } else {
    const int group = (warp - 2) >> 2, q = warp & 3, lane = threadIdx.x & 31;
    const int et = (threadIdx.x - 64) & 127;
    const uint32_t src = tmem + ((uint32_t)(q * 32) << 16);
    float* sc = s_scale + group * (kChunk * TN);
    auto sync_group = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); };
    // ... and whether every warp of the group saw its sums: one whose wait ran out takes the others with it
    auto sync_group_all = [&](bool mine) {
      int all;
      asm volatile("{.reg .pred p, q; setp.ne.s32 p, %1, 0; bar.red.and.pred q, %2, 128, p; selp.s32 %0, 1, 0, q;}"
                   : "=r"(all) : "r"((int)mine), "r"(1 + group) : "memory");
      return all != 0;
    };
    int a = 0, turn = 0;                                     // k blocks of this group's tiles so far, tiles of this CTA
    bool ok = true;
    for (int i = blockIdx.x; i < p.items && ok; i += gridDim.x) {
      const int mt = i / p.n_tiles, nt = i - mt * p.n_tiles, e = p.tile_expert[mt];
      if (e < 0) continue;
      if ((turn++ & 1) != group) continue;
      const int row0 = p.tile_row0[mt], rows = p.tile_nrows[mt];
      const float* wsp = p.w_scale + (size_t)((e * p.n_per_expert >> 7) + nt) * nkb;
      float acc[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[j] = 0.f;
      for (int k0 = 0; k0 < nkb && ok; k0 += kChunk) {
        const int kc = min(kChunk, nkb - k0);
        for (int x = et; x < kc * TN; x += 128) {
          const int kb = x / TN, r = x % TN;
          sc[x] = r < rows ? p.a_scale[(size_t)(k0 + kb) * p.a_ld + row0 + r] * __ldg(wsp + k0 + kb) : 0.f;
        }
        sync_group();
        for (int kb = 0; kb < kc; ++kb, ++a) {
          const int buf = group * kAccs + a % kAccs;
          ok = mb::mbar_wait(&acc_full[buf], (a / kAccs) & 1, p.status, MB_ST_TIMEOUT_EPI);
          if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
          mb::tc_fence_after();
#pragma unroll
          for (int c = 0; c < TN; c += 16) {
            float v[16];
            mb::tmem_ld16(src + buf * TN + c, v);
            if (c + 16 == TN) {                              // the accumulator is free
              mb::tc_fence_before();
              __syncwarp();
              if (lane == 0) mb::mbar_arrive(&acc_empty[buf]);
            }
            const float4* s4 = reinterpret_cast<const float4*>(sc + kb * TN + c);
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const float4 f = s4[h];
              acc[c + 4 * h] = fmaf(v[4 * h], f.x, acc[c + 4 * h]);
              acc[c + 4 * h + 1] = fmaf(v[4 * h + 1], f.y, acc[c + 4 * h + 1]);
              acc[c + 4 * h + 2] = fmaf(v[4 * h + 2], f.z, acc[c + 4 * h + 2]);
              acc[c + 4 * h + 3] = fmaf(v[4 * h + 3], f.w, acc[c + 4 * h + 3]);
            }
          }
        }
        ok = sync_group_all(ok);                             // the scales may be replaced
      }
      if (ok) {
        // a lane is a feature: a row's 32 are one piece of a line
        const size_t at = (size_t)row0 * p.ldo + nt * 128 + q * 32 + lane;
        if (p.out_f32) {
          float* o = reinterpret_cast<float*>(p.out) + at;
#pragma unroll
          for (int j = 0; j < TN; ++j)
            if (j < rows) o[(size_t)j * p.ldo] = acc[j];
        } else {
          __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + at;
#pragma unroll
          for (int j = 0; j < TN; ++j)
            if (j < rows) o[(size_t)j * p.ldo] = __float2bfloat16(acc[j]);
        }
      }
    }
    mb::tc_fence_before();
  }
  __syncthreads();
  if (warp == 1) {
    mb::tc_fence_after();
    mb::tmem_dealloc(tmem, C::kTmemCols);
  }
}

template <int TN>
int launch_few(const CUtensorMap* tm, const FewParams& p, int grid, cudaStream_t stream) {
  auto kern = gemm_few_kernel<TN>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FewCfg<TN>::kSmem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  return (int)mb::launch_kernel_cluster(kern, dim3(grid), dim3(kFewThreads), FewCfg<TN>::kSmem, stream, 1, tm[0], tm[1], p);
}

}  // namespace

bool mb_gemm_few_serves(const MbGemmArgs* a, int rows) {
  return a->tile_expert && (rows == 16 || rows == 32 || rows == 64) && a->n_per_expert % 128 == 0 && !a->residual;
}

int mb_gemm_few(const MbGemmArgs* a, int rows, cudaStream_t stream) {
  FewParams p{};
  p.num_kb = (a->K + 127) / 128;
  p.n_tiles = a->n_per_expert / 128;
  p.n_per_expert = a->n_per_expert;
  const long long items = (long long)a->max_tiles * p.n_tiles;
  if (items > 0x7fffffff) return MB_ERR_TOO_LARGE;
  p.items = (int)items;
  p.ldo = a->ldo; p.out = a->out; p.out_f32 = a->out_f32;
  p.w_scale = a->w_scale; p.a_scale = a->a_scale; p.a_ld = a->a_ld;
  p.tile_expert = a->tile_expert; p.tile_row0 = a->tile_row0; p.tile_nrows = a->tile_nrows;
  p.status = a->status;
  CUtensorMap tm[2];
  int rc;
  if ((rc = mbh::encode_2d(&tm[0], CU_TENSOR_MAP_DATA_TYPE_UINT8, a->W, (uint64_t)a->K, (uint64_t)a->N, (size_t)a->K, 128, 128))) return rc;
  if ((rc = mbh::encode_2d(&tm[1], CU_TENSOR_MAP_DATA_TYPE_UINT8, a->X, (uint64_t)a->K, (uint64_t)a->M, (size_t)a->K, 128, (uint32_t)rows))) return rc;
  const int sms = a->sm_count > 0 ? a->sm_count : 148, grid = items < sms ? (int)items : sms;
  if (rows == 16) return launch_few<16>(tm, p, grid, stream);
  if (rows == 32) return launch_few<32>(tm, p, grid, stream);
  return launch_few<64>(tm, p, grid, stream);
}
