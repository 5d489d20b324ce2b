// Linear layer over many token rows (prompts, portions of prompts, experts' rows), sm_100a:
//     out[m, n] = epilogue( sum_k X[m, k] * W[n, k] )
// The other way round than gemm_tcgen05.cu: the token tile is the UMMA "A" operand, so a TMEM lane is a token and a
// thread of the epilogue holds 64 or 128 neighbouring features of one token: gate / up pairs, the 16 values of an
// NVFP4 block and 16-byte stores are all inside a thread, without shuffles or a staging tile.
//
// gemm_pair_kernel (bf16, fp8 per row, NVFP4): a pair of CTAs owns a tile of 256 tokens x BN features
// (tcgen05.mma.cta_group::2, M = 256). Each CTA stages its own 128 tokens and half of the features, so a byte in shared
// memory feeds twice the products of a 128 x 128 tile of one CTA, whose operand reads (128 bytes a cycle at the fp4 rate)
// were what bounded prefill. Persistent: pairs walk tiles with token tiles fastest (the pairs that run together share
// weight tiles in L2) and the stage ring runs on across tiles. bf16 and fp8 have two accumulators; NVFP4 at BN = 256 has
// one, since two of 256 columns and the scale factors are more than TMEM's 512 columns: there the eight epilogue warps
// take the whole accumulator into registers at once and hand it back before they scale and store.
// Measured (B200, 8192 tokens; before = 128 x 128 tiles of one CTA): NVFP4 7168 x 5120 228 -> 139 us, 34816 x 5120 with
// SwiGLU 990 -> 570 us (5.1 PFLOP/s), 5120 x 17408 499 -> 302 us; bf16, 2532 tokens: 34816 x 5120 708 -> 567 us (1.5 PFLOP/s,
// under the power cap). The SwiGLU result leaves as NVFP4 from here too: the 134 us quantiser pass over 8192 x 17408 is gone.
//
// gemm_block_kernel (fp8 with 128 x 128 weight scales, also over the work list of grouped experts): one CTA per tile of
// 128 tokens x 128 or 256 features. Every 128-deep k block lands in one of four or two TMEM accumulators and is added to registers
// with its scale, which is one number per thread here (the token's scale times the weight block's). Work lists of entries of 16 to
// 64 rows are gemm_few.cu's; only where a residual joins the result do they come here, in boxes of their own rows: the rest of the
// tile's rows are whatever was there, and are not stored.
// Measured (2724 tokens x 8 of 256 experts and a shared one; before = 64-token tiles as the UMMA "B" operand): 1024 x 2048 per
// expert 500 -> 134 us (167 at 128 features a tile), 2048 x 512 417 -> 122 us (144), plain 8192 x 2048 237 -> 64 us (82).
#include "common.cuh"
#include "epilogue.cuh"
#include "gemm_rows.h"
#include "tensormap.h"
#include <type_traits>

namespace {

enum { KIND_BF16 = 0, KIND_FP8 = 1, KIND_NVFP4 = 2, KIND_FP8_BLOCK = 3 };

struct RowsParams {
  int M, N, num_kb, m_tiles, n_tiles;
  long long ldo;
  void* out;
  const __nv_bfloat16* residual;
  const float* w_scale;      // per feature or null; fp8 block: [features / 128, k blocks]
  const float* a_scale;      // per token or null; fp8 block: [k blocks, a_ld]
  float a_static;            // every token's scale where a_scale is null (not fp8 block)
  int a_ld;
  float alpha;
  int epilogue, out_f32, vec;   // vec: rows of `out` (and `residual`) are whole 16-byte vectors (32-bit results: 32 bytes)
  int sectors;                  // rows of a bf16 `out` are whole 32-byte sectors
  float epi_a, epi_b;
  int epi_n;
  const float* epi_bias;
  uint8_t* outq;             // SwiGLU result as NVFP4, see MbGemmArgs
  int ldq;
  uint8_t* outq_sf;
  int outq_sf_k64;
  float outq_gs;
  int sfa_rows, sfb_rows;    // scale-factor map rows (256 bytes each) per 128 tokens / features
  uint32_t* status;
  const int* tile_expert;    // grouped
  const int* tile_row0;
  const int* tile_nrows;
  int n_per_expert, a_bytes; // a_bytes: bytes of a token tile's box
};

constexpr int kThreads = 320;      // producer warp, MMA warp, eight epilogue warps
constexpr int kEpiWarps = 8;

// A whole 32-byte sector: a thread stores its own token's features, so that a warp's store touches 32 lines, and 16 bytes of each
// would be half a sector. NVFP4, 8192 x 2048, 8192 tokens: 32-bit results 154 -> 103 us, bf16 117 -> 80;
// fp8 bf16 151 -> 111, bf16 operands 195 -> 176; 4096 x 5120: 83 -> 74, 123 -> 111, 230 -> 220.
__device__ __forceinline__ void store_sector(void* dst, const uint32_t* w) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]),
               "r"(w[6]), "r"(w[7])
               : "memory");
}
__device__ __forceinline__ void store_f32x8(float* dst, const float* y) { store_sector(dst, reinterpret_cast<const uint32_t*>(y)); }

// 16 results of one token at feature n (of n_limit): residual and store
__device__ __forceinline__ void emit16(const RowsParams& p, size_t m, int n, int n_limit, float* y, const uint4* res) {
  const size_t o = m * (size_t)p.ldo + n;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (n + 8 * h + 8 > n_limit) {
#pragma unroll
      for (int i = 8 * h; i < 8 * h + 8; ++i) {
        if (n + i < n_limit) {
          float v = y[i];
          if (p.residual) v += __bfloat162float(p.residual[o + i]);
          if (p.out_f32) reinterpret_cast<float*>(p.out)[o + i] = v;
          else reinterpret_cast<__nv_bfloat16*>(p.out)[o + i] = __float2bfloat16(v);
        }
      }
    } else if (p.residual) {
      const __nv_bfloat162* rb = reinterpret_cast<const __nv_bfloat162*>(res + h);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(rb[i]);
        y[8 * h + 2 * i] += f.x; y[8 * h + 2 * i + 1] += f.y;
      }
    }
  }
  if (n + 8 > n_limit) return;
  const bool both = n + 16 <= n_limit;
  if (p.out_f32) {
    float* dst = reinterpret_cast<float*>(p.out) + o;
    store_f32x8(dst, y);
    if (both) store_f32x8(dst + 8, y + 8);
    return;
  }
  uint32_t w[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(y[2 * i], y[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&b);
  }
  __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.out) + o;
  if (both && p.sectors) {
    store_sector(dst, w);
    return;
  }
  *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
  if (both) *(reinterpret_cast<uint4*>(dst) + 1) = make_uint4(w[4], w[5], w[6], w[7]);
}

// Rows that are not whole vectors start anywhere in one: a thread moves its features up by what its row lacks to the next 16-byte
// boundary, one step per bit of that, and stores whole vectors between single elements at both ends. With single stores throughout
// (32 lines a store, 64 or 128 of them a tile) NVFP4 rows of 4099 features, 5120 deep, took 78 us at 1300 tokens and 377 at 8192,
// fp8 blocks of 257 by 7168 54 us at 300 tokens; now 31, 103 and 39.
template <int NC, bool F32>
__device__ __forceinline__ void emit_shifted(const RowsParams& p, size_t m, int n0, int left, float* v) {
  using T = std::conditional_t<F32, float, __nv_bfloat16>;
  constexpr int kPer = F32 ? 1 : 2, kWords = NC / kPer, kVec = 8, kVecWords = kVec / kPer;     // elements of a word, of a vector (16 or 32 bytes)
  left = min(left, NC);
  const size_t o = m * (size_t)p.ldo + n0;
  if (p.residual) {
#pragma unroll
    for (int i = 0; i < NC; ++i) v[i] += i < left ? __bfloat162float(p.residual[o + i]) : 0.f;
  }
  uint32_t w[kWords];
#pragma unroll
  for (int i = 0; i < kWords; ++i) {
    if constexpr (F32) {
      w[i] = __float_as_uint(v[i]);
    } else {
      const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&b);
    }
  }
  T* dst = reinterpret_cast<T*>(p.out) + o;
  auto single = [&](int i) {                                 // element i of the words as they stand
    if constexpr (F32) dst[i] = __uint_as_float(w[i]);
    else reinterpret_cast<uint16_t*>(dst)[i] = (uint16_t)(w[i >> 1] >> (16 * (i & 1)));
  };
  const int lead = (int)((0u - (uint32_t)(reinterpret_cast<uintptr_t>(dst) / sizeof(T))) & (kVec - 1));
#pragma unroll
  for (int i = 0; i < kVec - 1; ++i)
    if (i < lead && i < left) single(i);
  if constexpr (!F32) {
#pragma unroll
    for (int i = 0; i < kWords; ++i) w[i] = lead & 1 ? __byte_perm(w[i], i + 1 < kWords ? w[i + 1] : 0, 0x5432) : w[i];
  }
  const int up = lead / kPer;
#pragma unroll
  for (int i = 0; i < kWords; ++i) w[i] = up & 1 ? (i + 1 < kWords ? w[i + 1] : 0) : w[i];
#pragma unroll
  for (int i = 0; i < kWords; ++i) w[i] = up & 2 ? (i + 2 < kWords ? w[i + 2] : 0) : w[i];
  if constexpr (F32) {
#pragma unroll
    for (int i = 0; i < kWords; ++i) w[i] = up & 4 ? (i + 4 < kWords ? w[i + 4] : 0) : w[i];
  }
  dst += lead;
  auto vector = [&](int i) {                                 // the words from i on
    if constexpr (F32) store_f32x8(dst, reinterpret_cast<const float*>(w + i));
    else *reinterpret_cast<uint4*>(dst) = make_uint4(w[i], w[i + 1], w[i + 2], w[i + 3]);
  };
  if (left == NC) {
#pragma unroll
    for (int k = 0; k < NC / kVec - 1; ++k, dst += kVec) vector(k * kVecWords);
#pragma unroll
    for (int i = 0; i < kVecWords; ++i) w[i] = w[kWords - kVecWords + i];
    left = kVec;
  }
#pragma unroll 1
  for (left -= lead; left > 0; left -= kVec, dst += kVec) {
    if (left >= kVec) vector(0);
#pragma unroll
    for (int i = 0; i < kVec - 1; ++i)
      if (left < kVec && i < left) single(i);
#pragma unroll
    for (int i = 0; i < kWords - kVecWords; ++i) w[i] = w[i + kVecWords];
  }
}

template <int NC>
__device__ __forceinline__ void emit_ragged(const RowsParams& p, size_t m, int n0, int n_limit, float* v) {
  if (n0 >= n_limit) return;
  if (p.out_f32) emit_shifted<NC, true>(p, m, n0, n_limit - n0, v);
  else emit_shifted<NC, false>(p, m, n0, n_limit - n0, v);
}

__device__ __forceinline__ uint4 residual8(const RowsParams& p, size_t m, int n, int n_limit) {
  if (p.residual && n + 8 <= n_limit) return __ldg(reinterpret_cast<const uint4*>(p.residual + m * (size_t)p.ldo + n));
  return make_uint4(0, 0, 0, 0);
}

// One token's NC features from n0 on, accumulator values in v. VEC: rows are whole vectors (a kernel of its own for other rows: their
// code in the same one cost NVFP4 prompts 3 %).
template <int KIND, int NC, bool VEC>
__device__ __forceinline__ void finish_row(const RowsParams& p, float (&v)[NC], int m, int n0, float as) {
  const bool glu = p.epilogue == mb::EPI_SWIGLU || (KIND == KIND_BF16 && (p.epilogue == mb::EPI_CLAMP_GLU || p.epilogue == mb::EPI_GEGLU));
  constexpr bool kWScale = KIND == KIND_FP8 || KIND == KIND_NVFP4;
  if (kWScale && p.w_scale) {
    if (n0 + NC <= p.N && (reinterpret_cast<uintptr_t>(p.w_scale) & 15) == 0) {
      const float4* w4 = reinterpret_cast<const float4*>(p.w_scale + n0);      // the same address in the whole warp
#pragma unroll
      for (int i = 0; i < NC / 4; ++i) {
        const float4 w = __ldg(w4 + i);
        v[4 * i] = __fmul_rn(__fmul_rn(v[4 * i], p.alpha * w.x), as);
        v[4 * i + 1] = __fmul_rn(__fmul_rn(v[4 * i + 1], p.alpha * w.y), as);
        v[4 * i + 2] = __fmul_rn(__fmul_rn(v[4 * i + 2], p.alpha * w.z), as);
        v[4 * i + 3] = __fmul_rn(__fmul_rn(v[4 * i + 3], p.alpha * w.w), as);
      }
    } else {
#pragma unroll
      for (int i = 0; i < NC; ++i) v[i] = __fmul_rn(__fmul_rn(v[i], p.alpha * (n0 + i < p.N ? __ldg(p.w_scale + n0 + i) : 1.f)), as);
    }
  } else {
#pragma unroll
    for (int i = 0; i < NC; ++i) v[i] = __fmul_rn(__fmul_rn(v[i], p.alpha), as);
  }
  if (glu) {
    const bool clamp = KIND == KIND_BF16 && p.epilogue == mb::EPI_CLAMP_GLU, geglu = KIND == KIND_BF16 && p.epilogue == mb::EPI_GEGLU;
#pragma unroll
    for (int i = 0; i < NC / 2; ++i) {
      const float g = v[2 * i], u = v[2 * i + 1];
      v[i] = clamp ? mb::clamp_glu_fast(g, u, p.epi_a, p.epi_b) : geglu ? mb::geglu_fast(g, u) : mb::silu(g) * u;
    }
    if (p.outq) {
      const float inv6gs = 1.f / (6.f * p.outq_gs);
      uint32_t sfs = 0;
      uint32_t q[NC / 16];
#pragma unroll
      for (int b = 0; b < NC / 32; ++b) {
        float mx = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) mx = fmaxf(mx, fabsf(v[b * 16 + i]));
        const uint8_t sfc = mb::float_to_e4m3(mx * inv6gs);
        const float sff = mb::e4m3_to_float(sfc);
        const float qi = sff > 0.f ? __fdividef(1.f, sff * p.outq_gs) : 0.f;
        sfs |= (uint32_t)sfc << (8 * b);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t w = 0;
#pragma unroll
          for (int i = 0; i < 4; ++i) w |= mb::e2m1x2_pack(v[b * 16 + h * 8 + 2 * i] * qi, v[b * 16 + h * 8 + 2 * i + 1] * qi) << (8 * i);
          q[2 * b + h] = w;
        }
      }
      const int c0 = n0 / 2;                                 // first output column: a multiple of NC / 2
      if (m < p.M && n0 < p.N) {                             // N / 2 is a multiple of 16 * NC / 32 columns (checked by the launcher)
        uint4* dst = reinterpret_cast<uint4*>(p.outq + (size_t)m * p.ldq + c0 / 2);
#pragma unroll
        for (int i = 0; i < NC / 64; ++i) dst[i] = make_uint4(q[4 * i], q[4 * i + 1], q[4 * i + 2], q[4 * i + 3]);
        uint8_t* sf = p.outq_sf + ((size_t)(m >> 7) * p.outq_sf_k64 + (c0 >> 6)) * 512 + mb::sf_tile_offset(m & 127, (c0 >> 4) & 3);
        if constexpr (NC == 128) *reinterpret_cast<uint32_t*>(sf) = sfs;
        else *reinterpret_cast<uint16_t*>(sf) = (uint16_t)sfs;
      }
      return;
    }
    if (m >= p.M) return;
    if constexpr (!VEC) return emit_ragged<NC / 2>(p, (size_t)m, n0 / 2, p.N / 2, v);
#pragma unroll
    for (int c = 0; c < NC / 2; c += 16) {
      const uint4 none[2] = {};
      emit16(p, (size_t)m, n0 / 2 + c, p.N / 2, v + c, none);
    }
    return;
  }
  if (KIND == KIND_BF16 && p.epilogue != mb::EPI_PLAIN) {
    if (p.epilogue == mb::EPI_SILU_COLS) {
#pragma unroll
      for (int i = 0; i < NC; ++i) v[i] = n0 + i < p.epi_n ? mb::silu(v[i]) : v[i];
    } else if (p.epilogue == mb::EPI_RELU2) {
#pragma unroll
      for (int i = 0; i < NC; ++i) v[i] = mb::relu2(v[i]);
    } else {
#pragma unroll
      for (int i = 0; i < NC; ++i) v[i] += n0 + i < p.N ? __ldg(p.epi_bias + n0 + i) : 0.f;
      if (p.epilogue == mb::EPI_NEG_EXP) {
#pragma unroll
        for (int i = 0; i < NC; ++i) v[i] = -expf(v[i]);
      } else if (p.epilogue == mb::EPI_LOG_SIGMOID) {
#pragma unroll
        for (int i = 0; i < NC; ++i) v[i] = p.epi_a * mb::log_sigmoid(v[i]);
      } else if (p.epilogue == mb::EPI_SIGMOID) {
#pragma unroll
        for (int i = 0; i < NC; ++i) v[i] = p.epi_a * mb::sigmoid_fast(v[i]);
      }
    }
  }
  if (m >= p.M) return;
  if constexpr (!VEC) return emit_ragged<NC>(p, (size_t)m, n0, p.N, v);
#pragma unroll
  for (int c = 0; c < NC; c += 32) {                         // four residual vectors in flight at a time
    uint4 r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = residual8(p, (size_t)m, n0 + c + 8 * i, p.N);
#pragma unroll
    for (int i = 0; i < 4; i += 2) emit16(p, (size_t)m, n0 + c + 8 * i, p.N, v + c + 8 * i, r + i);
  }
}

// ------------------------------------------------------------------------------------------ pairs of CTAs
template <int KIND, int BN>
struct PairCfg {
  static constexpr int kABytes = 128 * 128;                  // this CTA's tokens
  static constexpr int kBBytes = BN / 2 * 128;               // this CTA's half of the features
  static constexpr int kSfaBytes = KIND == KIND_NVFP4 ? 2048 : 0;              // this CTA's tokens
  static constexpr int kSfbBytes = KIND == KIND_NVFP4 ? BN / 128 * 2048 : 0;   // all features: each CTA needs every scale
  static constexpr int kStageBytes = kABytes + kBBytes + kSfaBytes + kSfbBytes;
  static constexpr int kStagesRaw = (224 * 1024) / kStageBytes;
  static constexpr int kStages = kStagesRaw > 8 ? 8 : kStagesRaw;
  static constexpr int kAccs = KIND == KIND_NVFP4 && BN == 256 ? 1 : 2;
  static constexpr int kSfBase = kAccs * BN;
  static constexpr int kSfCols = 16 + BN / 128 * 16;         // scale factors of one k block; two sets, used in turn
  static constexpr int kNeedCols = kSfBase + (KIND == KIND_NVFP4 ? 2 * kSfCols : 0);
  static constexpr int kTmemCols = kNeedCols <= 256 ? 256 : 512;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024;
  static_assert(kStageBytes % 1024 == 0 && kNeedCols <= 512, "");
};

template <int KIND, int BN, bool VEC>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmSA, const __grid_constant__ CUtensorMap tmSB, const RowsParams p) {
  using C = PairCfg<KIND, BN>;
  constexpr int kStages = C::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full_bar[kStages];        // used in the leader: both CTAs' bytes of a stage
  __shared__ __align__(8) uint64_t empty_bar[kStages];       // in each CTA
  __shared__ __align__(8) uint64_t acc_full[2];              // in each CTA
  __shared__ __align__(8) uint64_t acc_empty[2];             // used in the leader: both CTAs' epilogue warps
  __shared__ uint32_t tmem_base_s;

  const int warp = threadIdx.x >> 5;
  const uint32_t rank = mb::cluster_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int tiles = p.m_tiles * p.n_tiles;
  const int my_tiles = (tiles - pair + pairs - 1) / pairs;   // tiles pair, pair + pairs, ...; the grid has at most `tiles` pairs
  const int nkb = p.num_kb;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mb::mbar_init(&full_bar[s], 1);
      mb::mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mb::mbar_init(&acc_full[i], 1);
      mb::mbar_init(&acc_empty[i], 2 * kEpiWarps);
    }
    mb::mbar_fence_init();
    mb::tma_prefetch_desc(&tmA);
    mb::tma_prefetch_desc(&tmB);
  }
  if (warp == 1) mb::tmem_alloc2(&tmem_base_s, C::kTmemCols);
  mb::tc_fence_before();
  __syncthreads();
  mb::cluster_sync_all();                                    // barriers of both CTAs stand before either signals the other
  mb::tc_fence_after();
  const uint32_t tmem = tmem_base_s;
  mb::pdl_launch_dependents();

  auto sA = [&](int s) { return smem + s * C::kStageBytes; };
  auto sB = [&](int s) { return smem + s * C::kStageBytes + C::kABytes; };
  auto sSFA = [&](int s) { return smem + s * C::kStageBytes + C::kABytes + C::kBBytes; };
  auto sSFB = [&](int s) { return smem + s * C::kStageBytes + C::kABytes + C::kBBytes + C::kSfaBytes; };
  constexpr int kCoordStep = KIND == KIND_BF16 ? 64 : 128;

  if (warp == 0) {
    // ------------------------------------------------------------ producer (each CTA its own half)
    if (mb::elect_one()) {
      const int total = my_tiles * nkb;
      int b_kb = 0, b_t = pair;
      auto load_b = [&](int g) {
        const int s = g % kStages, nt = b_t / p.m_tiles;
        const uint32_t bar = mb::dsmem_addr(mb::smem_u32(&full_bar[s]), 0);
        mb::tma_load_2d_pair(sB(s), &tmB, bar, b_kb * kCoordStep, nt * BN + (int)rank * (BN / 2));
        if constexpr (KIND == KIND_NVFP4) {
#pragma unroll
          for (int i = 0; i < BN / 128; ++i)
            mb::tma_load_2d_pair(sSFB(s) + i * 2048, &tmSB, bar, 0, (nt * (BN / 128) + i) * p.sfb_rows + b_kb * 8);
        }
        if (++b_kb == nkb) { b_kb = 0; b_t += pairs; }
      };
      int a_kb = 0, a_t = pair;
      auto load_a = [&](int g) {
        const int s = g % kStages, mt = a_t % p.m_tiles;
        const uint32_t bar = mb::dsmem_addr(mb::smem_u32(&full_bar[s]), 0);
        mb::tma_load_2d_pair(sA(s), &tmA, bar, a_kb * kCoordStep, (mt * 2 + (int)rank) * 128);
        if constexpr (KIND == KIND_NVFP4) mb::tma_load_2d_pair(sSFA(s), &tmSA, bar, 0, (mt * 2 + (int)rank) * p.sfa_rows + a_kb * 8);
        if (++a_kb == nkb) { a_kb = 0; a_t += pairs; }
      };
      const int pre = min(total, kStages);
      for (int g = 0; g < pre; ++g) {                        // weights do not depend on the preceding kernel
        if (rank == 0) mb::mbar_expect_tx(&full_bar[g], 2 * C::kStageBytes);
        load_b(g);
      }
      mb::pdl_wait();
      for (int g = 0; g < pre; ++g) load_a(g);
      for (int g = pre; g < total; ++g) {
        const int s = g % kStages;
        if (!mb::mbar_wait(&empty_bar[s], ((g / kStages) & 1) ^ 1, p.status, MB_ST_TIMEOUT_TMA)) break;
        if (rank == 0) mb::mbar_expect_tx(&full_bar[s], 2 * C::kStageBytes);
        load_b(g);
        load_a(g);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (the leader, for both CTAs)
    if (rank == 0 && mb::elect_one()) {
      uint32_t idesc;
      if constexpr (KIND == KIND_BF16) idesc = mb::umma_idesc(1, 1, 256, BN);
      else if constexpr (KIND == KIND_NVFP4) idesc = mb::umma_idesc_bs(1, 1, 256, BN, 0);
      else idesc = mb::umma_idesc(0, 0, 256, BN);
      bool ok = true;
      int g = 0;
      for (int it = 0; it < my_tiles && ok; ++it) {
        const int buf = it % C::kAccs;
        const uint32_t acc = tmem + buf * BN;
        for (int i = 0; i < nkb; ++i, ++g) {
          const int s = g % kStages;
          ok = mb::mbar_wait(&full_bar[s], (g / kStages) & 1, p.status, MB_ST_TIMEOUT_MMA);
          if (!ok) break;
          mb::tc_fence_after();
          const uint32_t a_base = mb::smem_u32(sA(s)), b_base = mb::smem_u32(sB(s));
          const uint32_t sfa_col = tmem + C::kSfBase + (g & 1) * C::kSfCols, sfb_col = sfa_col + 16;
          if constexpr (KIND == KIND_NVFP4) {
            const uint32_t sfa = mb::smem_u32(sSFA(s)), sfb = mb::smem_u32(sSFB(s));
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              mb::tmem_cp_sf2(sfa_col + j * 4, mb::umma_desc_sf(sfa + j * 512));
#pragma unroll
              for (int h = 0; h < BN / 128; ++h)
                mb::tmem_cp_sf2(sfb_col + j * (BN / 32) + h * 4, mb::umma_desc_sf(sfb + h * 2048 + j * 512));
            }
          }
          if (i == 0) {                                      // the epilogue has taken this accumulator's last tile
            ok = mb::mbar_wait(&acc_empty[buf], ((it / C::kAccs) & 1) ^ 1, p.status, MB_ST_TIMEOUT_MMA);
            if (!ok) break;
            mb::tc_fence_after();
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint64_t da = mb::umma_desc_sw128(a_base + j * 32), db = mb::umma_desc_sw128(b_base + j * 32);
            if constexpr (KIND == KIND_BF16) mb::umma2_f16(acc, da, db, idesc, (i | j) != 0);
            else if constexpr (KIND == KIND_FP8) mb::umma2_f8f6f4(acc, da, db, idesc, (i | j) != 0);
            else mb::umma2_nvfp4(acc, da, db, idesc, sfa_col + j * 4, sfb_col + j * (BN / 32), (i | j) != 0);
          }
          mb::tc_commit2(&empty_bar[s]);
        }
        if (ok) mb::tc_commit2(&acc_full[buf]);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ epilogue: lane = token, two warps share a lane quadrant
    constexpr int NC = BN / 2;
    const int q = warp & 3, half = (warp - 2) >> 2, lane = threadIdx.x & 31;
    const uint32_t src = tmem + ((uint32_t)(q * 32) << 16) + half * NC;
    const uint32_t empty0 = mb::dsmem_addr(mb::smem_u32(&acc_empty[0]), 0);
    mb::pdl_wait();
    bool ok = true;
    for (int it = 0; it < my_tiles && ok; ++it) {
      const int t = pair + it * pairs, mt = t % p.m_tiles, nt = t / p.m_tiles, buf = it % C::kAccs;
      const int m = (mt * 2 + (int)rank) * 128 + q * 32 + lane;
      float as = KIND == KIND_BF16 ? 1.f : p.a_static;
      if (KIND != KIND_BF16 && p.a_scale && m < p.M) as = __ldg(p.a_scale + m);
      ok = mb::mbar_wait(&acc_full[buf], (it / C::kAccs) & 1, p.status, MB_ST_TIMEOUT_EPI);
      if (!__all_sync(0xffffffffu, ok)) break;
      mb::tc_fence_after();
      float v[NC];
#pragma unroll
      for (int c = 0; c < NC; c += 32) mb::tmem_ld32_async(src + buf * BN + c, v + c);
      mb::tmem_ld_wait(v);
      mb::tc_fence_before();
      __syncwarp();
      if (lane == 0) mb::mbar_arrive_cluster(empty0 + buf * 8);
      finish_row<KIND, NC, VEC>(p, v, m, nt * BN + half * NC, as);
    }
    mb::tc_fence_before();
  }
  __syncthreads();
  mb::cluster_sync_all();                                    // nothing of the pair signals or reads a CTA that has left
  if (warp == 1) {
    mb::tc_fence_after();
    mb::tmem_dealloc2(tmem, C::kTmemCols);
  }
}

// ------------------------------------------------------------------------------------------ fp8, 128 x 128 weight scales
constexpr int kBlkThreads = 384;   // producer warp, MMA warp, two that wait; eight epilogue warps

template <int BN>
struct BlkCfg {
  static constexpr int kAccs = 512 / BN;
  static constexpr int kStageBytes = 128 * 128 + BN * 128;
  static constexpr int kStages = BN == 256 ? 4 : 6;
  static constexpr int kSmem = kStages * kStageBytes + 1024;
};

template <int BN, bool VEC>
__global__ void __launch_bounds__(kBlkThreads, 1)
gemm_block_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const RowsParams p) {
  constexpr int kBlkStages = BlkCfg<BN>::kStages, kBlkStageBytes = BlkCfg<BN>::kStageBytes, kBlkAccs = BlkCfg<BN>::kAccs;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full_bar[kBlkStages];
  __shared__ __align__(8) uint64_t empty_bar[kBlkStages];
  __shared__ __align__(8) uint64_t acc_full[kBlkAccs];
  __shared__ __align__(8) uint64_t acc_empty[kBlkAccs];
  __shared__ uint32_t tmem_base_s;
  const int warp = threadIdx.x >> 5;
  const int nkb = p.num_kb, items = p.m_tiles * p.n_tiles;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kBlkStages; ++s) {
      mb::mbar_init(&full_bar[s], 1);
      mb::mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < kBlkAccs; ++i) {
      mb::mbar_init(&acc_full[i], 1);
      mb::mbar_init(&acc_empty[i], kEpiWarps);
    }
    mb::mbar_fence_init();
    mb::tma_prefetch_desc(&tmA);
    mb::tma_prefetch_desc(&tmB);
  }
  if (warp == 1) mb::tmem_alloc(&tmem_base_s, 512);
  mb::tc_fence_before();
  __syncthreads();
  mb::tc_fence_after();
  const uint32_t tmem = tmem_base_s;
  mb::pdl_launch_dependents();
  mb::pdl_wait();                                            // the work list and the token rows come from preceding kernels

  // item i: token tile i / n_tiles, feature tile i % n_tiles (the CTAs that run together share the token rows in L2 and
  // stream different weights); entries of the work list without rows are passed over by every role alike
  struct Item { int row0, rows, w_row0; };
  auto item = [&](int i, Item& t) {
    const int mt = i / p.n_tiles, nt = i - mt * p.n_tiles;
    if (p.tile_expert) {
      const int e = __ldg(p.tile_expert + mt);
      if (e < 0) return false;
      t.row0 = __ldg(p.tile_row0 + mt);
      t.rows = __ldg(p.tile_nrows + mt);
      t.w_row0 = e * p.n_per_expert + nt * BN;
    } else {
      t.row0 = mt * 128;
      t.rows = min(128, p.M - t.row0);
      t.w_row0 = nt * BN;
    }
    return true;
  };

  // BN = 256: 128 sums and 64 fresh columns a thread; the registers come from the four warps that copy and issue
  if (warp < 4) {
  if constexpr (BN == 256) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
  if (warp == 0) {
    if (mb::elect_one()) {
      int g = 0;
      bool ok = true;
      for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
        Item t;
        if (!item(i, t)) continue;
        for (int kb = 0; kb < nkb; ++kb, ++g) {
          const int s = g % kBlkStages;
          ok = mb::mbar_wait(&empty_bar[s], ((g / kBlkStages) & 1) ^ 1, p.status, MB_ST_TIMEOUT_TMA);
          if (!ok) break;
          uint8_t* st = smem + s * kBlkStageBytes;
          mb::mbar_expect_tx(&full_bar[s], p.a_bytes + BN * 128);
          mb::tma_load_2d(st + 128 * 128, &tmB, &full_bar[s], kb * 128, t.w_row0);
          mb::tma_load_2d(st, &tmA, &full_bar[s], kb * 128, t.row0);   // rows past the box keep old bytes: they make rows nobody stores
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (mb::elect_one()) {
      const uint32_t idesc = mb::umma_idesc(0, 0, 128, BN);
      int g = 0;
      bool ok = true;
      for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
        Item t;
        if (!item(i, t)) continue;
        for (int kb = 0; kb < nkb; ++kb, ++g) {
          const int s = g % kBlkStages, buf = g % kBlkAccs;
          ok = mb::mbar_wait(&acc_empty[buf], ((g / kBlkAccs) & 1) ^ 1, p.status, MB_ST_TIMEOUT_MMA) &&
               mb::mbar_wait(&full_bar[s], (g / kBlkStages) & 1, p.status, MB_ST_TIMEOUT_MMA);
          if (!ok) break;
          mb::tc_fence_after();
          const uint32_t a_base = mb::smem_u32(smem + s * kBlkStageBytes), b_base = a_base + 128 * 128;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            mb::umma_f8f6f4(tmem + buf * BN, mb::umma_desc_sw128(a_base + j * 32), mb::umma_desc_sw128(b_base + j * 32), idesc, j != 0);
          mb::tc_commit(&empty_bar[s]);
          mb::tc_commit(&acc_full[buf]);
        }
      }
    }
    __syncwarp();
  }
  } else {
    if constexpr (BN == 256) asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
    constexpr int NC = BN / 2;
    const int q = warp & 3, half = (warp - 4) >> 2, lane = threadIdx.x & 31;
    const uint32_t src = tmem + ((uint32_t)(q * 32) << 16) + half * NC;
    int g = 0;
    bool ok = true;
    for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
      Item t;
      if (!item(i, t)) continue;
      const int r = q * 32 + lane;
      const bool live = r < t.rows;
      const float* asp = p.a_scale + t.row0 + r;
      const int n0 = (i % p.n_tiles) * BN + half * NC;
      const float* wsp = p.w_scale + (size_t)((t.w_row0 + (n0 < p.N ? half * NC : 0)) / 128) * nkb;   // a half behind the last feature reads the first's
      float acc[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) acc[c] = 0.f;
      // the scales of k block kb + 1 are on their way while block kb is added
      float a_next = live ? __ldg(asp) : 0.f, w_next = __ldg(wsp);
      for (int kb = 0; kb < nkb; ++kb, ++g) {
        const int buf = g % kBlkAccs;
        const float sc = a_next * w_next;
        if (kb + 1 < nkb) {
          a_next = live ? __ldg(asp + (size_t)(kb + 1) * p.a_ld) : 0.f;
          w_next = __ldg(wsp + kb + 1);
        }
        ok = mb::mbar_wait(&acc_full[buf], (g / kBlkAccs) & 1, p.status, MB_ST_TIMEOUT_EPI);
        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
        mb::tc_fence_after();
#pragma unroll
        for (int c0 = 0; c0 < NC; c0 += 64) {
          float v[64];
          mb::tmem_ld32_async(src + buf * BN + c0, v);
          mb::tmem_ld32_async(src + buf * BN + c0 + 32, v + 32);
          mb::tmem_ld_wait(v);
          if (c0 + 64 == NC) {                               // the accumulator is free for the next k block
            mb::tc_fence_before();
            __syncwarp();
            if (lane == 0) mb::mbar_arrive(&acc_empty[buf]);
          }
#pragma unroll
          for (int c = 0; c < 64; ++c) acc[c0 + c] = fmaf(v[c], sc, acc[c0 + c]);
        }
      }
      if (ok && live) {
        const size_t m = (size_t)t.row0 + r;
        if constexpr (VEC) {
#pragma unroll
          for (int c = 0; c < NC; c += 32) {
            uint4 res[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) res[k] = residual8(p, m, n0 + c + 8 * k, p.N);
#pragma unroll
            for (int k = 0; k < 4; k += 2) emit16(p, m, n0 + c + 8 * k, p.N, acc + c + 8 * k, res + k);
          }
        } else {
          emit_ragged<NC>(p, m, n0, p.N, acc);
        }
      }
    }
    mb::tc_fence_before();
  }
  __syncthreads();
  if (warp == 1) {
    mb::tc_fence_after();
    mb::tmem_dealloc(tmem, 512);
  }
}

template <int KIND, int BN, bool VEC>
int launch_pair(const CUtensorMap* tm, const RowsParams& p, int pairs, cudaStream_t stream) {
  using C = PairCfg<KIND, BN>;
  auto kern = gemm_pair_kernel<KIND, BN, VEC>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  return (int)mb::launch_kernel_cluster(kern, dim3(2 * pairs), dim3(kThreads), C::kSmemBytes, stream, 1, tm[0], tm[1], tm[2], tm[3], p);
}

template <int KIND>
int launch_pair(const CUtensorMap* tm, const RowsParams& p, bool wide, int pairs, cudaStream_t stream) {
  if (p.vec || p.outq) return wide ? launch_pair<KIND, 256, true>(tm, p, pairs, stream) : launch_pair<KIND, 128, true>(tm, p, pairs, stream);
  return wide ? launch_pair<KIND, 256, false>(tm, p, pairs, stream) : launch_pair<KIND, 128, false>(tm, p, pairs, stream);
}

template <int BN, bool VEC>
int launch_block(const CUtensorMap* tm, const RowsParams& p, int grid, cudaStream_t stream) {
  auto kern = gemm_block_kernel<BN, VEC>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, BlkCfg<BN>::kSmem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  return (int)mb::launch_kernel_cluster(kern, dim3(grid), dim3(kBlkThreads), BlkCfg<BN>::kSmem, stream, 1, tm[0], tm[1], p);
}

}  // namespace

// Few tiles of long rows: the kernels here walk the k blocks of a tile in series, a quarter of a microsecond each (fp8 blocks 0.58)
// however few tiles there are; one tile per CTA (gemm_tcgen05.cu) can split them, at a fixed price (the exchange of a tile of 128
// features by 256 tokens, NVFP4 128, fp8 blocks 64) that weighs more the fewer splits there are. Here / split, us (tiles x splits;
// depth in k blocks):
//   bf16       32: 12 x 8 18.1 / 18.5; 40: 12 x 8 20.3 / 18.7, 22 x 6 20.5 / 22.1; 64: 24 x 5 26.5 / 24.1, 36 x 3 26.9 / 26.9;
//              80: 12 x 8 28.9 / 20.8, 32 x 4 31.2 / 28.8, 48 x 2 30.9 / 34.9; 112: 44 x 3 40.7 / 37.4
//   fp8        32: 12 x 8 18.5 / 18.5, 16 x 6 18.6 / 20.5; 56: 12 x 8 24.7 / 18.7, 24 x 5 25.0 / 22.7, 48 x 2 26.2 / 28.9
//   NVFP4      12: 24 x 3 14.5 / 14.9; 16: 24 x 4 16.5 / 14.6; 20: 40 x 3 16.7 / 16.6; 28: 60 x 2 20.2 / 18.6; 68: 12 x 8 28.7 / 16.5
//   fp8 blocks 16: 32 x 4 16.4 / 14.8, 40 x 3 16.4 / 16.4, 48 x 2 16.4 / 18.5; 32: 8 x 8 26 / 16; 56: 10 x 8 39 / 17, 48 x 2 35 / 33
static bool splits_pay(const MbGemmArgs* a) {
  if (!a->ws) return false;
  const int kelems = a->kind == KIND_BF16 ? 64 : a->kind == KIND_NVFP4 ? 256 : 128;
  const int tn = a->kind == KIND_NVFP4 ? 128 : a->kind == KIND_FP8_BLOCK ? 64 : 256;
  const int num_kb = (a->K + kelems - 1) / kelems, sms = a->sm_count > 0 ? a->sm_count : 148;
  const long long tiles = (long long)((a->N + 127) / 128) * ((a->M + tn - 1) / tn);
  if (tiles >= sms) return false;
  const int splits = mb_gemm_auto_splits((int)tiles, num_kb, sms, true), saved = num_kb - (num_kb + splits - 1) / splits;
  return a->kind == KIND_NVFP4 ? saved > 11 : a->kind == KIND_FP8_BLOCK ? splits >= 3 && saved > 10 : saved > 64 - 4 * splits;
}

bool mb_gemm_rows_serves(const MbGemmArgs* a) {
  if (a->force_splits > 0 || a->no_cluster || (a->flags & (MB_GEMM_ONE_TILE_PER_CTA | MB_GEMM_DECODE_TILE_ORDER))) return false;
  if (a->kind == KIND_FP8_BLOCK) {
    if (a->epilogue != mb::EPI_PLAIN || a->outq) return false;
    return a->tile_expert ? true : a->force_tn == 0 && a->M > 64 && !splits_pay(a);
  }
  // bf16 of one token tile is bound by the weights' stream, which 74 pairs pull slower than 148 CTAs (or splits of K) do: two dense
  // layers of 5120 at 144 / 200 / 256 tokens 537 / 546 / 552 us here, 505 / 515 / 529 a tile per CTA; at 300 tokens 713 against 869.
  // NVFP4 weights are a quarter of the bytes: 159 / 161 / 165 here against 178 / 187 / 187.
  if (a->kind == KIND_BF16 && a->M <= 256 && !a->outq) return false;
  if (a->tile_expert || a->force_tn != 0 || a->M <= 128 || !(a->flags & MB_GEMM_PERSISTENT_PREFILL)) return false;
  return a->outq || !splits_pay(a);
}

int mb_gemm_rows(const MbGemmArgs* a, int tn, cudaStream_t stream) {
  const int kind = a->kind;
  const int kelems = kind == KIND_BF16 ? 64 : kind == KIND_NVFP4 ? 256 : 128, elem_bits = kind == KIND_BF16 ? 16 : kind == KIND_NVFP4 ? 4 : 8;
  const CUtensorMapDataType dt = kind == KIND_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
  const size_t row_bytes = (size_t)a->K * elem_bits / 8;
  const uint64_t inner = kind == KIND_BF16 ? (uint64_t)a->K : (uint64_t)row_bytes;
  const uint32_t box = kind == KIND_BF16 ? 64 : 128;
  const size_t x_pitch = a->ldx > 0 ? (size_t)a->ldx * 2 : row_bytes;
  const int sms = a->sm_count > 0 ? a->sm_count : 148;

  RowsParams p{};
  p.M = a->M; p.N = a->tile_expert ? a->n_per_expert : a->N; p.num_kb = (a->K + kelems - 1) / kelems;
  p.ldo = a->ldo; p.out = a->out; p.residual = reinterpret_cast<const __nv_bfloat16*>(a->residual);
  p.w_scale = a->w_scale; p.a_scale = a->a_scale; p.a_ld = a->a_ld; p.alpha = a->alpha;
  p.a_static = a->a_static != 0.f ? a->a_static : 1.f;
  p.epilogue = a->epilogue; p.out_f32 = a->out_f32;
  p.vec = a->ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(a->out) & (a->out_f32 ? 31 : 15)) == 0 && (reinterpret_cast<uintptr_t>(a->residual) & 15) == 0;
  p.sectors = a->ldo % 16 == 0 && (reinterpret_cast<uintptr_t>(a->out) & 31) == 0;
  p.epi_a = a->epi_a; p.epi_b = a->epi_b; p.epi_n = a->epi_n; p.epi_bias = a->epi_bias;
  p.status = a->status;
  CUtensorMap tm[4];
  int rc = 0;

  if (kind == KIND_FP8_BLOCK) {
    p.tile_expert = a->tile_expert; p.tile_row0 = a->tile_row0; p.tile_nrows = a->tile_nrows;
    p.n_per_expert = a->tile_expert ? a->n_per_expert : 0;
    const int box_rows = !a->tile_expert || a->force_tn == 128 ? 128 : tn;
    if (box_rows != 16 && box_rows != 32 && box_rows != 64 && box_rows != 128) return MB_ERR_UNSUPPORTED;
    if (mb_gemm_few_serves(a, box_rows)) return mb_gemm_few(a, box_rows, stream);
    p.a_bytes = box_rows * 128;
    p.m_tiles = a->tile_expert ? a->max_tiles : (a->M + 127) / 128;
    // 256 features a tile read the token rows half as often (at 128 x 128 the operands of 2700 tokens' experts come from L2 at its
    // rate); short entries of a work list are bound by the weights' stream and keep the finer tiles
    auto waves = [&](int bn) { return ((long long)p.m_tiles * ((p.N + bn - 1) / bn) + sms - 1) / sms; };
    const bool wide = a->tile_expert ? box_rows == 128 : waves(256) * 2.0 <= waves(128) * 1.3;
    const int bn = wide ? 256 : 128;
    p.n_tiles = (p.N + bn - 1) / bn;
    if ((rc = mbh::encode_2d(&tm[0], dt, a->X, inner, (uint64_t)a->M, x_pitch, box, (uint32_t)box_rows))) return rc;
    if ((rc = mbh::encode_2d(&tm[1], dt, a->W, inner, (uint64_t)a->N, row_bytes, box, (uint32_t)bn))) return rc;
    const long long items = (long long)p.m_tiles * p.n_tiles;
    if (items > 0x7fffffff) return MB_ERR_TOO_LARGE;
    const int grid = items < sms ? (int)items : sms;
    if (p.vec) return wide ? launch_block<256, true>(tm, p, grid, stream) : launch_block<128, true>(tm, p, grid, stream);
    return wide ? launch_block<256, false>(tm, p, grid, stream) : launch_block<128, false>(tm, p, grid, stream);
  }

  if (a->outq) {
    // a warp's 64 or 32 result columns are whole 16-column blocks, and whole 16-byte vectors of the packed row
    if (a->epilogue != mb::EPI_SWIGLU || !a->outq_sf || a->outq_gs <= 0.f || (a->N / 2) % 64 || a->outq_sf_k64 * 64 < a->N / 2 ||
        a->ldq % 16 || (reinterpret_cast<uintptr_t>(a->outq) & 15) || (reinterpret_cast<uintptr_t>(a->outq_sf) & 3))
      return MB_ERR_BAD_ARG;
    p.outq = reinterpret_cast<uint8_t*>(a->outq); p.ldq = a->ldq;
    p.outq_sf = reinterpret_cast<uint8_t*>(a->outq_sf); p.outq_sf_k64 = a->outq_sf_k64;
    p.outq_gs = a->outq_gs;
  }
  p.m_tiles = (a->M + 255) / 256;
  // BN = 256 feeds the tensor cores with half the operand bytes per product; BN = 128 gives twice the tiles where those of
  // 256 leave pairs idle in the last wave. The factor is a 128-feature tile's measured cost against half a 256-feature one.
  const int max_pairs = sms / 2;
  auto waves = [&](int bn) { return ((long long)p.m_tiles * ((a->N + bn - 1) / bn) + max_pairs - 1) / max_pairs; };
  const bool wide = waves(256) * 2.0 <= waves(128) * 1.3;
  const int bn = wide ? 256 : 128;
  p.n_tiles = (a->N + bn - 1) / bn;
  const long long tiles = (long long)p.m_tiles * p.n_tiles;
  if (tiles > 0x7fffffff) return MB_ERR_TOO_LARGE;
  const long long w = (tiles + max_pairs - 1) / max_pairs;
  const int pairs = (int)((tiles + w - 1) / w);                // as few as finish in the same number of waves
  if ((rc = mbh::encode_2d(&tm[0], dt, a->X, inner, (uint64_t)a->M, x_pitch, box, 128))) return rc;
  if ((rc = mbh::encode_2d(&tm[1], dt, a->W, inner, (uint64_t)a->N, row_bytes, box, (uint32_t)bn / 2))) return rc;
  tm[2] = tm[0]; tm[3] = tm[1];
  if (kind == KIND_NVFP4) {
    // tiled scale factors as rows of 256 bytes: a k block of 128 tokens or features is eight of them, one behind the other
    p.sfa_rows = p.sfb_rows = a->sf_k64 * 2;
    if ((rc = mbh::encode_2d(&tm[2], dt, a->sfb, 256, (uint64_t)((a->M + 127) / 128) * p.sfa_rows, 256, 256, 8, CU_TENSOR_MAP_SWIZZLE_NONE))) return rc;
    if ((rc = mbh::encode_2d(&tm[3], dt, a->sfa, 256, (uint64_t)((a->N + 127) / 128) * p.sfb_rows, 256, 256, 8, CU_TENSOR_MAP_SWIZZLE_NONE))) return rc;
  }
  switch (kind) {
    case KIND_BF16: return launch_pair<KIND_BF16>(tm, p, wide, pairs, stream);
    case KIND_FP8: return launch_pair<KIND_FP8>(tm, p, wide, pairs, stream);
    default: return launch_pair<KIND_NVFP4>(tm, p, wide, pairs, stream);
  }
}
