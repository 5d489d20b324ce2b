// Row-wise fused producer kernels: one CTA owns one token row, builds the fp32
// row in shared memory from one of several "input" recipes and writes it in one
// of several "output" encodings, so normalisation / activation / quantisation
// never make a separate trip through HBM.
//
// input recipes
//   IN_COPY          y = x
//   IN_RMSNORM       h = x (+ residual); residual_out = bf16(h);
//                    y = h * rsqrt(mean(h^2) + eps) * (w | 1 + w)
//   IN_SILU_MUL      y = silu(x[:, k]) * x[:, K + k]        (x is [M, 2K], gate | up)
//   IN_RELU2         y = relu(x)^2
//   IN_SIGMOID_GATE  y = x * sigmoid(gate), gate addressed per head with strides
//   IN_GATED_RMSNORM y = rmsnorm_group(x) * w * silu(gate)   (GDN / Mamba2 output norm;
//                    statistics over groups of `group` channels)
// output encodings
//   OUT_BF16         bf16 [M, K]
//   OUT_FP8_ROW      e4m3 [M, K] + scale[M] = amax / 448
//   OUT_FP8_G128     e4m3 [M, K] + scale[K/128][ld] per token per 128 channels
//   OUT_NVFP4        packed e2m1 [M, K/2] + ue4m3 scale factors in the 128x4 tiled
//                    layout tcgen05.cp consumes + per-token fp32 scale amax/(6*448)
// `also_bf16` additionally writes the bf16 row (router / MTP consumers).
//
// Reference behaviour covered: kernels/gb10/common/rms_norm.cu (rms_norm,
// residual_add_rms_norm, gated_rms_norm), rms_norm_act_quant.cu, moe_silu_mul.cu,
// relu_squared.cu, residual_add.cu::sigmoid_gate_mul, quantize_bf16_to_nvfp4.cu,
// w8a8_act_quant.cu, per_token_group_quant_fp8.
#include "common.cuh"
#include "op_args.h"
#include <cstdlib>
#include <type_traits>

namespace {

enum { IN_COPY = 0, IN_RMSNORM = 1, IN_SILU_MUL = 2, IN_RELU2 = 3, IN_SIGMOID_GATE = 4,
       IN_GATED_RMSNORM = 5 };
enum { OUT_BF16 = 0, OUT_FP8_ROW = 1, OUT_FP8_G128 = 2, OUT_NVFP4 = 3 };

struct RowParams {
  int M, K;
  int in_mode, out_mode;
  const __nv_bfloat16* x;
  long long x_ld;
  const __nv_bfloat16* residual;      // [M, K] or null
  __nv_bfloat16* residual_out;        // [M, K] or null
  const __nv_bfloat16* w;             // norm weight [K] or null
  int w_plus_one;
  float eps;
  const __nv_bfloat16* gate;          // IN_SIGMOID_GATE / IN_GATED_RMSNORM
  long long gate_ld;
  int head_dim, gate_head_stride, gate_head_off;
  int group;                          // IN_GATED_RMSNORM statistics group (0 = whole row)
  const float* xf32;                  // optional fp32 input instead of x (GDN core output)
  void* out;
  long long out_ld;                   // in elements of the output encoding (bytes for fp8/fp4)
  __nv_bfloat16* out_bf16;            // also_bf16 target or null
  long long out_bf16_ld;
  float* scale;                       // per-token scale(s)
  int scale_ld;                       // OUT_FP8_G128: tokens stride
  uint8_t* sf;                        // OUT_NVFP4 tiled scale factors
  int sf_k64;
  float static_gs;                    // OUT_NVFP4: > 0 = calibrated global scale instead of the row's amax / (6 * 448)
  const int* row_index;               // optional [M]: CTA i works on row row_index[i] (negative: none) instead of row i
  const void* gather;                 // optional [M] (IN_RMSNORM): row m of the input is row gather[m] of x, zeros where x has none
  int gather_wide;                    // gather holds 64-bit indices instead of 32-bit ones
  long long gather_rows;              // rows of x
  __nv_bfloat16* gather_out;          // [M, K] or null: the rows as gathered
  uint32_t* status;
};

// The row of x that output row m is made of. Taking rows of a table (the embedding, the rows that logits are wanted of) and
// normalising them was a launch of its own in front of the norm's: 3.5 us at 1 to 128 tokens, 20 us at 8192 rows of 5120 (168 MB
// that the norm then read again). A kernel of its own: with the branches in the one of all rows those took 2 to 7 % longer.
__device__ __forceinline__ long long source_row(const RowParams& p, int m, bool& live) {
  const long long i = p.gather_wide ? reinterpret_cast<const long long*>(p.gather)[m] : reinterpret_cast<const int*>(p.gather)[m];
  live = i >= 0 && i < p.gather_rows;
  if (!live && p.status) atomicCAS(p.status, 0u, MB_ST_BOUNDS);
  return live ? i : 0;
}

template <typename Row>
__device__ __forceinline__ float load_x(const RowParams& p, Row m, int k) {
  if (p.xf32) return p.xf32[(size_t)m * p.x_ld + k];
  return __bfloat162float(p.x[(size_t)m * p.x_ld + k]);
}

template <bool GATHER>
__global__ void __launch_bounds__(512) row_kernel(const RowParams p) {
  extern __shared__ float row[];
  __shared__ float red[32];
  const int K = p.K;
  const int tid = threadIdx.x, nt = blockDim.x;
  mb::pdl_wait();
  mb::pdl_launch_dependents();
  const int m = p.row_index ? p.row_index[blockIdx.x] : (int)blockIdx.x;
  if (m < 0) return;

  // ---- stage 1: build the fp32 row
  if (p.in_mode == IN_RMSNORM) {
    float ss = 0.f;
    bool live = true;
    std::conditional_t<GATHER, long long, int> from = m;
    if constexpr (GATHER) from = source_row(p, m, live);
    for (int k = tid; k < K; k += nt) {
      float h = live ? load_x(p, from, k) : 0.f;
      if (GATHER && p.gather_out) p.gather_out[(size_t)m * K + k] = __float2bfloat16(h);
      if (p.residual) {
        h += __bfloat162float(p.residual[(size_t)m * K + k]);
        h = __bfloat162float(__float2bfloat16(h));
      }
      if (p.residual_out) p.residual_out[(size_t)m * K + k] = __float2bfloat16(h);
      row[k] = h;
      ss += h * h;
    }
    ss = mb::block_sum(ss, red);
    const float inv = rsqrtf(ss / (float)K + p.eps);
    for (int k = tid; k < K; k += nt) {
      float w = p.w ? __bfloat162float(p.w[k]) : 1.f;
      if (p.w_plus_one) w += 1.f;
      row[k] = row[k] * inv * w;
    }
  } else if (p.in_mode == IN_GATED_RMSNORM) {
    const int G = p.group > 0 ? p.group : K;
    for (int k = tid; k < K; k += nt) row[k] = load_x(p, m, k);
    __syncthreads();
    // one warp per statistics group
    const int warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
    for (int g = warp; g * G < K; g += nw) {
      float ss = 0.f;
      for (int k = lane; k < G; k += 32) { const float v = row[g * G + k]; ss += v * v; }
      ss = mb::warp_sum(ss);
      const float inv = rsqrtf(ss / (float)G + p.eps);
      for (int k = lane; k < G; k += 32) {
        const int kk = g * G + k;
        const float w = p.w ? __bfloat162float(p.w[kk]) : 1.f;
        float y = row[kk] * inv * w;
        if (p.gate) y *= mb::silu(__bfloat162float(p.gate[(size_t)m * p.gate_ld + kk]));
        row[kk] = y;
      }
    }
  } else {
    for (int k = tid; k < K; k += nt) {
      float y;
      if (p.in_mode == IN_SILU_MUL) {
        const float g = load_x(p, m, k), u = load_x(p, m, K + k);
        y = mb::silu(g) * u;
      } else if (p.in_mode == IN_RELU2) {
        const float v = fmaxf(load_x(p, m, k), 0.f);
        y = v * v;
      } else if (p.in_mode == IN_SIGMOID_GATE) {
        const int h = k / p.head_dim, d = k - h * p.head_dim;
        const float g = __bfloat162float(
            p.gate[(size_t)m * p.gate_ld + (size_t)h * p.gate_head_stride + p.gate_head_off + d]);
        y = load_x(p, m, k) / (1.f + __expf(-g));
      } else {
        y = load_x(p, m, k);
      }
      row[k] = y;
    }
  }
  __syncthreads();

  if (p.out_bf16) {
    for (int k = tid; k < K; k += nt)
      p.out_bf16[(size_t)m * p.out_bf16_ld + k] = __float2bfloat16(row[k]);
  }

  // ---- stage 2: encode
  if (p.out_mode == OUT_BF16) {
    __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + (size_t)m * p.out_ld;
    for (int k = tid; k < K; k += nt) o[k] = __float2bfloat16(row[k]);
  } else if (p.out_mode == OUT_FP8_ROW) {
    float amax = 0.f;
    for (int k = tid; k < K; k += nt) amax = fmaxf(amax, fabsf(row[k]));
    amax = mb::block_max(amax, red);
    const float sc = amax > 0.f ? amax / 448.f : 1.f;
    const float inv = 1.f / sc;
    if (tid == 0) p.scale[m] = sc;
    uint8_t* o = reinterpret_cast<uint8_t*>(p.out) + (size_t)m * p.out_ld;
    for (int k = tid; k < K; k += nt) o[k] = mb::float_to_e4m3(row[k] * inv);
  } else if (p.out_mode == OUT_FP8_G128) {
    const int warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
    uint8_t* o = reinterpret_cast<uint8_t*>(p.out) + (size_t)m * p.out_ld;
    for (int g = warp; g * 128 < K; g += nw) {
      float v[4];
      float amax = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = g * 128 + lane * 4 + i;
        v[i] = k < K ? row[k] : 0.f;
        amax = fmaxf(amax, fabsf(v[i]));
      }
      amax = mb::warp_max(amax);
      const float sc = amax > 0.f ? amax / 448.f : 1.f;
      const float inv = 1.f / sc;
      if (lane == 0) p.scale[(size_t)g * p.scale_ld + m] = sc;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = g * 128 + lane * 4 + i;
        if (k < K) o[k] = mb::float_to_e4m3(v[i] * inv);
      }
    }
  } else {  // OUT_NVFP4
    float amax = 0.f;
    for (int k = tid; k < K; k += nt) amax = fmaxf(amax, fabsf(row[k]));
    amax = mb::block_max(amax, red);
    const float gs = p.static_gs > 0.f ? p.static_gs : (amax > 0.f ? amax / (6.f * 448.f) : 1.f);
    if (tid == 0) p.scale[m] = gs;
    uint8_t* o = reinterpret_cast<uint8_t*>(p.out) + (size_t)m * p.out_ld;
    uint8_t* sf_blk = p.sf + (size_t)(m >> 7) * p.sf_k64 * 512;
    const int r = m & 127;
    // one thread per 16-element block
    for (int b = tid; b * 16 < K; b += nt) {
      float v[16];
      float bmax = 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int k = b * 16 + i;
        v[i] = k < K ? row[k] : 0.f;
        bmax = fmaxf(bmax, fabsf(v[i]));
      }
      const uint8_t sfc = mb::float_to_e4m3(bmax / (6.f * gs));
      const float sff = mb::e4m3_to_float(sfc);
      const float inv = sff > 0.f ? 1.f / (sff * gs) : 0.f;
      uint32_t lo = 0, hi = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) lo |= mb::e2m1_code(v[i] * inv) << (4 * i);
#pragma unroll
      for (int i = 0; i < 8; ++i) hi |= mb::e2m1_code(v[8 + i] * inv) << (4 * i);
      *reinterpret_cast<uint2*>(o + b * 8) = make_uint2(lo, hi);
      sf_blk[(size_t)(b >> 2) * 512 + mb::sf_tile_offset(r, b & 3)] = sfc;
    }
  }
}

// sixteen neighbouring bf16 values from a 16-byte aligned address
__device__ __forceinline__ void load16(const __nv_bfloat16* src, float* v) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(src) + h);
    const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(b[i]);
      v[h * 8 + 2 * i] = f.x; v[h * 8 + 2 * i + 1] = f.y;
    }
  }
}

// ---------------------------------------------------------------------------------------
// Fast path for the hot recipes (copy / RMSNorm / SiLU-mul from bf16 rows): every thread owns
// whole 16-element blocks in registers (BPT of them), all global traffic is 16-byte vectors,
// and the row statistics (sum of squares and max |x * w|) share ONE block reduction, so the
// kernel is load -> reduce -> store. amax(y) is taken as max|x w| * inv_rms.
// The two gated recipes take the same road (GATED; statistics over 128 channels are eight neighbouring threads): through shared memory
// in 2-byte pieces 2724 rows of 4096 behind a sigmoid gate took 56 us and of 2048 behind the gated norm 24, here 20 and 12.
// WARP: a warp a row and eight rows a CTA, for many short rows: with a CTA a row an SM holds 32 of them however small they are
// (24300 rows of 512 behind SiLU, a warp each: 26 us, so 15).
// GATHER: row m comes from row gather[m].
template <int BPT, bool GATED, bool WARP, bool GATHER>
__global__ void __launch_bounds__(WARP ? 256 : 1024) row_kernel_v2(const RowParams p) {
  __shared__ float red[64];
  const int tid = WARP ? threadIdx.x & 31 : threadIdx.x, nt = WARP ? 32 : blockDim.x;
  const int K = p.K, nblk = K >> 4;
  mb::pdl_wait();
  mb::pdl_launch_dependents();
  const int at_row = WARP ? (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) : (int)blockIdx.x;
  if (WARP && at_row >= p.M) return;
  const int m = p.row_index ? p.row_index[at_row] : at_row;
  if (m < 0) return;
  float x[BPT][16];
  float ss = 0.f, mx = 0.f;
  const bool norm = p.in_mode == IN_RMSNORM;
  bool live = true;
  std::conditional_t<GATHER, long long, int> from = m;
  if constexpr (GATHER) from = source_row(p, m, live);
#pragma unroll
  for (int j = 0; j < BPT; ++j) {
    const int b = tid + j * nt;
    if constexpr (GATED) {
      const bool gnorm = p.in_mode == IN_GATED_RMSNORM;
      float gs[16];
      if (b < nblk) {
        if (p.xf32) {
          const float4* src = reinterpret_cast<const float4*>(p.xf32 + (size_t)m * p.x_ld + b * 16);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 f = __ldg(src + i);
            x[j][4 * i] = f.x; x[j][4 * i + 1] = f.y; x[j][4 * i + 2] = f.z; x[j][4 * i + 3] = f.w;
          }
        } else {
          load16(p.x + (size_t)m * p.x_ld + b * 16, x[j]);
        }
        size_t at = (size_t)m * p.gate_ld + b * 16;
        if (!gnorm) {
          const int h = b * 16 / p.head_dim;
          at = (size_t)m * p.gate_ld + (size_t)h * p.gate_head_stride + p.gate_head_off + (b * 16 - h * p.head_dim);
        }
        if (p.gate) load16(p.gate + at, gs);
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) x[j][i] = gs[i] = 0.f;
      }
      if (gnorm) {
        float sq = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) sq += x[j][i] * x[j][i];
        sq += __shfl_xor_sync(0xffffffffu, sq, 1);
        sq += __shfl_xor_sync(0xffffffffu, sq, 2);
        sq += __shfl_xor_sync(0xffffffffu, sq, 4);
        const float ri = rsqrtf(sq / 128.f + p.eps);
        float w[16];
        if (p.w && b < nblk) load16(p.w + b * 16, w);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float y = x[j][i] * ri * (p.w ? (b < nblk ? w[i] : 0.f) : 1.f);
          if (p.gate) y *= mb::silu(gs[i]);
          x[j][i] = y;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) x[j][i] = x[j][i] / (1.f + __expf(-gs[i]));
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) mx = fmaxf(mx, fabsf(x[j][i]));
      continue;
    }
    if (b < nblk) {
      const __nv_bfloat16* src = p.x + (size_t)from * p.x_ld + b * 16;
      uint4 v0 = __ldg(reinterpret_cast<const uint4*>(src));
      uint4 v1 = __ldg(reinterpret_cast<const uint4*>(src) + 1);
      if (!live) v0 = v1 = make_uint4(0, 0, 0, 0);
      if (GATHER && p.gather_out) {
        uint4* d = reinterpret_cast<uint4*>(p.gather_out + (size_t)m * K + b * 16);
        d[0] = v0; d[1] = v1;
      }
      const __nv_bfloat162* h0 = reinterpret_cast<const __nv_bfloat162*>(&v0);
      const __nv_bfloat162* h1 = reinterpret_cast<const __nv_bfloat162*>(&v1);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 a = __bfloat1622float2(h0[i]), c = __bfloat1622float2(h1[i]);
        x[j][2 * i] = a.x; x[j][2 * i + 1] = a.y; x[j][8 + 2 * i] = c.x; x[j][8 + 2 * i + 1] = c.y;
      }
      if (p.in_mode == IN_SILU_MUL) {
        const __nv_bfloat16* up = src + K;
        uint4 u0 = __ldg(reinterpret_cast<const uint4*>(up));
        uint4 u1 = __ldg(reinterpret_cast<const uint4*>(up) + 1);
        const __nv_bfloat162* g0 = reinterpret_cast<const __nv_bfloat162*>(&u0);
        const __nv_bfloat162* g1 = reinterpret_cast<const __nv_bfloat162*>(&u1);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 a = __bfloat1622float2(g0[i]), c = __bfloat1622float2(g1[i]);
          x[j][2 * i] = mb::silu(x[j][2 * i]) * a.x; x[j][2 * i + 1] = mb::silu(x[j][2 * i + 1]) * a.y;
          x[j][8 + 2 * i] = mb::silu(x[j][8 + 2 * i]) * c.x; x[j][8 + 2 * i + 1] = mb::silu(x[j][8 + 2 * i + 1]) * c.y;
        }
      }
      if (norm) {
        float w[16];
        if (p.w) {
          uint4 w0 = __ldg(reinterpret_cast<const uint4*>(p.w + b * 16));
          uint4 w1 = __ldg(reinterpret_cast<const uint4*>(p.w + b * 16) + 1);
          const __nv_bfloat162* q0 = reinterpret_cast<const __nv_bfloat162*>(&w0);
          const __nv_bfloat162* q1 = reinterpret_cast<const __nv_bfloat162*>(&w1);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 a = __bfloat1622float2(q0[i]), c = __bfloat1622float2(q1[i]);
            w[2 * i] = a.x; w[2 * i + 1] = a.y; w[8 + 2 * i] = c.x; w[8 + 2 * i + 1] = c.y;
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) w[i] = 1.f;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          ss += x[j][i] * x[j][i];
          x[j][i] *= p.w_plus_one ? (w[i] + 1.f) : w[i];      // x now holds x * w
        }
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) mx = fmaxf(mx, fabsf(x[j][i]));
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) x[j][i] = 0.f;
    }
  }
  // one block reduction for (sum of squares, max)
  const bool need_red = norm || p.out_mode == OUT_FP8_ROW || p.out_mode == OUT_NVFP4;
  float inv = 1.f, amax = mx;
  if (need_red) {
    ss = mb::warp_sum(ss);
    mx = mb::warp_max(mx);
    float a = ss, c = mx;
    if constexpr (!WARP) {
      const int w = tid >> 5, l = tid & 31, nw = (nt + 31) >> 5;
      if (l == 0) { red[w] = ss; red[32 + w] = mx; }
      __syncthreads();
      a = l < nw ? red[l] : 0.f; c = l < nw ? red[32 + l] : 0.f;
      a = mb::warp_sum(a);
      c = mb::warp_max(c);
    }
    if (norm) inv = rsqrtf(a / (float)K + p.eps);
    amax = c * inv;
  }
  float gs = 1.f, row_inv = 1.f;
  if (p.out_mode == OUT_FP8_ROW) {
    gs = amax > 0.f ? amax / 448.f : 1.f;
    row_inv = 1.f / gs;
    if (tid == 0) p.scale[m] = gs;
  } else if (p.out_mode == OUT_NVFP4) {
    gs = p.static_gs > 0.f ? p.static_gs : (amax > 0.f ? amax / (6.f * 448.f) : 1.f);
    if (tid == 0) p.scale[m] = gs;
  }
#pragma unroll
  for (int j = 0; j < BPT; ++j) {
    const int b = tid + j * nt;
    const bool valid = b < nblk;                       // no early exit: the group shuffles below need whole warps
    float y[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) y[i] = x[j][i] * inv;
    if (valid && (p.out_bf16 || p.out_mode == OUT_BF16)) {
      uint4 o0, o1;
      __nv_bfloat162* q0 = reinterpret_cast<__nv_bfloat162*>(&o0);
      __nv_bfloat162* q1 = reinterpret_cast<__nv_bfloat162*>(&o1);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        q0[i] = __floats2bfloat162_rn(y[2 * i], y[2 * i + 1]);
        q1[i] = __floats2bfloat162_rn(y[8 + 2 * i], y[8 + 2 * i + 1]);
      }
      if (p.out_bf16) {
        uint4* d = reinterpret_cast<uint4*>(p.out_bf16 + (size_t)m * p.out_bf16_ld + b * 16);
        d[0] = o0; d[1] = o1;
      }
      if (p.out_mode == OUT_BF16) {
        uint4* d = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.out) + (size_t)m * p.out_ld + b * 16);
        d[0] = o0; d[1] = o1;
      }
    }
    if (p.out_mode == OUT_FP8_ROW || p.out_mode == OUT_FP8_G128) {
      float sc_inv = row_inv;
      if (p.out_mode == OUT_FP8_G128) {
        float bm = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) bm = fmaxf(bm, fabsf(y[i]));
        // a 128-channel group is 8 consecutive blocks = 8 consecutive lanes
        bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 1));
        bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 2));
        bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 4));
        const float sc = bm > 0.f ? bm / 448.f : 1.f;
        sc_inv = 1.f / sc;
        if (valid && (b & 7) == 0) p.scale[(size_t)(b >> 3) * p.scale_ld + m] = sc;
      }
      uint32_t w4[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        w4[i] = (uint32_t)mb::float_to_e4m3(y[4 * i] * sc_inv) | ((uint32_t)mb::float_to_e4m3(y[4 * i + 1] * sc_inv) << 8) |
                ((uint32_t)mb::float_to_e4m3(y[4 * i + 2] * sc_inv) << 16) | ((uint32_t)mb::float_to_e4m3(y[4 * i + 3] * sc_inv) << 24);
      }
      if (valid)
        *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(p.out) + (size_t)m * p.out_ld + b * 16) =
            make_uint4(w4[0], w4[1], w4[2], w4[3]);
    } else if (p.out_mode == OUT_NVFP4) {
      float bmax = 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) bmax = fmaxf(bmax, fabsf(y[i]));
      const uint8_t sfc = mb::float_to_e4m3(bmax / (6.f * gs));
      const float sff = mb::e4m3_to_float(sfc);
      const float qi = sff > 0.f ? 1.f / (sff * gs) : 0.f;
      uint32_t lo = 0, hi = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) lo |= mb::e2m1x2_pack(y[2 * i] * qi, y[2 * i + 1] * qi) << (8 * i);
#pragma unroll
      for (int i = 0; i < 4; ++i) hi |= mb::e2m1x2_pack(y[8 + 2 * i] * qi, y[8 + 2 * i + 1] * qi) << (8 * i);
      if (valid)
        *reinterpret_cast<uint2*>(reinterpret_cast<uint8_t*>(p.out) + (size_t)m * p.out_ld + b * 8) = make_uint2(lo, hi);
      uint8_t* sf_blk = p.sf + (size_t)(m >> 7) * p.sf_k64 * 512;
      if ((nblk & 3) == 0) {
        // four consecutive blocks sit on four consecutive lanes and fill one 4-byte group of the tiled
        // scale-factor layout: one 32-bit store per group instead of four byte stores
        const uint32_t s1 = __shfl_down_sync(0xffffffffu, (uint32_t)sfc, 1);
        const uint32_t s2 = __shfl_down_sync(0xffffffffu, (uint32_t)sfc, 2);
        const uint32_t s3 = __shfl_down_sync(0xffffffffu, (uint32_t)sfc, 3);
        if (valid && (b & 3) == 0)
          *reinterpret_cast<uint32_t*>(sf_blk + (size_t)(b >> 2) * 512 + mb::sf_tile_offset(m & 127, 0)) =
              (uint32_t)sfc | (s1 << 8) | (s2 << 16) | (s3 << 24);
      } else if (valid) {
        sf_blk[(size_t)(b >> 2) * 512 + mb::sf_tile_offset(m & 127, b & 3)] = sfc;
      }
    }
  }
}

template <int BPT, bool GATED = false, bool WARP = false>
int launch_row_v2(const RowParams& p, int threads, cudaStream_t stream) {
  const dim3 grid(WARP ? (p.M + 7) / 8 : p.M);
  if constexpr (!GATED)
    if (p.gather) return (int)mb::launch_kernel(row_kernel_v2<BPT, GATED, WARP, true>, grid, dim3(threads), 0, stream, p);
  return (int)mb::launch_kernel(row_kernel_v2<BPT, GATED, WARP, false>, grid, dim3(threads), 0, stream, p);
}

// Repack row-major ue4m3 scale factors [N, K/16] into the tiled layout
// [ceil(N/128)][sf_k64][512] (zero padded).
__global__ void sf_repack_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, int N,
                                 int kblocks, int sf_k64) {
  const long long total = (long long)((N + 127) / 128) * sf_k64 * 512;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int within = (int)(i % 512);
    const long long chunk = i / 512;
    const int k64 = (int)(chunk % sf_k64);
    const int nb = (int)(chunk / sf_k64);
    const int kk = within & 3, rq = (within >> 2) & 3, r32 = within >> 4;
    const int r = nb * 128 + rq * 32 + r32;
    const int kb = k64 * 4 + kk;
    dst[i] = (r < N && kb < kblocks) ? src[(size_t)r * kblocks + kb] : 0;
  }
}

// bf16 elementwise add in place: dst += src (2-rank all-reduce tail).
__global__ void add_inplace_kernel(__nv_bfloat16* dst, const __nv_bfloat16* src, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    dst[i] = __float2bfloat16(__bfloat162float(dst[i]) + __bfloat162float(src[i]));
}

// Token embedding gather: out[m, :] = table[ids[m], :]; ids outside the table give zeros
// and set the status word (no out-of-bounds read).
__global__ void embed_kernel(const int* __restrict__ ids, const __nv_bfloat16* __restrict__ table,
                             __nv_bfloat16* __restrict__ out, int hidden, int vocab,
                             uint32_t* status) {
  const int m = blockIdx.x;
  mb::pdl_wait();
  mb::pdl_launch_dependents();
  const int id = ids[m];
  const bool ok = id >= 0 && id < vocab;
  if (!ok && threadIdx.x == 0 && status) atomicCAS(status, 0u, MB_ST_BOUNDS);
  const uint4* src = reinterpret_cast<const uint4*>(table + (size_t)(ok ? id : 0) * hidden);
  uint4* dst = reinterpret_cast<uint4*>(out + (size_t)m * hidden);
  for (int i = threadIdx.x; i < hidden / 8; i += blockDim.x)
    dst[i] = ok ? src[i] : make_uint4(0, 0, 0, 0);
}

}  // namespace

extern "C" {

static int g_pdl = -1;
int mb_pdl_enabled() {
  if (g_pdl < 0) {
    const char* e = getenv("METRALE_PDL");
    g_pdl = (e && e[0] >= '0' && e[0] <= '2') ? e[0] - '0' : 2;   // default: GEMMs launch programmatically   
  }
  return g_pdl;
}
void mb_set_pdl(int mode) { g_pdl = mode < 0 ? 0 : (mode > 2 ? 2 : mode); }

int mb_row_op(const MbRowArgs* a, cudaStream_t stream) {
  if (!a || a->M <= 0 || a->K <= 0 || (!a->x && !a->xf32) || !a->out) return MB_ERR_BAD_ARG;
  if (a->K > 48 * 1024) return MB_ERR_TOO_LARGE;
  if (a->out_mode == OUT_NVFP4 && (a->K % 16 || !a->sf || !a->scale || a->sf_k64 * 64 < a->K))
    return MB_ERR_BAD_ARG;
  if ((a->out_mode == OUT_FP8_ROW || a->out_mode == OUT_FP8_G128) && !a->scale)
    return MB_ERR_BAD_ARG;
  if (a->gather && (a->in_mode != IN_RMSNORM || !a->x || a->residual || a->residual_out || a->row_index || a->gather_rows <= 0)) return MB_ERR_BAD_ARG;
  if (a->in_mode == IN_SIGMOID_GATE && (!a->gate || a->head_dim <= 0)) return MB_ERR_BAD_ARG;
  RowParams p{};
  p.M = a->M; p.K = a->K; p.in_mode = a->in_mode; p.out_mode = a->out_mode;
  p.x = reinterpret_cast<const __nv_bfloat16*>(a->x); p.x_ld = a->x_ld;
  p.residual = reinterpret_cast<const __nv_bfloat16*>(a->residual);
  p.residual_out = reinterpret_cast<__nv_bfloat16*>(a->residual_out);
  p.w = reinterpret_cast<const __nv_bfloat16*>(a->w); p.w_plus_one = a->w_plus_one;
  p.eps = a->eps;
  p.gate = reinterpret_cast<const __nv_bfloat16*>(a->gate); p.gate_ld = a->gate_ld;
  p.head_dim = a->head_dim; p.gate_head_stride = a->gate_head_stride;
  p.gate_head_off = a->gate_head_off; p.group = a->group;
  p.xf32 = a->xf32;
  p.out = a->out; p.out_ld = a->out_ld;
  p.out_bf16 = reinterpret_cast<__nv_bfloat16*>(a->out_bf16); p.out_bf16_ld = a->out_bf16_ld;
  p.scale = a->scale; p.scale_ld = a->scale_ld;
  p.sf = reinterpret_cast<uint8_t*>(a->sf); p.sf_k64 = a->sf_k64;
  p.static_gs = a->static_gs;
  p.row_index = a->row_index;
  p.gather = a->gather; p.gather_wide = a->gather_wide; p.gather_rows = a->gather_rows;
  p.gather_out = a->gather ? reinterpret_cast<__nv_bfloat16*>(a->gather_out) : nullptr;
  p.status = a->status;
  {
    // fast path eligibility: bf16 input, whole 16-element blocks, 16-byte aligned vectors
    const bool modes = p.in_mode == IN_COPY || p.in_mode == IN_RMSNORM || p.in_mode == IN_SILU_MUL;
    const uintptr_t al = reinterpret_cast<uintptr_t>(p.x) | reinterpret_cast<uintptr_t>(p.out) |
                         reinterpret_cast<uintptr_t>(p.out_bf16) | reinterpret_cast<uintptr_t>(p.w) | reinterpret_cast<uintptr_t>(p.gather_out);
    const bool ld_ok = p.x_ld % 8 == 0 && p.out_ld % 8 == 0 && p.out_bf16_ld % 8 == 0;
    const int nblk = a->K / 16;
    // the gated recipes: a block of 16 lies in one head, a statistics group is 128 channels, every vector is aligned
    const bool sig = p.in_mode == IN_SIGMOID_GATE && p.x && !p.xf32 && p.head_dim % 16 == 0 && p.gate_head_stride % 8 == 0 && p.gate_head_off % 8 == 0;
    const bool gnorm = p.in_mode == IN_GATED_RMSNORM && p.group == 128;
    if ((sig || gnorm) && !p.residual && !p.residual_out && a->K % 128 == 0 && nblk <= 512 && p.gate_ld % 8 == 0 && (p.xf32 ? p.x_ld % 4 == 0 : ld_ok) &&
        p.out_ld % 8 == 0 && p.out_bf16_ld % 8 == 0 && !((al | reinterpret_cast<uintptr_t>(p.gate) | reinterpret_cast<uintptr_t>(p.xf32)) & 15))
      return launch_row_v2<1, true>(p, (nblk + 31) / 32 * 32, stream);
    if (modes && !p.xf32 && !p.residual && !p.residual_out && a->K % 16 == 0 && !(al & 15) && ld_ok &&
        (p.out_mode != OUT_FP8_G128 || a->K % 128 == 0) && nblk <= 4096) {
      // A warp would take the row anyway; rows of more than a block a lane are faster over a CTA (2700 of 2048: 7.7 us, a warp each 13). A CTA /
      // a warp each, us, 512 channels to nvfp4: copied 1300 rows 2.6 / 2.4, 2700 3.4 / 2.7, 8192 9.1 / 4.5; behind SiLU, twice the loads
      // and an exponential a value, 1300 2.8 / 2.9 (fp8 groups 2.6 / 2.8), 2700 3.3 / 3.5, 8192 9.2 / 5.7.
      const int many = 148 * (p.in_mode == IN_SILU_MUL ? 20 : 8);
      if (p.M >= many && nblk <= 32) return launch_row_v2<1, false, true>(p, 256, stream);
      const int bpt = (nblk + 511) / 512;
      int threads = ((nblk + bpt - 1) / bpt + 31) / 32 * 32;
      if (p.out_mode == OUT_FP8_G128) threads = (threads + 7) / 8 * 8;
      switch (bpt) {
        case 1: return launch_row_v2<1>(p, threads, stream);
        case 2: return launch_row_v2<2>(p, threads, stream);
        case 3: return launch_row_v2<3>(p, threads, stream);
        case 4: return launch_row_v2<4>(p, threads, stream);
        default: break;
      }
    }
  }
  const size_t smem = (size_t)a->K * sizeof(float);
  static bool configured = false;
  if (!configured) {
    for (auto kern : {row_kernel<false>, row_kernel<true>}) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 48 * 1024 * 4);
      if (e != cudaSuccess) return (int)e;
    }
    configured = true;
  }
  int threads = a->K >= 4096 ? 512 : (a->K >= 1024 ? 256 : 128);
  return (int)mb::launch_kernel(p.gather ? row_kernel<true> : row_kernel<false>, dim3(a->M), dim3(threads), smem, stream, p);
}

int mb_sf_repack(const void* src, void* dst, int N, int kblocks, int sf_k64, cudaStream_t stream) {
  if (!src || !dst || N <= 0 || kblocks <= 0 || sf_k64 * 4 < kblocks) return MB_ERR_BAD_ARG;
  const long long total = (long long)((N + 127) / 128) * sf_k64 * 512;
  int blocks = (int)((total + 255) / 256);
  if (blocks > 148 * 16) blocks = 148 * 16;
  sf_repack_kernel<<<blocks, 256, 0, stream>>>(reinterpret_cast<const uint8_t*>(src),
                                               reinterpret_cast<uint8_t*>(dst), N, kblocks, sf_k64);
  return (int)cudaGetLastError();
}

int mb_add_inplace(void* dst, const void* src, long long n, cudaStream_t stream) {
  if (!dst || !src || n <= 0) return MB_ERR_BAD_ARG;
  int blocks = (int)((n + 255) / 256);
  if (blocks > 148 * 8) blocks = 148 * 8;
  add_inplace_kernel<<<blocks, 256, 0, stream>>>(reinterpret_cast<__nv_bfloat16*>(dst),
                                                 reinterpret_cast<const __nv_bfloat16*>(src), n);
  return (int)cudaGetLastError();
}

int mb_embed(const int* ids, const void* table, void* out, int M, int hidden, int vocab,
             uint32_t* status, cudaStream_t stream) {
  if (!ids || !table || !out || M <= 0 || hidden % 8) return MB_ERR_BAD_ARG;
  return (int)mb::launch_kernel(embed_kernel, dim3(M), dim3(128), 0, stream, ids,
                                reinterpret_cast<const __nv_bfloat16*>(table),
                                reinterpret_cast<__nv_bfloat16*>(out), hidden, vocab, status);
}

}  // extern "C"
