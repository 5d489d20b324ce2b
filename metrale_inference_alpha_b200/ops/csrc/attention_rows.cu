// Prefill attention for the plain case (head dim 128, causal, softmax without sink, cap, window or gate): two tiles of 128
// query rows per CTA in turn on the tensor cores.
//
// The query rows of a sequence and key/value head are numbered token * G + head of the group, so the G query heads that
// read the same keys share a staged tile, and a CTA's 256 rows span only 256 / G tokens: little work is done behind a
// causal limit. Roles (512 threads, one CTA per SM, registers moved to the softmax warps with setmaxnreg):
//   warps 0-3, 4-7   softmax of row tile 0 / 1, thread = row: S from TMEM, P back to TMEM (over S), the output row at the end
//   warps 8-11       K and V tiles of 128 cached tokens into two stages of shared memory, 128-byte swizzle, a row's 16-byte
//                    pieces on neighbouring threads; an e4m3 cache becomes f16 on the way (exact, one conversion per two
//                    values; Q and P are f16 then), a bf16 cache is copied asynchronously
//   warp 12          issues the products: S0 S1 | PV0 S0' | PV1 S1' | ... so that one tile's softmax runs under the other
//                    tile's products. P is the A operand in TMEM, V is read as stored (MN-major).
// A commit covers everything issued before it, so S(j) seen means P V(j - 1) done: the output may be rescaled (only when a
// row's maximum has moved by more than 2^8) without a wait of its own.
//
// f16 has less range than the bf16 that queries come in and the exponentials have, so with an e4m3 cache a row's queries are scaled
// by the power of two that takes their largest to [2^14, 2^15) (elements down to 2^-31 of it keep their 8 bits; the scores' factor
// takes the power back), and the weights are held 2^7 larger than the running maximum says: up to 2^15, and the smallest that is not
// zero is 2^-32 of it.
//
// Bounds: per row tile and 128 tokens, 16384 exponentials are 1024 cycles of the special function units and the two products 1024
// of the tensor cores. Measured against attention_tc.cu (40 / 8 heads): 8192 tokens, e4m3 1720 -> 695 us (0.99 PFLOP/s); 64
// prompts of 128 tokens, e4m3 167 -> 123; two bf16 portions of 1001 and 1531 tokens behind 2500 to 2900, 644 -> 226. With the
// NVFP4 output written here the 36 us quantiser pass over 8192 x 5120 is gone. A CTA whose second row tile has no rows leaves it out:
// 128 tokens of one head a group behind 1000 / 16000, 8 kv heads, bf16 29.3 -> 25.5 / 317 -> 299 us. One form stays slower than in
// attention_tc.cu, whose CTAs share an SM: many prompts of 128 tokens with one head a group (16 prompts, 32 heads: 35 us there, 39 here).
#include "common.cuh"
#include "attention_rows.cuh"
#include "attention_rows.h"

namespace {

constexpr int kRows = 256, kT = 128, kD = 128;
constexpr int kThreads = 512;
constexpr int kTileB = kT * kD * 2;                       // a staged K or V tile
constexpr int kSmem = 2 * 128 * kD * 2 + 4 * kTileB + 1024;
constexpr float kLift = 7.f;                              // log2 of what f16 weights are held larger by

using namespace mbr;
template <int N>
__device__ __forceinline__ void more_regs() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void fewer_regs() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

template <bool FP8>
__global__ void __launch_bounds__(kThreads, 1) attn_rows_kernel(const AttnRowsParams p) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  uint8_t* sQ = smem_raw + ((1024u - (mb::smem_u32(smem_raw) & 1023u)) & 1023u);   // 2 row tiles x 2 halves of 64 dims x [128 x 128 B]
  uint8_t* sK = sQ + 2 * 128 * kD * 2;                    // 2 stages x 2 halves x [128 tokens x 128 B]
  uint8_t* sV = sK + 2 * kTileB;
  __shared__ __align__(8) uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_full[2], o_full[2];
  __shared__ uint32_t s_tmem;
  __shared__ float s_qscale[kRows];                       // what a row's scores are too large by (e4m3 cache)
  const int kvh = blockIdx.x, seq = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  mb::pdl_wait();
  const int qlen = p.q_len[seq], ctx = p.ctx_len[seq], qs = p.q_start[seq];
  const int G = p.Hq / p.Hkv, nrows = qlen * G;
  const int row0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * kRows;   // the longest rows first
  if (row0 >= nrows) return;
  const bool two = nrows - row0 > 128;                    // the second row tile has rows
  const int past = ctx - qlen;
  const int last_limit = past + (min(nrows, row0 + kRows) - 1) / G + 1;
  const int tiles = (last_limit + kT - 1) / kT;
  const int* bt = p.block_table + (size_t)seq * p.max_blocks;

  if (tid == 0) {
    mb::mbar_init(&q_full, 8);
    for (int i = 0; i < 2; ++i) {
      mb::mbar_init(&k_full[i], 4);
      mb::mbar_init(&v_full[i], 4);
      mb::mbar_init(&k_empty[i], 1);
      mb::mbar_init(&v_empty[i], 1);
      mb::mbar_init(&s_full[i], 1);
      mb::mbar_init(&p_full[i], 4);
      mb::mbar_init(&o_full[i], 1);
    }
    mb::mbar_fence_init();
  }
  if (warp == 12) mb::tmem_alloc(&s_tmem, 512);
  mb::tc_fence_before();
  __syncthreads();
  mb::tc_fence_after();
  mb::pdl_launch_dependents();                            // a dependent kernel allocates TMEM: not before this CTA has its own
  const uint32_t tmem = s_tmem;                           // S0 0-127, S1 128-255, O0 256-383, O1 384-511

  if (warp < 8) {
    // ------------------------------------------------------------ softmax
    more_regs<184>();
    const int w = warp >> 2, r = tid & 127, row = row0 + w * 128 + r;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tS = tmem + lanes + w * 128, tO = tmem + lanes + 256 + w * 128;
    // Q: 256 rows x 16 pieces of 8 dims, a thread's sixteen loads in flight together (rows past the last one read it again and
    // become zeros)
    {
      constexpr int kQ = kRows / 16;
      uint4 v[kQ];
#pragma unroll
      for (int i = 0; i < kQ; ++i) {
        const int at = min(row0 + (tid >> 4) + 16 * i, nrows - 1), tq = at / G;
        v[i] = __ldg(reinterpret_cast<const uint4*>(p.q + ((size_t)(qs + tq) * p.Hq + kvh * G + at - tq * G) * kD) + (tid & 15));
      }
#pragma unroll
      for (int i = 0; i < kQ; ++i) {
        const int qr = (tid >> 4) + 16 * i, c = tid & 15;
        if (row0 + qr >= nrows) v[i] = make_uint4(0, 0, 0, 0);
        if constexpr (FP8) {
          // bf16 bits without the sign order like the values: the row's largest over its sixteen threads
          const uint32_t x[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
          uint32_t top = 0;
#pragma unroll
          for (int j = 0; j < 4; ++j) top = __vmaxu2(top, x[j] & 0x7fff7fffu);
#pragma unroll
          for (int d = 1; d < 16; d <<= 1) top = __vmaxu2(top, __shfl_xor_sync(0xffffffffu, top, d));
          const int e = (int)(max(top & 0xffff, top >> 16) >> 7);              // its exponent, biased by 127
          // 2^(141 - e), and its inverse; zeros and subnormal rows as if their exponent were 15, infinities and NaN as they are
          const int up = e == 255 ? 0 : 141 - max(e, 15);
          const float f = __int_as_float((127 + up) << 23);
          uint32_t h[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x[j]));
            h[j] = pack2<true>(y.x * f, y.y * f);
          }
          v[i] = make_uint4(h[0], h[1], h[2], h[3]);
          if (c == 0) s_qscale[qr] = __int_as_float((127 - up) << 23);
        }
        *reinterpret_cast<uint4*>(sQ + (qr >> 7) * (128 * kD * 2) + (c >> 3) * (128 * 128) + sw_off(qr & 127, c & 7)) = v[i];
      }
    }
    fence_async_smem();
    __syncwarp();
    if (lane == 0) mb::mbar_arrive(&q_full);
    if constexpr (FP8) asm volatile("bar.sync 1, 256;" ::: "memory");         // the rows' scales come from other softmax warps
    const bool live = row < nrows;
    const int tok = live ? row / G : 0, limit = live ? past + tok + 1 : 0;   // tokens [0, limit) are visible
    const float sc = p.scale * (FP8 ? *p.k_scale : 1.f) * 1.44269504088896f * (FP8 ? s_qscale[w * 128 + r] : 1.f);
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    const int mine = w == 0 || two ? tiles : 0;
    for (int j = 0; j < mine; ++j) {
      ok = mb::mbar_wait(&s_full[w], j & 1, p.status, MB_ST_TIMEOUT_MMA);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      mb::tc_fence_after();
      float s[kT];
#pragma unroll
      for (int c = 0; c < kT; c += 32) mb::tmem_ld32_async(tS + c, s + c);
      mb::tmem_ld_wait(s);
      const int seen = limit - j * kT;                    // columns below this are visible
      if (!__all_sync(0xffffffffu, seen >= kT)) {
#pragma unroll
        for (int i = 0; i < kT; ++i)
          if (i >= seen) s[i] = -INFINITY;
      }
      float mx4[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
      for (int i = 4; i < kT; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], s[i]);
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sc;
      float alpha = 1.f;
      const bool move = mx > m_run + 8.f;                 // also true on a row's first finite tile
      if (move) {
        alpha = ex2(m_run - mx);                          // 0 when the row had seen nothing yet
        m_run = mx;
      }
      if (j > 0 && __any_sync(0xffffffffu, move)) {
#pragma unroll
        for (int c = 0; c < kD; c += 16) {
          float ov[16];
          mb::tmem_ld16(tO + c, ov);
#pragma unroll
          for (int i = 0; i < 16; ++i) ov[i] *= alpha;
          mb::tmem_st16(tO + c, ov);
        }
      }
      const float nm = m_run == -INFINITY ? 0.f : (FP8 ? kLift : 0.f) - m_run;
      const float2 sc2 = make_float2(sc, sc), nm2 = make_float2(nm, nm);
      float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t pk[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          float2 t = fma2(make_float2(s[h * 64 + 2 * i], s[h * 64 + 2 * i + 1]), sc2, nm2);
          t.x = ex2(t.x);
          t.y = ex2(t.y);
          sum[i & 1] = add2(sum[i & 1], t);
          pk[i] = pack2<FP8>(t.x, t.y);
        }
        tmem_st32(tS + h * 32, pk);
      }
      mb::tmem_st_wait();
      mb::tc_fence_before();
      __syncwarp();
      if (lane == 0) mb::mbar_arrive(&p_full[w]);
      l_run = l_run * alpha + ((sum[0].x + sum[0].y) + (sum[1].x + sum[1].y));
    }
    ok = ok && mine > 0;
    if (ok) {
      ok = mb::mbar_wait(&o_full[w], 0, p.status, MB_ST_TIMEOUT_MMA);
      mb::tc_fence_after();
    }
    if (__all_sync(0xffffffffu, ok)) {                    // uniform: tcgen05.ld is a whole-warp instruction
      const float inv = l_run > 0.f ? (FP8 ? *p.v_scale : 1.f) / l_run : 0.f;
      const size_t m = (size_t)qs + tok;
      const int head = kvh * G + (live ? row - tok * G : 0);
      float o[kD];
#pragma unroll
      for (int c = 0; c < kD; c += 32) mb::tmem_ld32_async(tO + c, o + c);
      mb::tmem_ld_wait(o);
      if (live && p.outq) {
        // eight blocks of 16 dims: packed e2m1 and two 32-bit words of scale factors
        const float inv6gs = 1.f / (6.f * p.outq_gs);
        uint32_t q[16], sf[2] = {0, 0};
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          float mx = 0.f;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            o[b * 16 + i] *= inv;
            mx = fmaxf(mx, fabsf(o[b * 16 + i]));
          }
          const uint8_t sfc = mb::float_to_e4m3(mx * inv6gs);
          const float sff = mb::e4m3_to_float(sfc);
          const float qi = sff > 0.f ? __fdividef(1.f, sff * p.outq_gs) : 0.f;
          sf[b >> 2] |= (uint32_t)sfc << (8 * (b & 3));
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t v = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) v |= mb::e2m1x2_pack(o[b * 16 + h * 8 + 2 * i] * qi, o[b * 16 + h * 8 + 2 * i + 1] * qi) << (8 * i);
            q[b * 2 + h] = v;
          }
        }
        uint4* dst = reinterpret_cast<uint4*>(p.outq + m * p.ldq + head * (kD / 2));
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = make_uint4(q[4 * i], q[4 * i + 1], q[4 * i + 2], q[4 * i + 3]);
        uint8_t* base = p.outq_sf + ((m >> 7) * p.outq_sf_k64 + head * 2) * 512 + mb::sf_tile_offset((uint32_t)(m & 127), 0);
        *reinterpret_cast<uint32_t*>(base) = sf[0];
        *reinterpret_cast<uint32_t*>(base + 512) = sf[1];
      } else if (live) {
        uint4* dst = reinterpret_cast<uint4*>(p.out + m * p.out_ld + (size_t)head * kD);
#pragma unroll
        for (int c = 0; c < kD / 8; ++c) {
          uint32_t v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) v[i] = pack2<false>(o[c * 8 + 2 * i] * inv, o[c * 8 + 2 * i + 1] * inv);
          dst[c] = make_uint4(v[0], v[1], v[2], v[3]);
        }
      }
    }
    mb::tc_fence_before();
  } else if (warp < 12) {
    // ------------------------------------------------------------ loader
    fewer_regs<80>();
    const int t = tid - 256;
    constexpr int kPieces = FP8 ? 8 : 16;                 // 16-byte pieces of a cached row
    constexpr int kStep = 128 / kPieces, kN = kT / kStep; // rows between a thread's pieces, and how many it has
    const int r0 = t / kPieces, c = t % kPieces;
    const size_t pitch = (size_t)p.Hkv * kD * (FP8 ? 1 : 2), at = (size_t)kvh * kD * (FP8 ? 1 : 2) + (size_t)c * 16;
    const int shift = (p.block_size & (p.block_size - 1)) == 0 ? 31 - __clz(p.block_size) : -1;
    // the places in the cache of this thread's rows of tile j (-1: behind the context), looked up a tile before they are read
    int bad = 0;
    auto places = [&](int j, int* place) {
#pragma unroll
      for (int i = 0; i < kN; ++i) {
        const int tok = j * kT + r0 + i * kStep, in = min(tok, ctx - 1);
        const int bi = shift >= 0 ? in >> shift : in / p.block_size;
        int blk = __ldg(bt + bi);
        const bool out = (unsigned)blk >= (unsigned long long)p.num_blocks;
        bad |= out;
        blk = out ? 0 : blk;
        place[i] = tok < ctx ? blk * p.block_size + (in - bi * p.block_size) : -1;
      }
    };
    bool ok = true;
    if constexpr (FP8) {
      uint4 kr[kN], vr[kN];
      int next[kN];
      auto fetch = [&](const void* cache, uint4* raw) {
        const uint8_t* base = reinterpret_cast<const uint8_t*>(cache) + at;
#pragma unroll
        for (int i = 0; i < kN; ++i)
          raw[i] = next[i] >= 0 ? __ldg(reinterpret_cast<const uint4*>(base + (size_t)next[i] * pitch)) : make_uint4(0, 0, 0, 0);
      };
      auto put = [&](uint8_t* tile, const uint4* raw) {
#pragma unroll
        for (int i = 0; i < kN; ++i) {
          const int r = r0 + i * kStep;
          const uint32_t x[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
          uint32_t h[8];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            h[2 * k] = e4m3x2(x[k]);
            h[2 * k + 1] = e4m3x2(x[k] >> 16);
          }
          uint8_t* half = tile + (c >> 2) * (kT * 128);
          *reinterpret_cast<uint4*>(half + sw_off(r, (c & 3) * 2)) = make_uint4(h[0], h[1], h[2], h[3]);
          *reinterpret_cast<uint4*>(half + sw_off(r, (c & 3) * 2 + 1)) = make_uint4(h[4], h[5], h[6], h[7]);
        }
      };
      places(0, next);
      fetch(p.k_cache, kr);
      fetch(p.v_cache, vr);
      places(1, next);
      for (int j = 0; j < tiles; ++j) {
        const int b = j & 1;
        const uint32_t ph = ((j >> 1) & 1) ^ 1;
        ok = mb::mbar_wait(&k_empty[b], ph, p.status, MB_ST_TIMEOUT_TMA);
        if (!__all_sync(0xffffffffu, ok)) break;
        put(sK + b * kTileB, kr);
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mb::mbar_arrive(&k_full[b]);
        fetch(p.k_cache, kr);
        ok = mb::mbar_wait(&v_empty[b], ph, p.status, MB_ST_TIMEOUT_TMA);
        if (!__all_sync(0xffffffffu, ok)) break;
        put(sV + b * kTileB, vr);
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mb::mbar_arrive(&v_full[b]);
        fetch(p.v_cache, vr);
        places(j + 2, next);
      }
    } else {
      int now[kN], next[kN];
      auto copy = [&](const void* cache, uint8_t* tile) {
        const uint8_t* base = reinterpret_cast<const uint8_t*>(cache) + at;
#pragma unroll
        for (int i = 0; i < kN; ++i) {
          const int r = r0 + i * kStep;
          const bool there = now[i] >= 0;
          const uint8_t* src = base + (there ? (size_t)now[i] * pitch : 0);
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(mb::smem_u32(tile + (c >> 3) * (kT * 128) + sw_off(r, c & 7))),
                       "l"(src), "r"(there ? 16 : 0)
                       : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      // the copies of a tile are announced while the next tile's are in flight
      auto announce = [&](uint64_t* bar) {
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mb::mbar_arrive(bar);
      };
      places(0, next);
      for (int j = 0; j < tiles; ++j) {
        const int b = j & 1;
        const uint32_t ph = ((j >> 1) & 1) ^ 1;
#pragma unroll
        for (int i = 0; i < kN; ++i) now[i] = next[i];
        places(j + 1, next);
        ok = mb::mbar_wait(&k_empty[b], ph, p.status, MB_ST_TIMEOUT_TMA);
        if (!__all_sync(0xffffffffu, ok)) break;
        copy(p.k_cache, sK + b * kTileB);
        if (j > 0) {
          asm volatile("cp.async.wait_group 1;" ::: "memory");
          announce(&v_full[b ^ 1]);
        }
        ok = mb::mbar_wait(&v_empty[b], ph, p.status, MB_ST_TIMEOUT_TMA);
        if (!__all_sync(0xffffffffu, ok)) break;
        copy(p.v_cache, sV + b * kTileB);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        announce(&k_full[b]);
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      if (__all_sync(0xffffffffu, ok)) announce(&v_full[(tiles - 1) & 1]);
    }
    if (bad && p.status) atomicCAS(p.status, 0u, MB_ST_BOUNDS);
  } else {
    fewer_regs<48>();
    if (warp == 12 && mb::elect_one()) {
      // ---------------------------------------------------------- products
      constexpr uint32_t kF = FP8 ? 0 : 1;
      constexpr uint32_t kIdS = mb::umma_idesc(kF, kF, 128, kT), kIdO = mb::umma_idesc(kF, kF, 128, kD, 0, 1);
      const uint32_t aQ = mb::smem_u32(sQ), aK = mb::smem_u32(sK), aV = mb::smem_u32(sV);
      bool ok = true;
      auto scores = [&](int w, int j) {
        mb::tc_fence_after();
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int s = 0; s < 4; ++s)
            mb::umma_f16(tmem + w * 128, mb::umma_desc_sw128(aQ + w * (128 * kD * 2) + h * (128 * 128) + s * 32),
                         mb::umma_desc_sw128(aK + (j & 1) * kTileB + h * (kT * 128) + s * 32), kIdS, (h | s) != 0);
        mb::tc_commit(&s_full[w]);
      };
      auto values = [&](int w, int j) {
        mb::tc_fence_after();
#pragma unroll
        for (int s = 0; s < kT / 16; ++s)
          umma_f16_ta(tmem + 256 + w * 128, tmem + w * 128 + s * 8,
                      mb::umma_desc_sw128_mn(aV + (j & 1) * kTileB + s * 2048, kT * 128, 1024), kIdO, (j | s) != 0);
      };
      ok = mb::mbar_wait(&q_full, 0, p.status, MB_ST_TIMEOUT_MMA) && mb::mbar_wait(&k_full[0], 0, p.status, MB_ST_TIMEOUT_MMA);
      if (ok) {
        scores(0, 0);
        if (two) scores(1, 0);
        mb::tc_commit(&k_empty[0]);
      }
      for (int j = 0; j < tiles && ok; ++j) {
        const int b = j & 1;
        const bool more = j + 1 < tiles;
        ok = mb::mbar_wait(&v_full[b], (j >> 1) & 1, p.status, MB_ST_TIMEOUT_MMA) && mb::mbar_wait(&p_full[0], j & 1, p.status, MB_ST_TIMEOUT_MMA);
        if (!ok) break;
        values(0, j);
        if (more) {
          ok = mb::mbar_wait(&k_full[b ^ 1], ((j + 1) >> 1) & 1, p.status, MB_ST_TIMEOUT_MMA);
          if (!ok) break;
          scores(0, j + 1);
        } else {
          mb::tc_commit(&o_full[0]);
        }
        if (two) {
          ok = mb::mbar_wait(&p_full[1], j & 1, p.status, MB_ST_TIMEOUT_MMA);
          if (!ok) break;
          values(1, j);
        }
        mb::tc_commit(&v_empty[b]);
        if (more) {
          if (two) scores(1, j + 1);
          mb::tc_commit(&k_empty[b ^ 1]);
        } else if (two) {
          mb::tc_commit(&o_full[1]);
        }
      }
    }
    __syncwarp();
  }
  __syncthreads();
  if (warp == 12) {
    mb::tc_fence_after();
    mb::tmem_dealloc(tmem, 512);
  }
}

template <bool FP8>
int launch(const AttnRowsParams& p, dim3 grid, cudaStream_t stream) {
  auto kern = attn_rows_kernel<FP8>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  return (int)mb::launch_kernel(kern, grid, dim3(kThreads), kSmem, stream, p);
}

}  // namespace

int mb_attn_rows(const AttnRowsParams& p, int max_q_len, int num_seqs, bool fp8, cudaStream_t stream) {
  const long long rows = (long long)max_q_len * (p.Hq / p.Hkv);
  const long long y = (rows + kRows - 1) / kRows;
  if (y > 65535 || num_seqs > 65535) return MB_ERR_TOO_LARGE;
  const dim3 grid(p.Hkv, (unsigned)y, num_seqs);
  return fp8 ? launch<true>(p, grid, stream) : launch<false>(p, grid, stream);
}
