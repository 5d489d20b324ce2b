// Prefill attention for the plain case at head dim 256 (causal, softmax without sink, cap, window or gate; bf16 cache): 128 query rows
// of a head group per CTA on the tensor cores.
//
// As in attention_rows.cu the query rows of a sequence and key / value head are numbered token * G + head of the group. An output
// tile of 128 x 256 is half of tensor memory, so one row tile fits, not two; its own chain is kept apart instead: the scores of 64
// cached tokens have two buffers, and tile j + 1's are issued in front of tile j's product with V, so that a softmax runs under them.
// Roles (288 threads, one CTA per SM):
//   warps 0-3   softmax, thread = row: S from TMEM, P back over it, the output row at the end
//   warps 4-7   K and V tiles of 64 tokens into two stages of shared memory, 128-byte swizzle, copied asynchronously
//   warp 8      issues the products: S0 | S1 PV0 | S2 PV1 | ...; P is the A operand in TMEM, V is read as stored (MN-major)
// The output is rescaled in TMEM only when a row's maximum has moved by more than 2^8, and then waits for the product before.
//
// Bounds: per 64 tokens the two products are 1024 cycles of the tensor cores, 8192 exponentials 512 of the special function units.
// Measured against attention_tc.cu (us, 16 / 2 heads): one prompt of 128 tokens 21 -> 10, three of 500 to 1300 233 -> 54, 64 of 128 153 -> 71, one
// of 4096 661 -> 204, 256 tokens behind 4000 281 -> 110.
#include "common.cuh"
#include "attention_rows.cuh"
#include "attention_rows.h"

namespace {

using namespace mbr;

constexpr int kRows = 128, kT = 64, kD = 256;
constexpr int kThreads = 288;
constexpr int kSpans = kD / 64;                           // 128-byte spans of a bf16 row
constexpr int kTileB = kT * kD * 2;                       // a staged K or V tile
constexpr int kQB = kRows * kD * 2;
constexpr int kSmem = kQB + 4 * kTileB + 1024;
constexpr int kOut = 256;                                 // TMEM: S0 0-63, S1 64-127, O 256-511

__global__ void __launch_bounds__(kThreads, 1) attn_rows256_kernel(const AttnRowsParams p) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  uint8_t* sQ = smem_raw + ((1024u - (mb::smem_u32(smem_raw) & 1023u)) & 1023u);   // 4 spans x [128 rows x 128 B]
  uint8_t* sK = sQ + kQB;                                 // 2 stages x 4 spans x [64 tokens x 128 B]
  uint8_t* sV = sK + 2 * kTileB;
  __shared__ __align__(8) uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_full[2], o_done;
  __shared__ uint32_t s_tmem;
  const int kvh = blockIdx.x, seq = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  mb::pdl_wait();
  const int qlen = p.q_len[seq], ctx = p.ctx_len[seq], qs = p.q_start[seq];
  const int G = p.Hq / p.Hkv, nrows = qlen * G;
  const int row0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * kRows;   // the longest rows first
  if (row0 >= nrows) return;
  const int past = ctx - qlen;
  const int last_limit = past + (min(nrows, row0 + kRows) - 1) / G + 1;
  const int tiles = (last_limit + kT - 1) / kT;
  const int* bt = p.block_table + (size_t)seq * p.max_blocks;

  if (tid == 0) {
    mb::mbar_init(&q_full, 4);
    mb::mbar_init(&o_done, 1);
    for (int i = 0; i < 2; ++i) {
      mb::mbar_init(&k_full[i], 4);
      mb::mbar_init(&v_full[i], 4);
      mb::mbar_init(&k_empty[i], 1);
      mb::mbar_init(&v_empty[i], 1);
      mb::mbar_init(&s_full[i], 1);
      mb::mbar_init(&p_full[i], 4);
    }
    mb::mbar_fence_init();
  }
  if (warp == 8) mb::tmem_alloc(&s_tmem, 512);
  mb::tc_fence_before();
  __syncthreads();
  mb::tc_fence_after();
  mb::pdl_launch_dependents();                            // a dependent kernel allocates TMEM: not before this CTA has its own
  const uint32_t tmem = s_tmem;

  if (warp < 4) {
    // ------------------------------------------------------------ softmax
    const int row = row0 + tid;
    const uint32_t lanes = (uint32_t)(warp * 32) << 16;
    const uint32_t tO = tmem + lanes + kOut;
    // Q: 128 rows x 32 pieces of 8 dims, sixteen of a thread's loads in flight together (rows past the last one are zeros)
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      uint4 v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int at = min(row0 + (tid >> 5) + 4 * (half * 16 + i), nrows - 1), tq = at / G;
        v[i] = __ldg(reinterpret_cast<const uint4*>(p.q + ((size_t)(qs + tq) * p.Hq + kvh * G + at - tq * G) * kD) + lane);
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int qr = (tid >> 5) + 4 * (half * 16 + i);
        if (row0 + qr >= nrows) v[i] = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4*>(sQ + (lane >> 3) * (kRows * 128) + sw_off(qr, lane & 7)) = v[i];
      }
    }
    fence_async_smem();
    __syncwarp();
    if (lane == 0) mb::mbar_arrive(&q_full);
    const bool live = row < nrows;
    const int tok = live ? row / G : 0, limit = live ? past + tok + 1 : 0;   // tokens [0, limit) are visible
    const float sc = p.scale * 1.44269504088896f;
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < tiles; ++j) {
      const uint32_t tS = tmem + lanes + (j & 1) * kT;
      ok = mb::mbar_wait(&s_full[j & 1], (j >> 1) & 1, p.status, MB_ST_TIMEOUT_MMA);
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
        ok = mb::mbar_wait(&o_done, (j - 1) & 1, p.status, MB_ST_TIMEOUT_MMA);     // P V of tile j - 1 (S(j) seen: that of j - 2 is done)
        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
        mb::tc_fence_after();
#pragma unroll
        for (int c = 0; c < kD; c += 16) {
          float ov[16];
          mb::tmem_ld16(tO + c, ov);
#pragma unroll
          for (int i = 0; i < 16; ++i) ov[i] *= alpha;
          mb::tmem_st16(tO + c, ov);
        }
      }
      const float nm = m_run == -INFINITY ? 0.f : -m_run;
      const float2 sc2 = make_float2(sc, sc), nm2 = make_float2(nm, nm);
      float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      uint32_t pk[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        float2 t = fma2(make_float2(s[2 * i], s[2 * i + 1]), sc2, nm2);
        t.x = ex2(t.x);
        t.y = ex2(t.y);
        sum[i & 1] = add2(sum[i & 1], t);
        pk[i] = pack2<false>(t.x, t.y);
      }
      tmem_st32(tS, pk);
      mb::tmem_st_wait();
      mb::tc_fence_before();
      __syncwarp();
      if (lane == 0) mb::mbar_arrive(&p_full[j & 1]);
      l_run = l_run * alpha + ((sum[0].x + sum[0].y) + (sum[1].x + sum[1].y));
    }
    // a wait tells a phase from its neighbours only, and S(j) seen means P V(j - 2) done: one phase after the other
    if (ok && tiles > 1) ok = mb::mbar_wait(&o_done, tiles & 1, p.status, MB_ST_TIMEOUT_MMA);
    if (ok) ok = mb::mbar_wait(&o_done, (tiles - 1) & 1, p.status, MB_ST_TIMEOUT_MMA);
    mb::tc_fence_after();
    if (__all_sync(0xffffffffu, ok)) {                    // uniform: tcgen05.ld is a whole-warp instruction
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      const size_t m = (size_t)qs + tok;
      const int head = kvh * G + (live ? row - tok * G : 0);
      uint4* dst = reinterpret_cast<uint4*>(p.out + m * p.out_ld + (size_t)head * kD);
#pragma unroll 1
      for (int c0 = 0; c0 < kD; c0 += 64) {
        float o[64];
        mb::tmem_ld32_async(tO + c0, o);
        mb::tmem_ld32_async(tO + c0 + 32, o + 32);
        mb::tmem_ld_wait(o);
        if (live) {
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            uint32_t v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = pack2<false>(o[c * 8 + 2 * i] * inv, o[c * 8 + 2 * i + 1] * inv);
            dst[c0 / 8 + c] = make_uint4(v[0], v[1], v[2], v[3]);
          }
        }
      }
    }
    mb::tc_fence_before();
  } else if (warp < 8) {
    // ------------------------------------------------------------ loader: a warp copies whole rows, 32 pieces of 16 bytes
    const int r0 = warp - 4;
    constexpr int kN = kT / 4;                            // rows of a warp, every fourth of a tile
    const size_t pitch = (size_t)p.Hkv * kD * 2, at = (size_t)kvh * kD * 2 + (size_t)lane * 16;
    const int shift = (p.block_size & (p.block_size - 1)) == 0 ? 31 - __clz(p.block_size) : -1;
    // the places in the cache of this warp's rows of tile j (-1: behind the context), lane i those of row i, looked up a tile ahead
    int bad = 0;
    auto places = [&](int j) {
      const int tok = j * kT + r0 + (lane & (kN - 1)) * 4, in = min(tok, ctx - 1);
      const int bi = shift >= 0 ? in >> shift : in / p.block_size;
      int blk = __ldg(bt + bi);
      const bool out = (unsigned)blk >= (unsigned long long)p.num_blocks;
      bad |= out;
      blk = out ? 0 : blk;
      return tok < ctx ? blk * p.block_size + (in - bi * p.block_size) : -1;
    };
    auto copy = [&](const void* cache, uint8_t* tile, int place) {
      const uint8_t* base = reinterpret_cast<const uint8_t*>(cache) + at;
#pragma unroll
      for (int i = 0; i < kN; ++i) {
        const int r = r0 + i * 4, from = __shfl_sync(0xffffffffu, place, i);
        const bool there = from >= 0;
        const uint8_t* src = base + (there ? (size_t)from * pitch : 0);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(mb::smem_u32(tile + (lane >> 3) * (kT * 128) + sw_off(r, lane & 7))),
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
    bool ok = true;
    int next = places(0);
    for (int j = 0; j < tiles; ++j) {
      const int b = j & 1, now = next;
      const uint32_t ph = ((j >> 1) & 1) ^ 1;
      next = places(j + 1);
      ok = mb::mbar_wait(&k_empty[b], ph, p.status, MB_ST_TIMEOUT_TMA);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      copy(p.k_cache, sK + b * kTileB, now);
      if (j > 0) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        announce(&v_full[b ^ 1]);
      }
      ok = mb::mbar_wait(&v_empty[b], ph, p.status, MB_ST_TIMEOUT_TMA);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      copy(p.v_cache, sV + b * kTileB, now);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      announce(&k_full[b]);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (ok) announce(&v_full[(tiles - 1) & 1]);
    if (bad && p.status) atomicCAS(p.status, 0u, MB_ST_BOUNDS);
  } else {
    if (mb::elect_one()) {
      // ---------------------------------------------------------- products
      constexpr uint32_t kIdS = mb::umma_idesc(1, 1, 128, kT), kIdO = mb::umma_idesc(1, 1, 128, kD, 0, 1);
      const uint32_t aQ = mb::smem_u32(sQ), aK = mb::smem_u32(sK), aV = mb::smem_u32(sV);
      auto scores = [&](int j) {
        mb::tc_fence_after();
#pragma unroll
        for (int h = 0; h < kSpans; ++h)
#pragma unroll
          for (int s = 0; s < 4; ++s)
            mb::umma_f16(tmem + (j & 1) * kT, mb::umma_desc_sw128(aQ + h * (kRows * 128) + s * 32),
                         mb::umma_desc_sw128(aK + (j & 1) * kTileB + h * (kT * 128) + s * 32), kIdS, (h | s) != 0);
        mb::tc_commit(&s_full[j & 1]);
        mb::tc_commit(&k_empty[j & 1]);
      };
      bool ok = mb::mbar_wait(&q_full, 0, p.status, MB_ST_TIMEOUT_MMA) && mb::mbar_wait(&k_full[0], 0, p.status, MB_ST_TIMEOUT_MMA);
      if (ok) scores(0);
      for (int j = 0; j < tiles && ok; ++j) {
        const int b = j & 1;
        if (j + 1 < tiles) {                              // over P of tile j - 1, whose product was issued in front
          ok = mb::mbar_wait(&k_full[b ^ 1], ((j + 1) >> 1) & 1, p.status, MB_ST_TIMEOUT_MMA);
          if (!ok) break;
          scores(j + 1);
        }
        ok = mb::mbar_wait(&v_full[b], (j >> 1) & 1, p.status, MB_ST_TIMEOUT_MMA) &&
             mb::mbar_wait(&p_full[b], (j >> 1) & 1, p.status, MB_ST_TIMEOUT_MMA);
        if (!ok) break;
        mb::tc_fence_after();
#pragma unroll
        for (int s = 0; s < kT / 16; ++s)
          umma_f16_ta(tmem + kOut, tmem + b * kT + s * 8, mb::umma_desc_sw128_mn(aV + b * kTileB + s * 2048, kT * 128, 1024), kIdO, (j | s) != 0);
        mb::tc_commit(&v_empty[b]);
        mb::tc_commit(&o_done);
      }
    }
    __syncwarp();
  }
  __syncthreads();
  if (warp == 8) {
    mb::tc_fence_after();
    mb::tmem_dealloc(tmem, 512);
  }
}

}  // namespace

int mb_attn_rows256(const AttnRowsParams& p, int max_q_len, int num_seqs, cudaStream_t stream) {
  const long long rows = (long long)max_q_len * (p.Hq / p.Hkv);
  const long long y = (rows + kRows - 1) / kRows;
  if (y > 65535 || num_seqs > 65535) return MB_ERR_TOO_LARGE;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(attn_rows256_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  return (int)mb::launch_kernel(attn_rows256_kernel, dim3(p.Hkv, (unsigned)y, num_seqs), dim3(kThreads), kSmem, stream, p);
}
