// Decode and verify attention for the plain case (softmax without sink, cap, window or gate; head dim 128 or 256; blocks of a
// multiple of 16 tokens): at most 32 query rows (tokens x heads of a group) against a paged bf16 or e4m3 cache.
//
// What bounds it at decode is instructions and their latency: few warps run per scheduler, and the split-KV kernel of
// attention.cu (which keeps the other cases) spends 2400 instructions per warp around its tiles. Here:
//   * the four warps of a CTA stream on their own: warp w takes every fourth step of 16 or 32 tokens of its partition, one TMA box
//     per 16 tokens and 128 bytes of row width for K and for V, issued by one lane into the warp's own ring. No CTA barrier until
//     the partition ends.
//   * a fixed number of CTAs walks the list of (sequence, partition, kv head) units. Each CTA finds its units from the lengths
//     alone (a prefix sum in shared memory), so neither idle partitions of a fixed launch geometry nor long ones cost a wave.
//     The next unit's first slices are under way while this one's warps are merged.
//   * partitions depend on the sequence's own length only (never on the batch): part_tokens each, but at most 32 of them;
//     the last to arrive merges them in order.
// The products are mma.sync m16n8k16. Up to 8 query rows of a group, and 17 to 24, have the cache on the 16-row side: scores are
// [16 tokens x 8 query rows], outputs [16 dims x 8 query rows], so five query rows (40 / 8 heads) waste three columns of eight, not
// eleven rows of sixteen, and every product, exponential and accumulator register is half of what the other way round takes; weights
// pass from the first product's layout to the second's through movmatrix. 9 to 16 and 25 to 32 rows fill tiles of 16 as well, and
// without the transpositions and the longer reductions over tokens these are faster with the queries there. Cache / queries on the
// 16-row side, us, four cache heads, one sequence of 700 tokens and 128 of 129 to 1151:
//   e4m3  8 rows 9.8, 31.8 / 10.5, 37.4;  10 rows 13.1, 41.6 / 11.9, 38.6;  20 rows 14.9, 80 / 16.8, 88;  32 rows 23.9, 131 / 17.6, 118
//   bf16  8 rows 11.1, 39.1 / 11.4, 40.4;  10 rows 15.5, 47.0 / 12.5, 41.3;  20 rows 17.7, 105 / 17.4, 106;  32 rows 23.9, 144 / 19.8, 121
// An e4m3 row is widened to f16 in registers, so with an e4m3 cache queries and weights are f16 as in attention.cu: a query element beyond
// 65504 makes its row NaN, weights below 2^-24 of the running maximum vanish.
// Measured against that kernel (us, single calls replayed from a graph): e4m3, 40 / 8 heads of 128: one sequence of 700 tokens 15.4 -> 10.3,
// 128 of 129 to 1151 70 -> 44, nine of 4000 to 16000 75 -> 48, eight verify steps of 4 rows 27 -> 17; bf16, 33 of 100 to 2047 95 -> 34;
// 16 / 2 heads of 256, bf16, sixteen of 200 to 2000 63 -> 17.
#include "common.cuh"
#include "attention_decode.h"
#include "tensormap.h"
#include <type_traits>

namespace {

constexpr int kMaxParts = 32, kMaxSeqs = 1024, kSlice = 16, kMaxSlots = 6;
constexpr size_t kCntBytes = 64 * 1024;      // arrival counters at the head of the workspace, as in attention.cu

struct DecodeParams {
  const __nv_bfloat16* q;
  const int* block_table;
  int max_blocks;
  const int* q_start;
  const int* q_len;
  const int* ctx_len;
  int num_seqs, Hq, Hkv, G, g_magic;         // r / G = r * g_magic >> 16 for r < 64
  int block_size, block_shift;               // shift -1: no power of two
  long long num_blocks;
  float scale;
  const float* k_scale;
  const float* v_scale;
  __nv_bfloat16* out;
  long long out_ld;
  uint8_t* outq;
  int ldq;
  uint8_t* outq_sf;
  int outq_sf_k64;
  float outq_gs;
  float* part_o;                             // [rows * Hq, parts, D]
  float2* part_ml;                           // [rows * Hq, parts]: log2-domain maximum, sum
  uint32_t* part_cnt;                        // [seqs * Hkv]
  int parts, part_tokens;
  int slots;                                 // of every warp's ring
  int ahead;                                 // slots of the ring that the next unit may fill while warps are merged
  int early;                                 // all but q and the cache's rows of this step's tokens stood before the kernel in front began
  uint32_t merge_off, tail_off, len_off;     // byte offsets of the merge buffer and of what lies behind both
  int over;                                  // the merge buffer lies over slots of the ring
  uint32_t* status;
};

__device__ __forceinline__ void mma16816_f16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma16816_bf16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <bool F16>
__device__ __forceinline__ void mma(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  if constexpr (F16) mma16816_f16(c, a, b0, b1);
  else mma16816_bf16(c, a, b0, b1);
}
__device__ __forceinline__ void ldsm4(uint32_t* r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t* r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
template <bool F16>
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  if constexpr (F16) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  } else {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
}
__device__ __forceinline__ uint32_t e4m3x2(uint32_t two) {
  uint32_t r;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(r) : "h"((uint16_t)two));
  return r;
}
__device__ __forceinline__ uint32_t transposed8x8(uint32_t a) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(a));
  return r;
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// NT: eights of query rows
template <int D, bool FP8, int NT>
struct DecodeCfg {
  static constexpr bool kPairs = NT % 2 == 0;                // queries on the products' 16-row side, else the cache
  static constexpr int kTiles = kPairs ? NT / 2 : NT;        // tiles of 16 or of 8 query rows
  static constexpr int kRowB = FP8 ? D : 2 * D;              // bytes of a cached row
  static constexpr int kSpans = kRowB / 128;                 // TMA boxes (and swizzled spans) across it
  // slices that a warp takes together: two chains of products in flight, and one maximum and one wait for 32 tokens
  static constexpr int kSub = FP8 && D == 128 ? 2 : 1;
  static constexpr int kTok = kSub * kSlice;
  static constexpr int kHalf = kTok * kRowB;                 // K or V of one step
  static constexpr int kSlot = 2 * kHalf;
  static constexpr int ring(int slots) { return 4 * slots * kSlot; }           // slot s of warp w at (s * 4 + w) * kSlot
  static constexpr int kCtas = D == 256 ? 1 : NT > 2 ? 2 : 3;
  static constexpr int kQPitch = 2 * D + 16;                 // bytes between query rows in shared memory
  // Place of a dim in a row of the merge buffer: a warp writes dims of one group from the rows 2 t, whose banks must differ. (Longer rows
  // would do too, but at 256 dims and 16 rows the buffer is just what fits over a slot.)
  static __device__ __forceinline__ int place(int r, int dim) { return kPairs ? dim : dim ^ ((r & 6) << 2); }
};

template <int D, bool FP8, int NT>
__global__ void __launch_bounds__(128, DecodeCfg<D, FP8, NT>::kCtas)
attn_decode_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const DecodeParams p) {
  using C = DecodeCfg<D, FP8, NT>;
  constexpr int kSpans = C::kSpans, kSub = C::kSub, kTok = C::kTok, kTiles = C::kTiles;
  constexpr bool kPairs = C::kPairs, kThroughBf16 = NT > 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t bars[4 * kMaxSlots];
  const int slots = p.slots;
  __shared__ int s_last, s_wsum[4];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  float* s_o = reinterpret_cast<float*>(smem + p.merge_off);                  // [4 warps][rows][D], see C::place
  int* s_off = reinterpret_cast<int*>(smem + p.tail_off);                     // [seqs + 1]
  float2* s_ml = reinterpret_cast<float2*>(s_off + ((p.num_seqs + 2) & ~1));  // [4][NT * 8]
  int4* s_len = reinterpret_cast<int4*>(smem + p.len_off);                    // [seqs]: q_len, ctx_len, q_start
  uint8_t* s_q = smem + p.len_off + p.num_seqs * 16;                          // the unit's query rows, as loaded
  if (tid == 0) {
    for (int i = 0; i < 4 * slots; ++i) mb::mbar_init(&bars[i], 1);
    mb::mbar_fence_init();
    mb::tma_prefetch_desc(&tmK);
    mb::tma_prefetch_desc(&tmV);
  }
  if (!p.early) mb::pdl_wait();

  // ---- the list of units: partitions of every sequence in front of it
  auto part_size = [&](int len) { return max(p.part_tokens, ((len + kMaxParts - 1) / kMaxParts + 63) & ~63); };
  auto count = [&](int len, int P) { return len <= P ? 1 : (len + P - 1) / P; };
  {
    int base = 0;
    for (int s0 = 0; s0 < p.num_seqs; s0 += 128) {
      const int s = s0 + tid;
      int n = 0;
      if (s < p.num_seqs) {
        const int4 x = make_int4(p.q_len[s], p.ctx_len[s], p.q_start[s], 0);
        const int len = max(1, x.y);
        s_len[s] = x;
        if (x.x > 0) n = min(count(len, part_size(len)), p.parts);
      }
      int x = n;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
      }
      if (lane == 31) s_wsum[warp] = x;
      __syncthreads();
      int before = base;
      for (int w = 0; w < warp; ++w) before += s_wsum[w];
      if (s < p.num_seqs) s_off[s + 1] = before + x;
      base += s_wsum[0] + s_wsum[1] + s_wsum[2] + s_wsum[3];
      __syncthreads();
    }
    if (tid == 0) s_off[0] = 0;
    __syncthreads();
  }
  const int units = s_off[p.num_seqs] * p.Hkv;

  // ---- one unit: its place and this warp's slices of it
  struct Unit {
    int seq, part, nparts, kvh, begin, slices;               // slices: of this warp
    int qlen, ctx, qs;
    int blk, within;                                         // lane l: block and first token in it of this warp's slice l
  };
  auto find = [&](int u, Unit& x) {
    const int at = u / p.Hkv;
    x.kvh = u - at * p.Hkv;
    int lo = 0, hi = p.num_seqs;                             // s_off[lo] <= at < s_off[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (s_off[mid] <= at) lo = mid;
      else hi = mid;
    }
    x.seq = lo;
    x.part = at - s_off[lo];
    x.nparts = s_off[lo + 1] - s_off[lo];
    const int4 ln = s_len[lo];
    x.qlen = ln.x;
    x.ctx = ln.y;
    x.qs = ln.z;
    const int len = (((x.ctx + x.nparts - 1) / x.nparts) + 63) & ~63;
    x.begin = x.part * len;
    const int end = min(x.ctx, x.begin + len), n = (max(0, end - x.begin) + kTok - 1) / kTok;
    x.slices = (n - warp + 3) >> 2;
  };
  // places of the slices of this warp's steps i0 .. i0 + 32 / kSub - 1, one per lane
  auto blocks = [&](Unit& x, int i0) {
    const int i = i0 + lane / kSub, tok = x.begin + (warp + 4 * i) * kTok + lane % kSub * kSlice;
    x.blk = x.within = 0;                                    // a slice behind the context reads the null block
    if (i < x.slices && tok < x.ctx) {
      const int bi = p.block_shift >= 0 ? tok >> p.block_shift : tok / p.block_size;
      int b = __ldg(p.block_table + (size_t)x.seq * p.max_blocks + bi);
      if (b < 0 || b >= p.num_blocks) {
        if (p.status) atomicCAS(p.status, 0u, MB_ST_BOUNDS);
        b = 0;
      }
      x.blk = b;
      x.within = tok - bi * p.block_size;
    }
  };
  const uint32_t my = mb::smem_u32(smem) + warp * C::kSlot;
  auto issue = [&](const Unit& x, int i, int slot) {         // whole warp; one lane issues
    const int place = x.blk * p.block_size + x.within;
    uint64_t* bar = &bars[slot * 4 + warp];
    uint8_t* dst = smem + (slot * 4 + warp) * C::kSlot;
    if (lane == 0) mb::mbar_expect_tx(bar, C::kSlot);
#pragma unroll
    for (int b = 0; b < kSub; ++b) {
      const int tok = __shfl_sync(0xffffffffu, place, (i * kSub + b) & 31);
      if (lane == 0) {
#pragma unroll
        for (int h = 0; h < kSpans; ++h) {
          mb::tma_load_3d(dst + (b * kSpans + h) * (kSlice * 128), &tmK, bar, h * 128, x.kvh, tok);
          mb::tma_load_3d(dst + C::kHalf + (b * kSpans + h) * (kSlice * 128), &tmV, bar, h * 128, x.kvh, tok);
        }
      }
    }
  };
  // the unit's query rows into shared memory: the whole CTA, 16 bytes a copy
  auto fetch_q = [&](const Unit& x) {
    const int n = p.G * x.qlen * (D / 8);
    for (int i = tid; i < n; i += 128) {
      const int r = i / (D / 8), c = i % (D / 8), tq = (r * p.g_magic) >> 16;
      const __nv_bfloat16* src = p.q + ((size_t)(x.qs + tq) * p.Hq + x.kvh * p.G + (r - tq * p.G)) * D + c * 8;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(mb::smem_u32(s_q + r * C::kQPitch + c * 16)), "l"(src) : "memory");
    }
  };

  const float kmul = FP8 ? *p.k_scale : 1.f, vmul = FP8 ? *p.v_scale : 1.f;
  const float sc_log2 = p.scale * kmul * 1.44269504088896f;
  uint32_t phase = 0;                                        // bit s: parity of slot s's next completion
  Unit cur;
  int u = blockIdx.x, begun = 0;
  if (u < units) {
    find(u, cur);
    blocks(cur, 0);
    // slices of tokens that were cached before this step travel under the end of the kernel in front, which writes the step's own
    const int old = max(0, cur.ctx - cur.qlen - cur.begin) / kTok;
    if (p.early)
      for (; begun < min(min(cur.slices, slots), (old - warp + 3) >> 2); ++begun) issue(cur, begun, begun);
  }
  if (p.early) mb::pdl_wait();
  mb::pdl_launch_dependents();
  if (u < units) {
    for (; begun < min(cur.slices, slots); ++begun) issue(cur, begun, begun);
    fetch_q(cur);
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  __syncthreads();
  bool ok = true;
  int started = slots;                                      // slices of `cur` that are under way already, at most
  while (u < units) {
    const int R = p.G * cur.qlen;
    // A lane has scores and outputs of two rows of a tile, g and g + 8 or 2 t and 2 t + 1; of row e the elements at(e, 0) and at(e, 1) of
    // every fragment. The lanes of a row differ in the bits of `t` or in those of `g`.
    auto row_of = [&](int tile, int e) { return kPairs ? tile * 16 + g + 8 * e : tile * 8 + 2 * t + e; };
    auto at = [](int e, int j) { return kPairs ? 2 * e + j : 2 * j + e; };
    auto over_row = [&](auto x, auto&& f) {
#pragma unroll
      for (int o = kPairs ? 1 : 4; o < (kPairs ? 4 : 32); o <<= 1) x = f(x, __shfl_xor_sync(0xffffffffu, x, o));
      return x;
    };
    // ---- queries as A fragments (rows g and g + 8 of each tile of 16) or B fragments (row g of each tile of 8)
    uint32_t qf[kTiles][D / 16][kPairs ? 4 : 2];
    int lim[kTiles][2], min_limit = 0x7fffffff;
#pragma unroll
    for (int tile = 0; tile < kTiles; ++tile) {
#pragma unroll
      for (int hr = 0; hr < (kPairs ? 2 : 1); ++hr) {
        const int r = kPairs ? tile * 16 + g + hr * 8 : tile * 8 + g;
        const bool live = r < R;
        const uint8_t* qrow = s_q + r * C::kQPitch;
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          uint32_t a = 0, b = 0;
          if (live) {
            if constexpr (FP8) {                             // four neighbouring dims: the order e4m3 fragments come in
              const uint2 v = *reinterpret_cast<const uint2*>(qrow + ks * 32 + 8 * t);
              const float2 f0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x));
              const float2 f1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
              a = pack2<true>(f0.x, f0.y);
              b = pack2<true>(f1.x, f1.y);
            } else {
              a = *reinterpret_cast<const uint32_t*>(qrow + ks * 32 + 4 * t);
              b = *reinterpret_cast<const uint32_t*>(qrow + ks * 32 + 4 * t + 16);
            }
          }
          qf[tile][ks][hr] = a;
          qf[tile][ks][kPairs ? 2 + hr : 1] = b;
        }
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = row_of(tile, e);
        lim[tile][e] = r < R ? cur.ctx - cur.qlen + ((r * p.g_magic) >> 16) + 1 : 0x7fffffff;    // rows past R are never stored
        min_limit = min(min_limit, lim[tile][e]);
      }
    }
    // over all rows of the tiles
#pragma unroll
    for (int o = kPairs ? 4 : 1; o < (kPairs ? 32 : 4); o <<= 1) min_limit = min(min_limit, __shfl_xor_sync(0xffffffffu, min_limit, o));

    // o: 8 dims a fragment, or 16 (dims 2 g, 2 g + 1 of an e4m3 group of 16, else g, g + 8)
    constexpr int kO = kPairs ? D / 8 : D / 16;
    float o[kTiles][kO][4], m_run[kTiles][2], l_run[kTiles][2];
#pragma unroll
    for (int tile = 0; tile < kTiles; ++tile) {
      m_run[tile][0] = m_run[tile][1] = -INFINITY;
      l_run[tile][0] = l_run[tile][1] = 0.f;
#pragma unroll
      for (int n = 0; n < kO; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[tile][n][i] = 0.f;
    }

    for (int i = started; i < min(cur.slices, slots); ++i) issue(cur, i, i);
    int slot = 0;
    for (int i = 0; i < cur.slices; ++i) {
      ok = ok && mb::mbar_wait(&bars[slot * 4 + warp], (phase >> slot) & 1, p.status, MB_ST_TIMEOUT_TMA);
      phase ^= 1u << slot;
      const uint32_t kT = my + slot * 4 * C::kSlot, vT = kT + C::kHalf;
      const int pos0 = cur.begin + (warp + 4 * i) * kTok;
      if (pos0 + kTok > cur.ctx) {
        // rows behind the context hold whatever the block holds: a weight of zero must not meet a NaN there
        const int from = cur.ctx - pos0;
        for (int c = lane; c < (kTok - from) * 8 * kSpans; c += 32) {
          const int r = from + c / (8 * kSpans), cc = c % (8 * kSpans);
          asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(vT + ((r >> 4) * kSpans + (cc >> 3)) * (kSlice * 128) + (r & 15) * 128 + (cc & 7) * 16),
                       "r"(0)
                       : "memory");
        }
        __syncwarp();
      }
      constexpr int kS = kPairs ? 2 * kSub : kSub;           // fragments of 8 or of 16 tokens
      float s[kTiles][kS][4];
#pragma unroll
      for (int tile = 0; tile < kTiles; ++tile)
#pragma unroll
        for (int n = 0; n < kS; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) s[tile][n][e] = 0.f;
      const int krow = (lane & 7) + ((lane >> 4) << 3), kc = (lane >> 3) & 1, ksw = lane & 7;
      // keys of 16 tokens at 16 dims: k0, k1 of the first eight tokens, k2, k3 of the others
      auto score = [&](int b, int ks, uint32_t k0, uint32_t k1, uint32_t k2, uint32_t k3) {
#pragma unroll
        for (int tile = 0; tile < kTiles; ++tile) {
          if constexpr (kPairs) {
            mma<FP8>(s[tile][2 * b], qf[tile][ks], k0, k1);
            mma<FP8>(s[tile][2 * b + 1], qf[tile][ks], k2, k3);
          } else {
            const uint32_t a[4] = {k0, k2, k1, k3};
            mma<FP8>(s[tile][b], a, qf[tile][ks][0], qf[tile][ks][1]);
          }
        }
      };
      if constexpr (FP8) {
#pragma unroll
        for (int kg = 0; kg < D / 32; ++kg) {
#pragma unroll
          for (int b = 0; b < kSub; ++b) {
            uint32_t r[4];
            ldsm4(r, kT + (b * kSpans + (kg >> 2)) * (kSlice * 128) + krow * 128 + (((((kg & 3) * 2) + kc) ^ ksw) << 4));
#pragma unroll
            for (int h = 0; h < 2; ++h) score(b, kg * 2 + h, e4m3x2(r[h]), e4m3x2(r[h] >> 16), e4m3x2(r[2 + h]), e4m3x2(r[2 + h] >> 16));
          }
        }
      } else {
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          uint32_t r[4];
          ldsm4(r, kT + (ks >> 2) * (kSlice * 128) + krow * 128 + (((((ks & 3) * 2) + kc) ^ ksw) << 4));
          score(0, ks, r[0], r[1], r[2], r[3]);
        }
      }
      // ---- online softmax; the running maximum moves when the new one is more than 2^8 above it
      const bool mask = pos0 + kTok > min_limit;
      uint32_t pw[kTiles][kSub][kPairs ? 4 : 2];             // weights, as the second product's operand
#pragma unroll
      for (int tile = 0; tile < kTiles; ++tile) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float mx = -INFINITY;
#pragma unroll
          for (int n = 0; n < kS; ++n)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              float& v = s[tile][n][at(e, j)];
              v *= sc_log2;
              if (mask && pos0 + (kPairs ? n * 8 + 2 * t + j : n * 16 + j * 8 + g) >= lim[tile][e]) v = -INFINITY;
              mx = fmaxf(mx, v);
            }
          mx = over_row(mx, [](float x, float y) { return fmaxf(x, y); });
          if (mx > m_run[tile][e] + 8.f) {                   // also true on a row's first visible token
            const float alpha = ex2(m_run[tile][e] - mx);
            m_run[tile][e] = mx;
            l_run[tile][e] *= alpha;
#pragma unroll
            for (int n = 0; n < kO; ++n) {
              o[tile][n][at(e, 0)] *= alpha;
              o[tile][n][at(e, 1)] *= alpha;
            }
          }
          const float m_use = m_run[tile][e] == -INFINITY ? 0.f : m_run[tile][e];
#pragma unroll
          for (int n = 0; n < kS; ++n)
#pragma unroll
            for (int j = 0; j < 2; ++j) s[tile][n][at(e, j)] = ex2(s[tile][n][at(e, j)] - m_use);
#pragma unroll
          for (int b = 0; b < kSub; ++b) {
            if constexpr (kPairs) {
              const float *v0 = s[tile][2 * b] + 2 * e, *v1 = s[tile][2 * b + 1] + 2 * e;
              l_run[tile][e] += (v0[0] + v0[1]) + (v1[0] + v1[1]);
              pw[tile][b][e] = pack2<FP8>(v0[0], v0[1]);
              pw[tile][b][2 + e] = pack2<FP8>(v1[0], v1[1]);
            } else {
              l_run[tile][e] += s[tile][b][e] + s[tile][b][2 + e];
            }
          }
        }
        if constexpr (!kPairs) {
#pragma unroll
          for (int b = 0; b < kSub; ++b) {
            pw[tile][b][0] = transposed8x8(pack2<FP8>(s[tile][b][0], s[tile][b][1]));
            pw[tile][b][1] = transposed8x8(pack2<FP8>(s[tile][b][2], s[tile][b][3]));
          }
        }
      }
      const int vrow = (lane & 7) + (((lane >> 3) & 1) << 3), vc = lane >> 4;
      // values of 16 tokens at 16 dims: v0, v1 of the first eight dims (of an e4m3 group the even ones), v2, v3 of the others
      auto weigh = [&](int b, int n, uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3) {
#pragma unroll
        for (int tile = 0; tile < kTiles; ++tile) {
          if constexpr (kPairs) {
            mma<FP8>(o[tile][2 * n], pw[tile][b], v0, v1);
            mma<FP8>(o[tile][2 * n + 1], pw[tile][b], v2, v3);
          } else {
            const uint32_t a[4] = {v0, v2, v1, v3};
            mma<FP8>(o[tile][n], a, pw[tile][b][0], pw[tile][b][1]);
          }
        }
      };
      if constexpr (FP8) {
#pragma unroll
        for (int d2 = 0; d2 < D / 32; ++d2) {
#pragma unroll
          for (int b = 0; b < kSub; ++b) {
            uint32_t r[4];
            ldsm4t(r, vT + (b * kSpans + (d2 >> 2)) * (kSlice * 128) + vrow * 128 + (((((d2 & 3) * 2) + vc) ^ ksw) << 4));
#pragma unroll
            for (int h = 0; h < 2; ++h)
              weigh(b, d2 * 2 + h, e4m3x2(__byte_perm(r[2 * h], 0, 0x4420)), e4m3x2(__byte_perm(r[2 * h + 1], 0, 0x4420)),
                    e4m3x2(__byte_perm(r[2 * h], 0, 0x4431)), e4m3x2(__byte_perm(r[2 * h + 1], 0, 0x4431)));
          }
        }
      } else {
#pragma unroll
        for (int n2 = 0; n2 < D / 16; ++n2) {
          uint32_t r[4];
          ldsm4t(r, vT + (n2 >> 2) * (kSlice * 128) + vrow * 128 + (((((n2 & 3) * 2) + vc) ^ ksw) << 4));
          weigh(0, n2, r[0], r[1], r[2], r[3]);
        }
      }
      __syncwarp();                                          // every lane has read the slot
      const int nx = i + slots;
      if (nx < cur.slices) {
        if (nx * kSub % 32 == 0) blocks(cur, nx);
        issue(cur, nx, slot);
      }
      slot = slot + 1 == slots ? 0 : slot + 1;
    }

    // ---- the next unit's first slices travel while this one is merged (slots behind `ahead` hold the merge buffer)
    const int un = u + gridDim.x;
    Unit next;
    started = 0;
    // zeros written behind a context must not be overtaken by the copies that come into the slot next
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (p.over) __syncthreads();                             // no warp writes the merge buffer before all slots are free
    else __syncwarp();
    if (un < units) {
      find(un, next);
      blocks(next, 0);
      for (; started < min(next.slices, p.ahead); ++started) issue(next, started, started);
    }
    if (!p.over) __syncthreads();                            // every warp has its query fragments: the rows may be replaced
    if (un < units) fetch_q(next);
    constexpr int RP = NT * 8;
#pragma unroll
    for (int tile = 0; tile < kTiles; ++tile)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = row_of(tile, e);
        const float l = over_row(l_run[tile][e], [](float x, float y) { return x + y; });
        if (r < R) {
          if ((kPairs ? t : g) == 0) s_ml[warp * RP + r] = make_float2(m_run[tile][e], l);
          float* orow = s_o + (warp * R + r) * D;
#pragma unroll
          for (int n = 0; n < D / 16; ++n) {
            if constexpr (kPairs && FP8) {                   // even dims (2 t, 2 t + 1 of their eight), odd ones: dims 4 t to 4 t + 3
              *reinterpret_cast<float4*>(orow + n * 16 + 4 * t) =
                  make_float4(o[tile][2 * n][2 * e], o[tile][2 * n + 1][2 * e], o[tile][2 * n][2 * e + 1], o[tile][2 * n + 1][2 * e + 1]);
            } else if constexpr (kPairs) {
#pragma unroll
              for (int h = 0; h < 2; ++h)
                *reinterpret_cast<float2*>(orow + n * 16 + h * 8 + 2 * t) = make_float2(o[tile][2 * n + h][2 * e], o[tile][2 * n + h][2 * e + 1]);
            } else if constexpr (FP8) {
              *reinterpret_cast<float2*>(orow + C::place(r, n * 16 + 2 * g)) = make_float2(o[tile][n][e], o[tile][n][2 + e]);
            } else {
              orow[C::place(r, n * 16 + g)] = o[tile][n][e];
              orow[C::place(r, n * 16 + 8 + g)] = o[tile][n][2 + e];
            }
          }
        }
      }
    __syncthreads();
    // final values of four dims of row r: the group's head, the token's row, bf16 or a quantised block (four lanes a block of 16)
    auto store = [&](int r, int c4, float4 a) {
      const int tq = (r * p.g_magic) >> 16, head = cur.kvh * p.G + r - tq * p.G;
      const uint32_t m = cur.qs + tq;
      // 17 rows and more quantise the bf16 value, as the row kernel behind this one did: the same bits as with it. Up to 16 the 32-bit one.
      if (kThroughBf16 && p.outq) {
        auto rounded = [](float x) { return __bfloat162float(__float2bfloat16(x)); };
        a = make_float4(rounded(a.x), rounded(a.y), rounded(a.z), rounded(a.w));
      }
      if (p.outq) {
        float bmax = fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w)));
        bmax = fmaxf(bmax, __shfl_xor_sync(0xffffffffu, bmax, 1));
        bmax = fmaxf(bmax, __shfl_xor_sync(0xffffffffu, bmax, 2));
        const uint8_t sfc = mb::float_to_e4m3(bmax / (6.f * p.outq_gs));
        const float sff = mb::e4m3_to_float(sfc);
        const float qi = sff > 0.f ? (kThroughBf16 ? 1.f / (sff * p.outq_gs) : __fdividef(1.f, sff * p.outq_gs)) : 0.f;
        const uint32_t w = mb::e2m1x2_pack(a.x * qi, a.y * qi) | (mb::e2m1x2_pack(a.z * qi, a.w * qi) << 8);
        const int col = head * D + c4 * 4, kb = col >> 4;
        *reinterpret_cast<uint16_t*>(p.outq + (size_t)m * p.ldq + (col >> 1)) = (uint16_t)w;
        if ((c4 & 3) == 0) p.outq_sf[((size_t)(m >> 7) * p.outq_sf_k64 + (kb >> 2)) * 512 + mb::sf_tile_offset(m & 127, kb & 3)] = sfc;
        return;
      }
      __nv_bfloat162 lo = __floats2bfloat162_rn(a.x, a.y), hi = __floats2bfloat162_rn(a.z, a.w);
      *reinterpret_cast<uint2*>(p.out + (size_t)m * p.out_ld + (size_t)head * D + c4 * 4) =
          make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
    };
    constexpr int kC4 = D / 4;                               // a multiple of 32: whole warps go round together
    for (int idx = tid; idx < R * kC4; idx += 128) {
      const int r = idx / kC4, c4 = idx % kC4;
      float2 ml[4];
      float mx = -INFINITY;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        ml[w] = s_ml[w * RP + r];
        mx = fmaxf(mx, ml[w].x);
      }
      float l = 0.f;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const float f = ml[w].x == -INFINITY ? 0.f : ex2(ml[w].x - mx);
        const float4 ov = *reinterpret_cast<const float4*>(s_o + (w * R + r) * D + C::place(r, c4 * 4));
        l += ml[w].y * f;
        acc.x += ov.x * f; acc.y += ov.y * f; acc.z += ov.z * f; acc.w += ov.w * f;
      }
      if (cur.nparts == 1) {
        const float inv = l > 0.f ? vmul / l : 0.f;
        store(r, c4, make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv));
      } else {                                               // sums as they are, relative to 2^mx
        const int tq = (r * p.g_magic) >> 16;
        const size_t row = ((size_t)(cur.qs + tq) * p.Hq + cur.kvh * p.G + r - tq * p.G) * p.parts + cur.part;
        *reinterpret_cast<float4*>(p.part_o + row * D + c4 * 4) = acc;
        if (c4 == 0) p.part_ml[row] = make_float2(mx, l);
      }
    }
    if (cur.nparts > 1) {
      // the last partition of this (sequence, kv head) to arrive sums all of them in order and re-arms the counter
      __threadfence();
      __syncthreads();
      if (tid == 0) {
        const uint32_t prev = atomicAdd(&p.part_cnt[cur.seq * p.Hkv + cur.kvh], 1u);
        s_last = prev == (uint32_t)cur.nparts - 1;
        if (s_last) p.part_cnt[cur.seq * p.Hkv + cur.kvh] = 0;
      }
      __syncthreads();
      if (s_last) {
        __threadfence();
        for (int idx = tid; idx < R * kC4; idx += 128) {
          const int r = idx / kC4, c4 = idx % kC4, tq = (r * p.g_magic) >> 16;
          const size_t row = ((size_t)(cur.qs + tq) * p.Hq + cur.kvh * p.G + r - tq * p.G) * p.parts;
          const float* po = p.part_o + row * D + c4 * 4;
          float mx = -INFINITY, l = 0.f;
          float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int s0 = 0; s0 < cur.nparts; s0 += 4) {       // four partitions' loads in flight
            float2 ml[4];
            float4 ov[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int sx = min(s0 + k, cur.nparts - 1);
              ml[k] = __ldcg(p.part_ml + row + sx);
              ov[k] = __ldcg(reinterpret_cast<const float4*>(po + (size_t)sx * D));
              if (s0 + k >= cur.nparts) ml[k] = make_float2(-INFINITY, 0.f);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const float mn = fmaxf(mx, ml[k].x);
              const float fa = mx == -INFINITY ? 0.f : ex2(mx - mn), fb = ml[k].x == -INFINITY ? 0.f : ex2(ml[k].x - mn);
              mx = mn;
              l = l * fa + ml[k].y * fb;
              acc.x = acc.x * fa + ov[k].x * fb; acc.y = acc.y * fa + ov[k].y * fb;
              acc.z = acc.z * fa + ov[k].z * fb; acc.w = acc.w * fa + ov[k].w * fb;
            }
          }
          const float inv = l > 0.f ? vmul / l : 0.f;
          store(r, c4, make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv));
        }
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the merge buffer's slots are filled by copies again
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    cur = next;
    u = un;
  }
}

int parts_of(int max_ctx, int part) {
  const int n = (max_ctx + part - 1) / part;
  return n < 1 ? 1 : n > kMaxParts ? kMaxParts : n;
}
// Long partitions pay a unit's fixed instructions less often, short ones fill the chip with fewer sequences. The size depends on the
// cache's heads alone, so that a sequence's sums never depend on its batch; a tensor-parallel shard, which has fewer heads, cuts the
// same sequence finer. Where the line lies, 512 / 1024 tokens, us (e4m3, five heads of 128 a group):
//                                    8 kv heads     4              2              1
//   1 sequence of 4000               12.1 / 14.7    12.0 / 14.4    11.8 / 13.9    10.8 / 14.1
//   16 of 200 to 2000                14.2 / 16.3    11.3 / 15.1    11.6 / 14.0    11.2 / 14.0
//   33 of 100 to 2047                24.5 / 19.7    13.6 / 15.9    11.9 / 14.4    11.4 / 14.4
//   128 of 129 to 1151               57.3 / 45.3    27.3 / 25.3    14.6 / 14.5    12.2 / 12.4
//   9 of 4000 to 16000               70.5 / 49.8    28.9 / 21.4    18.3 / 17.5    17.0 / 16.9
// Nine such batches together, time at 1024 over time at 512: e4m3 0.88, 1.03, 1.08, 1.13; bf16 0.97, 1.07, 1.13, 1.27; eight heads of 256 a
// group e4m3 0.80, 0.88, 1.00, 1.02, bf16 0.81, 0.85, 0.96, 1.03.
int part_tokens_of(const AttnDecodeArgs& a) { return ((a.part_tokens > 0 ? a.part_tokens : a.Hkv >= 8 ? 1024 : 512) + 63) & ~63; }

struct Layout {
  int slots, ahead, over;
  uint32_t merge_off, tail_off, len_off;
  size_t smem;
  int per_sm;                                                // CTAs that an SM holds
};
// Shared memory of a launch. What lies beside the ring grows with the rows (the merge buffer, the queries) and with the batch (the
// list of units), so it may leave room for fewer CTAs than the registers do: the grid has as many as are resident, since the
// units are shared out over it evenly and CTAs beyond would start on theirs when the others are done (with all products in the queries'
// order: e4m3, 40 / 8 heads, 512 sequences of 100 to 1000 tokens 229 -> 172 us, 32 rows 225 -> 219; the former takes 139 now, the split-KV
// kernel 204).
template <int D, bool FP8, int NT>
Layout layout(int rows, int num_seqs, int slots = 2) {
  using C = DecodeCfg<D, FP8, NT>;
  Layout l;
  l.slots = slots;
  // the merge buffer lies over the ring's last slots where it fits in front of the next unit's first ones
  const int merge = 4 * rows * D * 4, behind = (merge + 4 * C::kSlot - 1) / (4 * C::kSlot);
  l.over = behind < slots;
  l.ahead = l.over ? slots - behind : slots;
  l.merge_off = l.over ? (uint32_t)(l.ahead * 4 * C::kSlot) : (uint32_t)C::ring(slots);
  l.tail_off = l.over ? (uint32_t)C::ring(slots) : (uint32_t)(C::ring(slots) + merge);
  l.len_off = (l.tail_off + (uint32_t)(num_seqs + 2) * 4 + 4 * NT * 8 * 8 + 8 + 15) & ~15u;
  l.smem = 1024 + (size_t)l.len_off + (size_t)num_seqs * 16 + (size_t)rows * C::kQPitch;
  const int fit = (int)(228 * 1024 / (l.smem + 1024 + 256));   // a block's own kilobyte, its static arrays
  l.per_sm = fit < 1 ? 1 : fit < C::kCtas ? fit : C::kCtas;
  return l;
}

template <int D, bool FP8, int NT>
int launch(const AttnDecodeArgs& a, DecodeParams& p, cudaStream_t stream) {
  using C = DecodeCfg<D, FP8, NT>;
  auto kern = attn_decode_kernel<D, FP8, NT>;
  CUtensorMap tm[2];
  for (int i = 0; i < 2; ++i) {
    const int rc = mbh::encode_3d(&tm[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, i ? a.v_cache : a.k_cache, C::kRowB, a.Hkv, (uint64_t)a.num_blocks * a.block_size,
                                  C::kRowB, (uint64_t)a.Hkv * C::kRowB, 128, 1, kSlice);
    if (rc) return rc;
  }
  const int rows = a.max_q_len * (a.Hq / a.Hkv), sms = a.sm_count > 0 ? a.sm_count : 148;
  const long long most = (long long)a.num_seqs * a.Hkv * p.parts;
  Layout l = layout<D, FP8, NT>(rows, a.num_seqs);
  // few units: as deep a ring as leaves each of them a CTA of its own. 25 to 32 rows spill registers, which go through what the ring leaves
  // of L1: one e4m3 sequence of 700 tokens at 32 rows 17.4 us with two steps, 17.6 with four, 19.4 with six.
  for (int slots = NT > 3 ? 4 : kMaxSlots; slots > 2; --slots) {
    const Layout deep = layout<D, FP8, NT>(rows, a.num_seqs, slots);
    if (deep.smem <= 220 * 1024 && (long long)sms * deep.per_sm >= most) {
      l = deep;
      break;
    }
  }
  p.slots = l.slots;
  p.ahead = l.ahead;
  p.over = l.over;
  p.merge_off = l.merge_off;
  p.tail_off = l.tail_off;
  p.len_off = l.len_off;
  static size_t configured = 0;
  if (l.smem > 220 * 1024) return MB_ERR_TOO_LARGE;
  if (l.smem > configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    if (e != cudaSuccess) return (int)e;
    configured = 220 * 1024;
  }
  const int grid = most < (long long)sms * l.per_sm ? (int)most : sms * l.per_sm;
  p.early = a.early && mb_pdl_enabled() == 2;
  return (int)mb::launch_kernel_ex(kern, dim3(grid), dim3(128), l.smem, stream, 1, p.early || mb_pdl_enabled() == 1, tm[0], tm[1], p);
}

}  // namespace

namespace {

// f(D, FP8, NT) as types, for rows of either kind
template <typename F>
auto by_shape(int D, bool fp8, int rows, F&& f) {
  auto tiles = [&](auto d, auto eight) {
    using std::integral_constant;
    if constexpr (d.value == 256) {
      return rows <= 8 ? f(d, eight, integral_constant<int, 1>{}) : f(d, eight, integral_constant<int, 2>{});
    } else {
      return rows <= 8    ? f(d, eight, integral_constant<int, 1>{})
             : rows <= 16 ? f(d, eight, integral_constant<int, 2>{})
             : rows <= 24 ? f(d, eight, integral_constant<int, 3>{})
                          : f(d, eight, integral_constant<int, 4>{});
    }
  };
  if (D == 256) return fp8 ? tiles(std::integral_constant<int, 256>{}, std::true_type{}) : tiles(std::integral_constant<int, 256>{}, std::false_type{});
  return fp8 ? tiles(std::integral_constant<int, 128>{}, std::true_type{}) : tiles(std::integral_constant<int, 128>{}, std::false_type{});
}

}  // namespace

extern "C" int mb_attn_decode_per_sm(int D, int fp8, int rows, int num_seqs, size_t* smem) {
  const Layout l = by_shape(D, fp8 != 0, rows, [&](auto d, auto eight, auto nt) { return layout<d.value, eight.value, nt.value>(rows, num_seqs); });
  if (smem) *smem = l.smem;
  return l.per_sm;
}

bool mb_attn_decode_serves(const AttnDecodeArgs& a) {
  const int G = a.Hq / a.Hkv, rows = G * a.max_q_len;
  const uintptr_t al = reinterpret_cast<uintptr_t>(a.k_cache) | reinterpret_cast<uintptr_t>(a.v_cache);
  return (a.D == 128 || a.D == 256) && rows <= (a.D == 256 ? 16 : 32) && a.num_seqs <= kMaxSeqs && a.block_size % kSlice == 0 && !(al & 15) &&
         !(reinterpret_cast<uintptr_t>(a.q) & 15) && a.num_blocks * a.block_size < (1ll << 31) &&
         (a.outq || (a.out_ld % 4 == 0 && !(reinterpret_cast<uintptr_t>(a.out) & 7)));
}

size_t mb_attn_decode_ws(const AttnDecodeArgs& a) {
  const int parts = parts_of(a.max_ctx, part_tokens_of(a));
  return parts <= 1 ? 0 : kCntBytes + (size_t)a.total_rows * a.Hq * parts * (a.D + 2) * sizeof(float);
}

int mb_attn_decode(const AttnDecodeArgs& a, cudaStream_t stream) {
  DecodeParams p{};
  p.q = a.q; p.block_table = a.block_table; p.max_blocks = a.max_blocks;
  p.q_start = a.q_start; p.q_len = a.q_len; p.ctx_len = a.ctx_len;
  p.num_seqs = a.num_seqs; p.Hq = a.Hq; p.Hkv = a.Hkv; p.G = a.Hq / a.Hkv; p.g_magic = (65536 + p.G - 1) / p.G;
  p.block_size = a.block_size;
  p.block_shift = (a.block_size & (a.block_size - 1)) == 0 ? 31 - __builtin_clz(a.block_size) : -1;
  p.num_blocks = a.num_blocks; p.scale = a.scale; p.k_scale = a.k_scale; p.v_scale = a.v_scale;
  p.out = a.out; p.out_ld = a.out_ld;
  p.outq = a.outq; p.ldq = a.ldq; p.outq_sf = a.outq_sf; p.outq_sf_k64 = a.outq_sf_k64; p.outq_gs = a.outq_gs;
  p.status = a.status;
  p.part_tokens = part_tokens_of(a);
  p.parts = parts_of(a.max_ctx, p.part_tokens);
  if (p.parts > 1) {
    if (!a.ws || a.ws_bytes < mb_attn_decode_ws(a) || (size_t)a.num_seqs * a.Hkv * 4 > kCntBytes) return MB_ERR_TOO_LARGE;
    p.part_cnt = reinterpret_cast<uint32_t*>(a.ws);
    p.part_o = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(a.ws) + kCntBytes);
    p.part_ml = reinterpret_cast<float2*>(p.part_o + (size_t)a.total_rows * a.Hq * p.parts * a.D);
  }
  return by_shape(a.D, a.fp8 != 0, a.max_q_len * p.G, [&](auto d, auto eight, auto nt) { return launch<d.value, eight.value, nt.value>(a, p, stream); });
}
