// A dense NVFP4 decoder layer (RMSNorm, q|k|v, rotation and cache write, attention, output projection, RMSNorm, gate|up with SwiGLU,
// down) as one call: host code that issues the launches which models/decoder.py's blocks issue one by one, with the same arguments.
//
// For prompts, which run outside a graph: filling a launcher's arguments and allocating its outputs in Python takes about as long
// as 10 us of kernels, and a layer has eight launches. A layer of a 40-token prompt cost 150 us of host time against 70 us of
// kernels.
#include <cuda_bf16.h>
#include "epilogue.cuh"
#include "gemm_args.h"
#include "noalloc.h"
#include "op_args.h"

namespace {

constexpr int kHead = 128;
enum { IN_COPY = 0, IN_RMSNORM = 1, OUT_NVFP4 = 3, KIND_NVFP4 = 2 };

}  // namespace

#define MB_DENSE_LAYER_GROW (-100)         // nothing was launched: the attention workspace is too small

struct MbDenseLinear {
  const void* W;
  const void* sf;            // tiled scale factors
  const float* row_scale;    // per output feature, or null
  float alpha;
};

struct MbDenseLayerArgs {
  int T, num_seqs, max_q_len, max_ctx;
  int hidden, heads, kv_heads, inter;      // every input length a multiple of 256
  int rot, max_pos, plus_one, block_size, cache_fp8, max_blocks;
  int sm_count, gemm_flags, attn_tc, attn_tc_vmn, part_tokens, part_fixed, gather_wide;
  long long num_blocks, gather_rows;
  float eps, scale, o_static, down_static;
  MbDenseLinear qkv, o, gate_up, down;
  const void* x;             // bf16 [T, hidden], or with `gather` the table whose rows they are
  const void* gather;
  void* out;                 // bf16 [T, hidden]
  const void *ln1, *ln2, *q_norm, *k_norm;
  const float *cos_tab, *sin_tab;
  const int* positions;
  const long long* slots;
  void *k_cache, *v_cache;
  const float *k_scale, *v_scale;
  const int *block_table, *q_start, *q_len, *ctx_len;
  void* scratch;
  size_t scratch_bytes;
  void* ws;
  size_t ws_bytes;
  void* attn_ws;
  size_t attn_ws_bytes;
  uint32_t* status;
  // results
  int launches;
  size_t attn_ws_need;       // with MB_DENSE_LAYER_GROW: what the attention workspace has to hold
};

namespace {

// The layer's intermediate tensors in one block of memory. What is read up to the attention's output lies under what comes behind it.
struct Places {
  size_t rows, x1;                         // the residual stream in front (gathered) and between the two halves
  size_t a1, a1_scale, a1_sf, qkv, q, o16, oq, oq_scale, oq_sf;
  size_t a2, a2_scale, a2_sf, h16, hq, hq_scale, hq_sf;
  size_t total;
};

size_t sf_bytes(const MbDenseLayerArgs& a, int K) { return (size_t)((a.T + 127) / 128) * (K / 64) * 512; }

// whether the attention kernel that takes the call leaves its output quantised
bool attention_quantises(const MbDenseLayerArgs& a) {
  if (a.attn_tc && a.max_q_len >= 128) return a.scale > 0.f && a.attn_tc_vmn;
  const bool plain = a.block_size % 16 == 0 && a.num_seqs <= 1024;             // attention_decode.cu
  return a.heads / a.kv_heads * a.max_q_len <= (plain ? 32 : 16);
}
// ... and the gate|up GEMM its SwiGLU result: few tokens and more tiles than SMs, or more than 128 tokens
bool swiglu_quantises(const MbDenseLayerArgs& a) {
  return a.T <= 128 ? (2 * a.inter + 127) / 128 > a.sm_count : (a.gemm_flags & MB_GEMM_PERSISTENT_PREFILL) != 0;
}

Places places(const MbDenseLayerArgs& a) {
  Places p{};
  size_t at = 0;
  auto take = [&](size_t n) {
    const size_t here = at;
    at += (n + 1023) & ~(size_t)1023;      // operands of TMA boxes
    return here;
  };
  const size_t T = a.T, H = a.hidden, Q = (size_t)a.heads * kHead, KV = (size_t)a.kv_heads * kHead, I = a.inter;
  p.rows = take(a.gather ? T * H * 2 : 0);
  p.x1 = take(T * H * 2);
  const size_t base = at;
  p.a1 = take(T * H / 2); p.a1_scale = take(T * 4); p.a1_sf = take(sf_bytes(a, a.hidden));
  p.qkv = take(T * (Q + 2 * KV) * 2);
  p.q = take(T * Q * 2);
  p.o16 = take(attention_quantises(a) ? 0 : T * Q * 2);
  p.oq = take(T * Q / 2); p.oq_scale = take(T * 4); p.oq_sf = take(sf_bytes(a, (int)Q));
  const size_t first = at;
  at = base;
  p.a2 = take(T * H / 2); p.a2_scale = take(T * 4); p.a2_sf = take(sf_bytes(a, a.hidden));
  p.h16 = take(swiglu_quantises(a) ? 0 : T * I * 2);
  p.hq = take(T * I / 2); p.hq_scale = take(T * 4); p.hq_sf = take(sf_bytes(a, a.inter));
  p.total = first > at ? first : at;
  return p;
}

bool takes(const MbDenseLayerArgs& a) {
  return a.T > 0 && a.num_seqs > 0 && a.hidden > 0 && a.heads > 0 && a.kv_heads > 0 && a.inter > 0 && a.heads % a.kv_heads == 0 && a.hidden % 256 == 0 &&
         a.heads * kHead % 256 == 0 && a.inter % 256 == 0 && a.o_static > 0.f && a.down_static > 0.f;
}

// an NVFP4 activation [T, K]
struct Quantised {
  void* data;
  float* scale;              // per token, or null: `fixed`
  void* sf;
  int K;
  float fixed;
};

}  // namespace

// scratch_bytes of this call
extern "C" int mb_dense_layer_scratch(MbDenseLayerArgs* a) {
  if (!takes(*a)) return MB_ERR_BAD_ARG;
  a->scratch_bytes = places(*a).total;
  return 0;
}

extern "C" int mb_dense_layer(MbDenseLayerArgs* args, cudaStream_t stream) {
  MbDenseLayerArgs& a = *args;
  if (!takes(a) || !a.scratch) return MB_ERR_BAD_ARG;
  const Places pl = places(a);
  if (a.scratch_bytes < pl.total) return MB_ERR_BAD_ARG;
  const int T = a.T, H = a.hidden, Q = a.heads * kHead, KV = a.kv_heads * kHead, I = a.inter, N = Q + 2 * KV;
  a.launches = 0;
  uint8_t* s = static_cast<uint8_t*>(a.scratch);
  auto f32 = [&](size_t at) { return reinterpret_cast<float*>(s + at); };

  // attention first: the one call that may ask for more workspace
  const bool prefill = a.attn_tc && a.max_q_len >= 128, attn_fused = attention_quantises(a);
  MbAttnArgs at{};
  at.q = s + pl.q; at.k_cache = a.k_cache; at.v_cache = a.v_cache;
  at.block_table = a.block_table; at.max_blocks = a.max_blocks;
  at.q_start = a.q_start; at.q_len = a.q_len; at.ctx_len = a.ctx_len;
  at.num_seqs = a.num_seqs; at.max_q_len = a.max_q_len; at.max_ctx = a.max_ctx;
  at.Hq = a.heads; at.Hkv = a.kv_heads; at.D = kHead; at.block_size = a.block_size; at.num_blocks = a.num_blocks;
  at.scale = a.scale; at.cache_fp8 = a.cache_fp8; at.k_scale = a.k_scale; at.v_scale = a.v_scale;
  at.out = attn_fused ? s + pl.oq : s + pl.o16;
  at.total_rows = T; at.part_tokens = a.part_tokens; at.part_fixed = a.part_fixed; at.sm_count = a.sm_count; at.status = a.status; at.early = 1;
  if (!prefill) {
    a.attn_ws_need = mb_attn_ws_need(&at);
    if (a.attn_ws_need > a.attn_ws_bytes) return MB_DENSE_LAYER_GROW;
    at.ws = a.attn_ws; at.ws_bytes = a.attn_ws_bytes;
  }

  int rc;
  auto row = [&](int mode, const void* x, int K, const void* w, float fixed, const Quantised& to, const void* gather, void* rows) {
    MbRowArgs r{};
    r.M = T; r.K = K; r.in_mode = mode; r.out_mode = OUT_NVFP4;
    r.x = x; r.x_ld = K; r.w = w; r.w_plus_one = a.plus_one; r.eps = a.eps;
    r.out = to.data; r.out_ld = K / 2; r.scale = to.scale; r.sf = to.sf; r.sf_k64 = K / 64; r.static_gs = fixed;
    if (gather) {
      r.gather = gather; r.gather_wide = a.gather_wide; r.gather_rows = a.gather_rows; r.gather_out = rows; r.status = a.status;
    }
    ++a.launches;
    return mb_row_op(&r, stream);
  };
  auto gemm = [&](const MbDenseLinear& w, int n, const Quantised& x, void* out, const void* residual, bool swiglu, const Quantised* to) {
    MbGemmArgs g{};
    g.kind = KIND_NVFP4; g.M = T; g.N = n; g.K = x.K; g.ldo = swiglu ? n / 2 : n;
    g.W = w.W; g.X = x.data; g.out = out; g.residual = residual;
    g.w_scale = w.row_scale; g.a_scale = x.scale; g.a_static = x.scale ? 0.f : x.fixed; g.alpha = w.alpha;
    g.sfa = w.sf; g.sfb = x.sf; g.sf_k64 = x.K / 64;
    g.epilogue = swiglu ? (int)mb::EPI_SWIGLU : (int)mb::EPI_PLAIN;
    g.ws = a.ws; g.ws_bytes = a.ws_bytes; g.status = a.status; g.sm_count = a.sm_count; g.flags = a.gemm_flags;
    if (to) {
      g.out = to->data; g.outq = to->data; g.ldq = to->K / 2; g.outq_sf = to->sf; g.outq_sf_k64 = to->K / 64; g.outq_gs = to->fixed;
    }
    ++a.launches;
    return mb_gemm(&g, stream);
  };

  const Quantised a1{s + pl.a1, f32(pl.a1_scale), s + pl.a1_sf, H, 0.f}, a2{s + pl.a2, f32(pl.a2_scale), s + pl.a2_sf, H, 0.f};
  const void* x = a.gather ? s + pl.rows : a.x;
  if ((rc = row(IN_RMSNORM, a.x, H, a.ln1, 0.f, a1, a.gather, s + pl.rows))) return rc;
  if ((rc = gemm(a.qkv, N, a1, s + pl.qkv, nullptr, false, nullptr))) return rc;
  MbRopeKvArgs rk{};
  rk.M = T; rk.Hq = a.heads; rk.Hkv = a.kv_heads; rk.D = kHead; rk.rot = a.rot;
  rk.qkv = s + pl.qkv; rk.qkv_ld = N; rk.q_head_stride = kHead; rk.k_off = Q; rk.v_off = Q + KV;
  rk.positions = a.positions; rk.slots = a.slots; rk.q_norm_w = a.q_norm; rk.k_norm_w = a.k_norm; rk.norm_plus_one = a.plus_one; rk.eps = a.eps;
  rk.cos_tab = a.cos_tab; rk.sin_tab = a.sin_tab; rk.max_pos = a.max_pos;
  rk.q_out = s + pl.q; rk.k_cache = a.k_cache; rk.v_cache = a.v_cache; rk.cache_fp8 = a.cache_fp8; rk.k_scale = a.k_scale; rk.v_scale = a.v_scale;
  rk.num_slots = a.num_blocks * a.block_size; rk.status = a.status; rk.early = 1;
  ++a.launches;
  if ((rc = mb_qk_norm_rope_kvwrite(&rk, stream))) return rc;

  const Quantised oq{s + pl.oq, attn_fused ? nullptr : f32(pl.oq_scale), s + pl.oq_sf, Q, a.o_static};
  ++a.launches;
  if (prefill) {
    MbAttnTcArgs t{};
    t.q = at.q; t.k_cache = a.k_cache; t.v_cache = a.v_cache; t.block_table = a.block_table;
    t.q_start = a.q_start; t.q_len = a.q_len; t.ctx_len = a.ctx_len; t.k_scale = a.k_scale; t.v_scale = a.v_scale;
    t.out = attn_fused ? nullptr : s + pl.o16; t.status = a.status; t.num_blocks = a.num_blocks; t.max_blocks = a.max_blocks; t.num_seqs = a.num_seqs;
    t.max_q_len = a.max_q_len; t.Hq = a.heads; t.Hkv = a.kv_heads; t.D = kHead; t.block_size = a.block_size; t.cache_fp8 = a.cache_fp8;
    t.scale = a.scale; t.v_mn = a.attn_tc_vmn;
    if (attn_fused) {
      t.outq = oq.data; t.ldq = Q / 2; t.outq_sf = oq.sf; t.outq_sf_k64 = Q / 64; t.outq_gs = a.o_static;
    }
    if ((rc = mb_attn_prefill_tc(&t, stream))) return rc;
  } else {
    if (attn_fused) {
      at.outq = oq.data; at.ldq = Q / 2; at.outq_sf = oq.sf; at.outq_sf_k64 = Q / 64; at.outq_gs = a.o_static;
    }
    if ((rc = mb_paged_attention(&at, stream))) return rc;
  }
  if (!attn_fused && (rc = row(IN_COPY, s + pl.o16, Q, nullptr, a.o_static, oq, nullptr, nullptr))) return rc;
  if ((rc = gemm(a.o, H, oq, s + pl.x1, x, false, nullptr))) return rc;

  if ((rc = row(IN_RMSNORM, s + pl.x1, H, a.ln2, 0.f, a2, nullptr, nullptr))) return rc;
  const bool ffn_fused = swiglu_quantises(a);
  const Quantised hq{s + pl.hq, ffn_fused ? nullptr : f32(pl.hq_scale), s + pl.hq_sf, I, a.down_static};
  if ((rc = gemm(a.gate_up, 2 * I, a2, s + pl.h16, nullptr, true, ffn_fused ? &hq : nullptr))) return rc;
  if (!ffn_fused && (rc = row(IN_COPY, s + pl.h16, I, nullptr, a.down_static, hq, nullptr, nullptr))) return rc;
  return gemm(a.down, H, hq, a.out, s + pl.x1, false, nullptr);
}
