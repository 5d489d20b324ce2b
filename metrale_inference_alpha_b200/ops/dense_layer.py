"""A dense NVFP4 decoder layer as one native call (csrc/dense_layer.cu): the launches of ``models.decoder.Decoder.layer`` without
the host time of issuing them one by one."""
from __future__ import annotations

import ctypes as C

import torch

from . import _native, _count, _ptr, _stream, runtime
from ._native import c_float, c_int, c_ll, c_size_t, c_void_p

_GROW = -100                               # MB_DENSE_LAYER_GROW


class DenseLinear(C.Structure):
    _fields_ = [("W", c_void_p), ("sf", c_void_p), ("row_scale", c_void_p), ("alpha", c_float)]


class DenseLayerArgs(C.Structure):
    _fields_ = [
        ("T", c_int), ("num_seqs", c_int), ("max_q_len", c_int), ("max_ctx", c_int),
        ("hidden", c_int), ("heads", c_int), ("kv_heads", c_int), ("inter", c_int),
        ("rot", c_int), ("max_pos", c_int), ("plus_one", c_int), ("block_size", c_int), ("cache_fp8", c_int), ("max_blocks", c_int),
        ("sm_count", c_int), ("gemm_flags", c_int), ("attn_tc", c_int), ("attn_tc_vmn", c_int), ("part_tokens", c_int), ("part_fixed", c_int),
        ("gather_wide", c_int), ("num_blocks", c_ll), ("gather_rows", c_ll),
        ("eps", c_float), ("scale", c_float), ("o_static", c_float), ("down_static", c_float),
        ("qkv", DenseLinear), ("o", DenseLinear), ("gate_up", DenseLinear), ("down", DenseLinear),
        ("x", c_void_p), ("gather", c_void_p), ("out", c_void_p),
        ("ln1", c_void_p), ("ln2", c_void_p), ("q_norm", c_void_p), ("k_norm", c_void_p), ("cos_tab", c_void_p), ("sin_tab", c_void_p),
        ("positions", c_void_p), ("slots", c_void_p), ("k_cache", c_void_p), ("v_cache", c_void_p), ("k_scale", c_void_p), ("v_scale", c_void_p),
        ("block_table", c_void_p), ("q_start", c_void_p), ("q_len", c_void_p), ("ctx_len", c_void_p),
        ("scratch", c_void_p), ("scratch_bytes", c_size_t), ("ws", c_void_p), ("ws_bytes", c_size_t), ("attn_ws", c_void_p), ("attn_ws_bytes", c_size_t),
        ("status", c_void_p), ("launches", c_int), ("attn_ws_need", c_size_t),
    ]


_native.register_optional("mb_dense_layer", [C.POINTER(DenseLayerArgs), c_void_p])
_native.register_optional("mb_dense_layer_scratch", [C.POINTER(DenseLayerArgs)])


def observed() -> bool:
    """Somebody counts or times single launches: they are issued one by one then."""
    return _native._trace is not None or _native._launch_hook is not None or _native._audit is not None


def serves_weights(lw, hidden: int, head_dim: int) -> bool:
    """The layer's weights are of the form that the native call takes."""
    w, f = lw.mixer, lw.ffn
    return (all(m.fmt == "nvfp4" and m.K % 256 == 0 and m.sf_tiled is not None for m in (w.qkv, w.o, f.gate_up, f.down)) and head_dim == 128
            and w.qkv.K == f.gate_up.K == w.o.N == f.down.N == hidden and w.o.K == w.heads * head_dim
            and w.qkv.N == (w.heads + 2 * w.kv_heads) * head_dim and f.gate_up.N == 2 * f.down.K
            and w.qkv_bias is None and f.interleaved and f.clamp_glu is None
            and torch.is_tensor(lw.ln1) and torch.is_tensor(lw.ln2) and lw.post_attn is None and lw.post_ffn is None and lw.out is None and lw.side is None)


def _linear(to: DenseLinear, w) -> None:
    to.W, to.sf, to.row_scale, to.alpha = _ptr(w.data), _ptr(w.sf_tiled), _ptr(w.row_gscale), w.gscale


def dense_layer(x: torch.Tensor, lw, batch, kc, vc, ks, vs, *, cos, sin, scale: float, eps: float, plus_one: bool, gather=None) -> torch.Tensor:
    """bf16 [T, hidden] -> bf16 [T, hidden]. `gather`: the layer's input is those rows of `x`."""
    from . import _ATTN_PART_TOKENS, _ATTN_TC, _ATTN_TC_VMN, _GROUPED_CTAS, _PART_LEVER, _PERSIST_PREFILL
    w, f = lw.mixer, lw.ffn
    dev, hidden = x.device, x.shape[1]
    rt = runtime(dev)
    L = _native.lib()
    a = DenseLayerArgs()
    T = a.T = x.shape[0] if gather is None else gather.numel()
    assert x.dtype == torch.bfloat16 and x.is_contiguous()
    a.num_seqs, a.max_q_len, a.max_ctx = batch.q_len.numel(), batch.max_q_len, batch.max_ctx
    a.hidden, a.heads, a.kv_heads, a.inter = hidden, w.heads, w.kv_heads, f.down.K
    if cos is not None:
        a.max_pos, half = cos.shape
        a.rot = 2 * half
    a.plus_one, a.eps, a.scale, a.o_static, a.down_static = plus_one, eps, scale, w.o_in_scale, f.down_in_scale
    a.num_blocks, a.block_size = kc.shape[0], kc.shape[1]
    a.cache_fp8, a.max_blocks = kc.dtype == torch.uint8, batch.block_table.stride(0)
    a.sm_count, a.gemm_flags = rt.sm_count, _PERSIST_PREFILL | _GROUPED_CTAS
    a.attn_tc, a.attn_tc_vmn, a.part_fixed, a.part_tokens = _ATTN_TC, _ATTN_TC_VMN, _PART_LEVER, _ATTN_PART_TOKENS
    _linear(a.qkv, w.qkv)
    _linear(a.o, w.o)
    _linear(a.gate_up, f.gate_up)
    _linear(a.down, f.down)
    a.x = _ptr(x)
    if gather is not None:
        assert gather.dtype in (torch.int32, torch.int64) and gather.is_contiguous()
        a.gather, a.gather_wide, a.gather_rows = _ptr(gather), gather.dtype == torch.int64, x.shape[0]
    out = torch.empty(T, hidden, dtype=torch.bfloat16, device=dev)
    a.out, a.ln1, a.ln2, a.q_norm, a.k_norm = _ptr(out), _ptr(lw.ln1), _ptr(lw.ln2), _ptr(w.q_norm), _ptr(w.k_norm)
    a.cos_tab, a.sin_tab = _ptr(cos), _ptr(sin)
    a.positions, a.slots, a.k_cache, a.v_cache = _ptr(batch.positions), _ptr(batch.slot_mapping), _ptr(kc), _ptr(vc)
    a.k_scale, a.v_scale = _ptr(ks), _ptr(vs)
    a.block_table, a.q_start, a.q_len, a.ctx_len = _ptr(batch.block_table), _ptr(batch.q_start), _ptr(batch.q_len), _ptr(batch.ctx_len)
    _native.check(L.mb_dense_layer_scratch(C.byref(a)), "dense_layer_scratch")
    scratch = torch.empty(a.scratch_bytes, dtype=torch.uint8, device=dev)
    a.scratch = _ptr(scratch)
    a.ws, a.ws_bytes, a.status = _ptr(rt.ws), rt.ws_bytes, _ptr(rt.status)
    a.attn_ws, a.attn_ws_bytes = _ptr(rt.attn_ws), rt.attn_ws.numel()
    rc = L.mb_dense_layer(C.byref(a), _stream())
    if rc == _GROW:
        rt.ensure_attn_ws(a.attn_ws_need)
        a.attn_ws, a.attn_ws_bytes = _ptr(rt.attn_ws), rt.attn_ws.numel()
        rc = L.mb_dense_layer(C.byref(a), _stream())
    if rc != 0:
        _native.check(rc, f"dense_layer[T={T}]")
    _count(a.launches)
    return out
