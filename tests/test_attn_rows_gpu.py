"""Prefill attention on two row tiles per CTA (csrc/attention_rows.cu) at the edges of its tiles, against attention in 64 bits."""
import math

import pytest
import torch

from metrale_inference_alpha_b200 import ops
from metrale_inference_alpha_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _case(fp8, Hq, Hkv, q_lens, ctx_lens, bs, seed=0):
    """Caches whose unwritten tokens are NaN: a row that saw one would show it."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    D, S = 128, len(q_lens)
    need = [(c + bs - 1) // bs for c in ctx_lens]
    perm = (torch.randperm(sum(need), generator=g, device=DEV) + 1).to(torch.int32)
    bt = torch.full((S, max(need) + 1), sum(need) + 50, dtype=torch.int32, device=DEV)       # entries behind a sequence name no block
    kv = []
    for std in (1.0, 1.4):
        x = torch.full((sum(need) + 1, bs, Hkv, D), float("nan"), device=DEV)
        at = 0
        for s, (n, c) in enumerate(zip(need, ctx_lens)):
            bt[s, :n] = perm[at:at + n]
            rows = torch.full((n * bs, Hkv, D), float("nan"), device=DEV)
            rows[:c] = torch.randn(c, Hkv, D, generator=g, device=DEV) * std
            x[perm[at:at + n].long()] = rows.view(n, bs, Hkv, D)
            at += n
        kv.append(x.to(torch.float8_e4m3fn) if fp8 else x.bfloat16())
    q = torch.randn(sum(q_lens), Hq, D, generator=g, device=DEV).bfloat16()
    scales = (torch.tensor([0.8], device=DEV), torch.tensor([1.3], device=DEV)) if fp8 else (None, None)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    q_len = i32(q_lens)
    args = (q, *(t.view(torch.uint8) if fp8 else t for t in kv), bt, torch.cumsum(q_len, 0, dtype=torch.int32) - q_len, q_len, i32(ctx_lens))
    kw = dict(max_q_len=max(q_lens), max_ctx=max(ctx_lens), scale=D ** -0.5, k_scale=scales[0], v_scale=scales[1])
    out, at = torch.empty(sum(q_lens), Hq, D, dtype=torch.float64, device=DEV), 0
    for s, (n, c) in enumerate(zip(q_lens, ctx_lens)):
        k, v = (t[bt[s, :need[s]].long()].reshape(-1, Hkv, D)[:c].double() * (1.0 if sc is None else sc.double())
                for t, sc in zip(kv, scales))
        mask = torch.arange(c, device=DEV)[None] <= torch.arange(c - n, c, device=DEV)[:, None]
        for h in range(Hq):
            w = torch.softmax((q[at:at + n, h].double() @ k[:, h // (Hq // Hkv)].t() * D ** -0.5).masked_fill(~mask, -math.inf), -1)
            out[at:at + n, h] = w @ v[:, h // (Hq // Hkv)]
        at += n
    return args, kw, out


# one row tile short of, at and past 128 and 256 rows; contexts around a tile of 128 tokens; one and many heads a group; blocks that
# are no power of two; a short sequence beside long ones; enough tiles for both stages to come round several times
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("Hq,Hkv,q_lens,ctx_lens,bs", [
    (1, 1, [128], [128], 16), (1, 1, [255], [255], 16), (2, 1, [129, 1], [129, 700], 16), (5, 1, [128, 127], [1000, 127], 16),
    (40, 8, [333], [333], 16), (8, 1, [130], [256], 32), (3, 1, [257], [257], 24), (16, 2, [128, 200, 5], [385, 200, 5], 64),
    (4, 2, [1500], [1500], 16), (2, 2, [131], [1900], 16)])
def test_matches_attention_in_64_bits(fp8, Hq, Hkv, q_lens, ctx_lens, bs):
    args, kw, want = _case(fp8, Hq, Hkv, q_lens, ctx_lens, bs)
    got = ops.paged_attention(*args, **kw)
    ops.check_status(DEV)
    # the result's bf16 rounding (2^-9 of each value at most) and the weights' (2^-9 in bf16, 2^-12 in f16, independent per token)
    assert (got.double() - want).norm() <= 2.0 ** -8 * want.norm()
    assert (got.double() - want).abs().max() <= 2.0 ** -6 * want.abs().max()


def test_scores_that_grow_along_the_context_rescale_the_output():
    """Keys that point ever more along the queries: the running maximum moves by more than 2^8 again and again."""
    args, kw, _ = _case(False, 2, 1, [256], [1024], 16)
    q, kc, vc, bt, qs, ql, ctx = args
    k = torch.zeros(1024, 1, 128, device=DEV)
    k[:, :, 0] = torch.linspace(-60, 90, 1024, device=DEV)[:, None]
    kc[bt[0, :64].long()] = k.bfloat16().view(64, 16, 1, 128)
    q.zero_()
    q[:, :, 0] = 12.0
    got = ops.paged_attention(*args, **kw).double()
    ops.check_status(DEV)
    kk, vv = (t[bt[0, :64].long()].reshape(-1, 128).double() for t in (kc, vc))
    mask = torch.arange(1024, device=DEV)[None] <= torch.arange(768, 1024, device=DEV)[:, None]
    want = torch.softmax((q[:, 0].double() @ kk.t() * 128 ** -0.5).masked_fill(~mask, -math.inf), -1) @ vv
    assert (got[:, 0] - want).norm() <= 2.0 ** -8 * want.norm()


@pytest.mark.parametrize("power", [20, 120, -30, -100])
def test_queries_keep_the_range_of_bf16(power):
    """An e4m3 cache is read as f16; queries far outside its range give the same bits with a softmax scale that takes the power back."""
    args, kw, _ = _case(True, 10, 2, [129, 200], [129, 900], 16)
    want = ops.paged_attention(*args, **kw)
    got = ops.paged_attention(args[0] * 2.0 ** power, *args[1:], **dict(kw, scale=kw["scale"] * 2.0 ** -power))
    ops.check_status(DEV)
    assert got.isfinite().all() and torch.equal(got, want)


def test_a_large_query_leaves_its_row_finite():
    """One element of a row beyond f16, on a dim where the keys are zero: the row's other dims decide, as for its neighbours."""
    args, kw, _ = _case(True, 2, 1, [140], [140], 16)
    q, kc = args[0], args[1]
    kc[..., 7] = 0
    want = ops.paged_attention(*args, **kw).double()
    q[3:90, :, 7] = 1e6
    got = ops.paged_attention(*args, **kw).double()
    ops.check_status(DEV)
    # elements above 2^-31 of 1e6 keep their bits, smaller ones are off by 2^-20 at most: far less than the weights' and the result's rounding
    assert (got - want).norm() <= 2.0 ** -8 * want.norm()


def test_small_weights_beside_a_large_one_reach_the_output():
    """The first token takes the row's maximum and has no value; some four thousand others of 2^-26 of its weight make the output."""
    args, kw, _ = _case(True, 1, 1, [128], [4096], 16)
    q, kc, vc, bt, qs, ql, ctx = args
    g = torch.Generator(device=DEV).manual_seed(3)
    k = torch.randn(4096, 128, generator=g, device=DEV) * 0.25
    k[:, 0] = 0
    k[0] = 0
    k[0, 0] = 16.0
    v = torch.rand(4096, 128, generator=g, device=DEV) + 0.5
    v[0] = 0
    for cache, x in ((kc, k), (vc, v)):
        cache[bt[0, :256].long()] = x.to(torch.float8_e4m3fn).view(torch.uint8).view(256, 16, 1, 128)
    q.copy_(torch.randn(128, 1, 128, generator=g, device=DEV) * 0.25)
    q[:, :, 0] = 25.75 * math.log(2) * 128 ** 0.5 / (16 * 0.8)      # k_scale is 0.8
    got = ops.paged_attention(*args, **kw)[:, 0].double()
    ops.check_status(DEV)
    kk, vv = (t[bt[0, :256].long()].view(torch.float8_e4m3fn).reshape(-1, 128).double() * s.double() for t, s in ((kc, kw["k_scale"]), (vc, kw["v_scale"])))
    mask = torch.arange(4096, device=DEV)[None] <= torch.arange(3968, 4096, device=DEV)[:, None]
    want = torch.softmax((q[:, 0].double() @ kk.t() * 128 ** -0.5).masked_fill(~mask, -math.inf), -1) @ vv
    # the result's bf16 rounding; the weights' steps of 2^-31 of the maximum average out over the tokens
    assert (got - want).norm() <= 2.0 ** -8 * want.norm()


@pytest.mark.parametrize("Hq,Hkv,q_lens,ctx_lens", [(40, 8, [129], [129]), (4, 2, [140, 300], [500, 300])])
def test_quantised_output(Hq, Hkv, q_lens, ctx_lens):
    args, kw, want = _case(True, Hq, Hkv, q_lens, ctx_lens, 16)
    plain = ops.paged_attention(*args, **kw)
    T, K, gs = sum(q_lens), Hq * 128, 2 * 6.0 / 2688
    got, row = ops.paged_attention(*args, quant_out=gs, **kw), ops.quantize_act(plain.view(T, K), "nvfp4", static_scale=gs)
    ops.check_status(DEV)

    def values(a):
        sf = ref.tiled_to_sf(a.sf.cpu().view(-1, a.sf_k64, 512), T, K // 16)
        return ref.dequantize_nvfp4(a.data.cpu(), sf, a.scale[:T].cpu()).double()
    g, v, w = values(got), values(row), want.view(T, K).cpu()
    # the row kernel reads a bf16 output, this one the fp32 value: they differ where that rounding crosses an edge of the grid
    assert (g != v).double().mean() < 0.03 and (g - w).norm() <= 1.01 * (v - w).norm()
