"""Decode / verify attention over a list of (sequence, partition, head) units (csrc/attention_decode.cu), against attention in 64 bits."""
import pytest
import torch

from metrale_inference_alpha_b200 import ops
from metrale_inference_alpha_b200.ops import reference as ref
from test_attn_rows_gpu import _case as _case128

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _case(fp8, D, Hq, Hkv, q_lens, ctx_lens, bs, seed=0):
    if D == 128:
        return _case128(fp8, Hq, Hkv, q_lens, ctx_lens, bs, seed)
    # two heads of 128 seen as one of 256: the same caches and queries, their own answer
    (q, kc, vc, bt, qs, ql, ctx), kw, _ = _case128(fp8, 2 * Hq, 2 * Hkv, q_lens, ctx_lens, bs, seed)
    q, kc, vc = q.reshape(-1, Hq, 256), kc.view(*kc.shape[:2], Hkv, 256), vc.view(*vc.shape[:2], Hkv, 256)
    out, at, G = torch.empty(q.shape, dtype=torch.float64, device=DEV), 0, Hq // Hkv
    for s, (n, c) in enumerate(zip(q_lens, ctx_lens)):
        k, v = ((t.view(torch.float8_e4m3fn) if fp8 else t)[bt[s, :(c + bs - 1) // bs].long()].reshape(-1, Hkv, 256)[:c].double() *
                (1.0 if sc is None else sc.double()) for t, sc in ((kc, kw["k_scale"]), (vc, kw["v_scale"])))
        mask = torch.arange(c, device=DEV)[None] <= torch.arange(c - n, c, device=DEV)[:, None]
        for h in range(Hq):
            w = torch.softmax((q[at:at + n, h].double() @ k[:, h // G].t() * kw["scale"]).masked_fill(~mask, -torch.inf), -1)
            out[at:at + n, h] = w @ v[:, h // G]
        at += n
    return (q, kc, vc, bt, qs, ql, ctx), kw, out


# one token and the edges of a slice of 16, of four warps' slices, of a partition; ragged batches with verify rows among them; one
# head a group and sixteen; two row tiles; blocks that hold several slices or are no power of two; more units than CTAs
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("D,Hq,Hkv,q_lens,ctx_lens,bs", [
    (128, 40, 8, [1], [1], 16), (128, 5, 1, [1, 1, 1, 1, 1], [15, 16, 17, 64, 65], 16), (128, 40, 8, [1, 1, 1], [255, 256, 257], 16),
    (128, 1, 1, [1, 1], [8191, 9000], 16), (128, 16, 1, [1], [700], 64), (128, 5, 1, [4, 1, 3], [4, 333, 600], 16),
    (128, 4, 1, [8, 2], [100, 513], 48), (128, 40, 8, [1] * 130, [7 * i % 900 + 1 for i in range(130)], 16),
    (256, 16, 2, [1, 1], [90, 1025], 16), (256, 8, 1, [1, 2], [33, 300], 32), (128, 32, 8, [8] * 41, [9 + 29 * i % 700 for i in range(41)], 16)])
def test_matches_attention_in_64_bits(fp8, D, Hq, Hkv, q_lens, ctx_lens, bs):
    args, kw, want = _case(fp8, D, Hq, Hkv, q_lens, ctx_lens, bs)
    for part in (0, 64, 1024):
        got = ops.paged_attention(*args, part_tokens=part, **kw)
        ops.check_status(DEV)
        # the result's bf16 rounding (2^-9 of each value at most) and the weights' (2^-9 in bf16, 2^-12 in f16, independent per token)
        assert (got.double() - want).norm() <= 2.0 ** -8 * want.norm(), part
        assert torch.equal(got, ops.paged_attention(*args, part_tokens=part, **kw))
    other = ops.paged_attention(*args, force_mode=1, **kw)              # the split-KV kernel
    assert (got.double() - other.double()).norm() <= 2.0 ** -7 * want.norm()


def test_a_sequence_does_not_depend_on_its_batch():
    lens = [3000, 17, 900, 1, 256, 2047, 700, 64]
    (q, kc, vc, bt, qs, ql, ctx), kw, _ = _case(True, 128, 40, 8, [1] * 8, lens, 16)
    many = ops.paged_attention(q, kc, vc, bt, qs, ql, ctx, **kw)
    for i in range(8):
        one = ops.paged_attention(q[i:i + 1], kc, vc, bt[i:i + 1], qs[:1], ql[:1], ctx[i:i + 1], **dict(kw, max_ctx=8192))
        assert torch.equal(one[0], many[i])


def test_sequences_without_queries_and_padding_rows_are_passed_over():
    (q, kc, vc, bt, qs, ql, ctx), kw, want = _case(False, 128, 8, 2, [1, 1, 1], [40, 300, 77], 16)
    keep = torch.tensor([0, 2], device=DEV)
    ql[1] = 0
    got = torch.full_like(q, 3.0)
    got[keep] = ops.paged_attention(q, kc, vc, bt, qs, ql, ctx, **kw)[keep]
    ops.check_status(DEV)
    assert (got[keep].double() - want[keep]).norm() <= 2.0 ** -8 * want.norm()


@pytest.mark.parametrize("q_lens,ctx_lens", [([1] * 3, [200, 1, 1500]), ([3, 2], [3, 700])])
def test_quantised_output(q_lens, ctx_lens):
    args, kw, want = _case(True, 128, 40, 8, q_lens, ctx_lens, 16)
    T, K, gs = sum(q_lens), 40 * 128, 2 * 6.0 / 2688
    plain, got = ops.paged_attention(*args, **kw), ops.paged_attention(*args, quant_out=gs, **kw)
    row = ops.quantize_act(plain.view(T, K), "nvfp4", static_scale=gs)
    ops.check_status(DEV)

    def values(a):
        sf = ref.tiled_to_sf(a.sf.cpu().view(-1, a.sf_k64, 512), T, K // 16)
        return ref.dequantize_nvfp4(a.data.cpu(), sf, a.scale[:T].cpu()).double()
    g, v, w = values(got), values(row), want.view(T, K).cpu()
    assert (g != v).double().mean() < 0.03 and (g - w).norm() <= 1.01 * (v - w).norm()
