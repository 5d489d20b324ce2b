"""Prefill attention at head dim 256 (csrc/attention_rows256.cu) at the edges of its tiles, against attention in 64 bits."""
import math

import pytest
import torch

from metrale_inference_alpha_b200 import ops
from test_attn_decode_gpu import _case

pytestmark = pytest.mark.gpu
DEV = "cuda"


# a row short of, at and past tiles of 128 rows; contexts around tiles of 64 tokens; one tile beside many; groups that do not divide 128
# and eight heads; blocks that are no power of two; rows of very unequal sequences; enough tiles for the stages to come round
@pytest.mark.parametrize("Hq,Hkv,q_lens,ctx_lens,bs", [
    (1, 1, [128], [128], 16), (1, 1, [129], [129], 16), (2, 1, [128, 63, 64, 65], [128, 63, 64, 65], 16), (2, 2, [130, 5], [130, 5], 16),
    (5, 1, [128, 127], [1000, 127], 16), (3, 1, [257], [257], 24), (16, 2, [128, 200, 5, 1], [385, 200, 5, 700], 64),
    (8, 1, [130], [256], 48), (4, 2, [700], [700], 16), (2, 2, [131], [1900], 16)])
def test_matches_attention_in_64_bits(Hq, Hkv, q_lens, ctx_lens, bs):
    args, kw, want = _case(False, 256, Hq, Hkv, q_lens, ctx_lens, bs)
    got = ops.paged_attention(*args, **kw)
    ops.check_status(DEV)
    # the result's bf16 rounding and the weights' (2^-9 of each value at most, the latter independent per token)
    assert (got.double() - want).norm() <= 2.0 ** -8 * want.norm()
    assert (got.double() - want).abs().max() <= 2.0 ** -6 * want.abs().max()
    assert torch.equal(got, ops.paged_attention(*args, **kw))


@pytest.mark.parametrize("other", [12.0, -12.0, 0.0])
def test_scores_that_grow_along_the_context_rescale_the_output(other):
    """Keys that point ever more along every second query: its running maximum moves by more than 2^8 at every tile, beside rows
    whose maximum does the same, stands in the first tile, or has nothing to move by."""
    (q, kc, vc, bt, qs, ql, ctx), kw, _ = _case(False, 256, 2, 1, [256], [1024], 16)
    k = torch.zeros(1024, 1, 256, device=DEV)
    k[:, :, 0] = torch.linspace(-60, 90, 1024, device=DEV)[:, None]
    kc[bt[0, :64].long()] = k.bfloat16().view(64, 16, 1, 256)
    q = torch.zeros_like(q)
    q[::2, :, 0], q[1::2, :, 0] = 12.0, other
    got = ops.paged_attention(q, kc, vc, bt, qs, ql, ctx, **kw).double()
    ops.check_status(DEV)
    kk, vv = (t[bt[0, :64].long()].reshape(-1, 256).double() for t in (kc, vc))
    mask = torch.arange(1024, device=DEV)[None] <= torch.arange(768, 1024, device=DEV)[:, None]
    want = torch.softmax((q[:, 0].double() @ kk.t() * kw["scale"]).masked_fill(~mask, -math.inf), -1) @ vv
    for h in range(2):
        assert (got[:, h] - want).norm() <= 2.0 ** -8 * want.norm()
