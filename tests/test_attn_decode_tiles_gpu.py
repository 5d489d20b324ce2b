"""Decode attention at every count of eights of query rows (csrc/attention_decode.cu: odd counts have the cache on the products' 16-row side,
even ones the queries), at their first and last row."""
import pytest
import torch

from metrale_inference_alpha_b200 import ops
from test_attn_decode_gpu import _case

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("D,G,n", [(128, 8, 1), (128, 3, 3), (128, 16, 1), (128, 17, 1), (128, 8, 3), (128, 5, 5), (128, 16, 2),
                                   (256, 8, 1), (256, 3, 3), (256, 8, 2)])
def test_every_count_of_rows_matches_attention_in_64_bits(fp8, D, G, n):
    q_lens, ctx_lens = [n, 1, n, n], [n, 40, 700, 1300]                 # one token seen, a slice's edge, several partitions
    args, kw, want = _case(fp8, D, 2 * G, 2, q_lens, ctx_lens, 16)
    got = ops.paged_attention(*args, **kw)
    ops.check_status(DEV)
    # the result's bf16 rounding (2^-9 of each value at most) and the weights' (2^-9 in bf16, 2^-12 in f16, independent per token)
    assert (got.double() - want).norm() <= 2.0 ** -8 * want.norm()
    assert (got.double() - want).abs().max() <= 2.0 ** -6 * want.abs().max()
    assert torch.equal(got, ops.paged_attention(*args, **kw))
