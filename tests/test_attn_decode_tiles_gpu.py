"""Decode attention at every count of eights of query rows (csrc/attention_decode.cu: odd counts have the cache on the products' 16-row side,
even ones the queries), at their first and last row."""
import pytest
import torch

from metrale_inference_alpha_b200 import ops
from metrale_inference_alpha_b200.ops import reference as ref
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


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("G,n", [(17, 1), (5, 4), (8, 3), (5, 5), (16, 2)])
def test_quantised_output_of_17_to_32_rows_is_the_row_kernels(fp8, G, n):
    """What leaves quantised is the bf16 output, as a row kernel behind the plain call reads it: the same bits."""
    q_lens, ctx_lens, Hq = [n, 1, n, n], [n, 40, 700, 1300], 2 * G
    args, kw, _ = _case(fp8, 128, Hq, 2, q_lens, ctx_lens, 16)
    T, gs = sum(q_lens), 2 * 6.0 / 2688
    got = ops.paged_attention(*args, quant_out=gs, **kw)
    row = ops.quantize_act(ops.paged_attention(*args, **kw).view(T, Hq * 128), "nvfp4", static_scale=gs)
    ops.check_status(DEV)
    assert torch.equal(got.data, row.data)
    sf = lambda a: ref.tiled_to_sf(a.sf.cpu().view(-1, a.sf_k64, 512), T, Hq * 8)
    assert torch.equal(sf(got), sf(row))
