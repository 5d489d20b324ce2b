"""Many short rows (csrc/rowops.cu: eight rows a CTA, a warp each) against the same rows in launches of fewer, a CTA each: the same bits."""
import pytest
import torch

from metrale_inference_alpha_b200 import ops
from metrale_inference_alpha_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
PART = 600                                                               # rows of a launch that takes a CTA a row


def _values(act, rows):
    """Everything that the listed rows of an encoded matrix hold."""
    out = [act.data[rows]]
    if act.fmt == "fp8_g128":
        out.append(act.scale[:, rows])
    elif act.fmt != "bf16":
        out.append(act.scale[rows])
    if act.fmt == "nvfp4":
        M, K = act.data.shape[0], act.K
        out.append(ref.tiled_to_sf(act.sf.view(-1, act.sf_k64, 512), M, K // 16)[rows])
    if act.bf16 is not None:
        out.append(act.bf16[rows])
    return out


# the first number of rows that takes this form, a last CTA with one row and with seven
@pytest.mark.parametrize("mode,M", [(m, n + k) for m, n in (("copy", 1184), ("norm", 1184), ("silu", 2960)) for k in (0, 1, 7)])
@pytest.mark.parametrize("K,fmt", [(16, "bf16"), (272, "bf16"), (512, "bf16"), (16, "fp8_row"), (272, "fp8_row"), (512, "fp8_row"),
                                   (128, "fp8_g128"), (512, "fp8_g128"), (64, "nvfp4"), (256, "nvfp4"), (512, "nvfp4")])
def test_rows_are_the_same_a_warp_or_a_cta_each(M, K, fmt, mode):
    g = torch.Generator(device=DEV).manual_seed(M + K)
    x = (torch.randn(M, 2 * K if mode == "silu" else K, generator=g, device=DEV) * 3).bfloat16()
    kw = dict(copy=dict(mode=ops.IN_COPY), norm=dict(mode=ops.IN_RMSNORM, w=torch.randn(K, generator=g, device=DEV).bfloat16(), plus_one=True),
              silu=dict(mode=ops.IN_SILU_MUL))[mode]
    kw["also_bf16"] = fmt != "bf16"
    every = torch.arange(M, device=DEV)
    got = _values(ops.row_op(x, fmt, **kw)[0], every)
    parts = [_values(ops.row_op(x[i:i + PART], fmt, **kw)[0], torch.arange(len(x[i:i + PART]), device=DEV)) for i in range(0, M, PART)]
    for k, a in enumerate(got):
        along = 1 if fmt == "fp8_g128" and k == 1 else 0
        assert torch.equal(a, torch.cat([p[k] for p in parts], along))
    # a list of rows with holes, in another order
    index = torch.randperm(M, generator=g, device=DEV).int()
    index[3::7] = -1
    listed = index[index >= 0].long()
    some = _values(ops.row_op(x, fmt, row_index=index, **kw)[0], listed)
    for k, (a, b) in enumerate(zip(some, got)):
        assert torch.equal(a, b[:, listed] if fmt == "fp8_g128" and k == 1 else b[listed])
