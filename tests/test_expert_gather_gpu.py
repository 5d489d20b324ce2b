"""Gathering rows by expert (csrc/moe.cu), a warp or a CTA a row: every sorted row is its token's, scales included."""
import pytest
import torch

from metrale_inference_alpha_b200 import ops
from metrale_inference_alpha_b200.ops import moe_cuda

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# lengths around a turn of a warp's (2048 bytes) and of a CTA's (8192 bytes) vectors and around the lines between them; few and many rows
@pytest.mark.parametrize("T", [1, 3, 255, 256])
@pytest.mark.parametrize("fmt,H", [("bf16", 8), ("bf16", 1024), ("bf16", 1032), ("bf16", 2560), ("bf16", 2568), ("bf16", 4104), ("fp8_g128", 128),
                                   ("fp8_g128", 2176), ("fp8_g128", 8320), ("fp8_row", 2064)])
def test_rows_follow_their_pairs(T, fmt, H):
    K, E = 8, 12
    g = torch.Generator(device=DEV).manual_seed(T + H)
    idx = torch.randint(0, E, (T, K), generator=g, device=DEV, dtype=torch.int32)
    idx[T // 2, 3] = -1                                                  # an expert that is not here
    sp = moe_cuda.SortedPairs(idx, 0, E, 64)
    a = ops.row_op(torch.randn(T, H, generator=g, device=DEV).bfloat16(), fmt)[0]
    got = moe_cuda.gather_act(a, sp)
    row = sp.pair_row.long()
    pairs = (row >= 0).nonzero()[:, 0]
    assert torch.equal(got.data[row[pairs]].view(torch.uint8), a.data[pairs // K].view(torch.uint8))
    if fmt == "fp8_g128":
        assert torch.equal(got.scale[:, row[pairs]], a.scale[:, pairs // K])
    elif fmt == "fp8_row":
        assert torch.equal(got.scale[row[pairs]], a.scale[pairs // K])
