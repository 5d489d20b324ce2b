"""The grouped fp8-block GEMM of few rows an expert against 64-bit sums of the same quantised operands."""
import pytest
import torch

from metrale_inference_alpha_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("tile_rows", [16, 32, 64])
@pytest.mark.parametrize("K,N,out_f32,E", [(128, 128, True, 5), (2048, 256, False, 5), (17 * 128, 128, True, 5),
                                           (128, 1024, True, 60), (512, 1152, True, 60), (640, 1024, False, 120)])   # several tiles a CTA
def test_few_rows_per_expert(tile_rows, K, N, out_f32, E):
    g = torch.Generator().manual_seed(K + tile_rows)
    counts = [1, 0, tile_rows, tile_rows + 3, 2] * (E // 5)              # an expert without rows, one of two entries
    w = [ops.make_weight(torch.randn(N, K, generator=g) * 0.05, "fp8_block") for _ in range(E)]
    rows = sum(counts)
    x = ops.row_op(torch.randn(rows, K, generator=g).bfloat16().to(DEV), "fp8_g128", scale_pad=64)[0]
    tiles, at = [], 0
    for e, n in enumerate(counts):
        tiles += [(e, at + j, min(tile_rows, n - j)) for j in range(0, n, tile_rows)]
        at += n
    tiles = tiles[:2] + [(-1, 0, 0)] + tiles[2:] + [(-1, 0, 0)] * 3
    te, r0, nr = (torch.tensor(c, dtype=torch.int32, device=DEV) for c in zip(*tiles))
    stacked = ops.QuantWeight("fp8_block", E * N, K, torch.cat([q.data for q in w]).to(DEV), torch.cat([q.scale for q in w]).to(DEV))
    got = ops.linear(x, stacked, out_f32=out_f32, grouped=(te, r0, nr, N, len(tiles), tile_rows))
    ops.check_status(DEV)
    a = ops.ref.from_e4m3(x.data.cpu()).double() * x.scale[:, :rows].cpu().t().double().repeat_interleave(128, 1)
    at = 0
    for e, n in enumerate(counts):
        rows_e, we = a[at:at + n], w[e].dequant().double()
        # K / 128 scaled blocks summed in 32 bits, each a sum of 128 exact products whose rounding is below 2^-20 of their size
        bound = 2.0 ** -19 * (rows_e.abs() @ we.abs().t()) + (0 if out_f32 else 2.0 ** -8) * (rows_e @ we.t()).abs()
        assert ((got[at:at + n].cpu().double() - rows_e @ we.t()).abs() <= bound + 1e-9).all(), e
        at += n
