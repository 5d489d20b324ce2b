"""The tail of an expert block (csrc/moe.cu) at sizes of whole 16-byte vectors and others, against the sum in slot order."""
import pytest
import torch

from metrale_inference_alpha_b200.ops import _native, moe_cuda  # noqa: F401

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("T,K,H,pad", [(1, 1, 4, 0), (3, 4, 512, 0), (17, 9, 2048, 0), (5, 5, 516, 4), (5, 3, 130, 2), (2049, 2, 256, 0)])
@pytest.mark.parametrize("extra", [False, True])
def test_finish_sums_the_rows_of_every_slot(T, K, H, pad, extra):
    g = torch.Generator(device=DEV).manual_seed(T * K)
    y = torch.randn(T * K + 3, H + pad, generator=g, device=DEV)[:, :H]
    row = torch.randperm(T * K, generator=g, device=DEV).to(torch.int32).view(T, K)
    row[0, K - 1] = -1                                    # an expert that is not here
    w = torch.rand(T, K, generator=g, device=DEV)
    shared = torch.randn(T, H, generator=g, device=DEV).bfloat16() if extra else None
    gate = torch.randn(T, 1, generator=g, device=DEV) if extra else None
    res = torch.randn(T, H, generator=g, device=DEV).bfloat16() if extra else None
    out = torch.empty(T, H, dtype=torch.bfloat16, device=DEV)
    p = lambda t: None if t is None else t.data_ptr()
    rc = _native.lib().mb_moe_finish(p(y), y.stride(0), p(row), p(w), T, K, H, p(shared), H if extra else 0, p(gate), 1 if extra else 0, p(res),
                                     p(out), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    want = (torch.where(row[..., None] >= 0, y[row.clamp(min=0).long()].double(), 0.0) * w[..., None].double()).sum(1)
    if extra:
        want += torch.sigmoid(gate.double()) * shared.double() + res.double()
    assert (out.double() - want).abs().max() <= 2.0 ** -8 * want.abs().max()        # the result's bf16 rounding
