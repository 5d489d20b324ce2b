"""The gated row recipes in registers (csrc/rowops.cu), against the kernel that takes rows of any alignment and the oracle."""
import pytest
import torch

from metrale_inference_alpha_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one group of eight threads, a row that ends inside a warp, the widest; heads of one block and of several
@pytest.mark.parametrize("K,D", [(128, 16), (640, 64), (4096, 256), (8192, 128)])
@pytest.mark.parametrize("fmt", ["bf16", "fp8_row", "fp8_g128", "nvfp4"])
@pytest.mark.parametrize("mode", [ops.IN_SIGMOID_GATE, ops.IN_GATED_RMSNORM])
def test_gated_rows(K, D, fmt, mode):
    M, g = 37, torch.Generator().manual_seed(K + D)
    norm = mode == ops.IN_GATED_RMSNORM
    x = torch.randn(M, K, generator=g) * 3
    x = x if norm else x.bfloat16()
    wide = torch.randn(M, 2 * K + 9, generator=g).bfloat16()
    kw = dict(w=(torch.randn(K, generator=g) * 0.2 + 1).bfloat16(), group=128, eps=1e-6) if norm else dict(head_dim=D, gate_head_stride=2 * D, gate_head_off=D)
    dev = {k: v.to(DEV) if torch.is_tensor(v) else v for k, v in kw.items()}
    run = lambda gate: ops.row_op(x.to(DEV), fmt, mode, gate=gate, also_bf16=True, **dev)[0]
    cols = K if norm else 2 * K
    gate = wide[:, :cols].contiguous()
    got, other = run(gate.to(DEV)), run(wide.to(DEV)[:, :cols])               # the second's rows start off a 16-byte boundary
    want = ops.row_op(x, fmt, mode, gate=gate, also_bf16=True, **kw)[0]
    ops.check_status(DEV)
    top = want.bf16.float().abs().max()
    # the sums of a group in another order and the fast exponential: an ulp of fp32 before the bf16 rounding
    for a, b in ((got, other), (got, want)):
        assert (a.bf16.cpu().float() - b.bf16.cpu().float()).abs().max() <= 2.0 ** -7 * top
    assert (got.bf16 != other.bf16).float().mean() < 0.01
    if fmt != "bf16":
        assert (got.data != other.data).float().mean() < 0.01
        s, t = (a.scale[:, :M] if fmt == "fp8_g128" else a.scale for a in (got, other))
        assert ((s - t).abs() <= 1e-5 * t.abs()).all()
