"""The vector kernel of rotation, head norms and cache writes (csrc/attention.cu) against the oracle and the warp-per-head kernel."""
import pytest
import torch

from metrale_inference_alpha_b200 import ops
from metrale_inference_alpha_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


# heads that fill no whole pass of a CTA, gates between the query heads, every head size, one token and more than a wave of them
@pytest.mark.parametrize("norm,rotate", [(True, True), (False, True), (True, False)])
@pytest.mark.parametrize("M,Hq,Hkv,D,rot,gap", [(1, 40, 8, 128, 128, 1), (700, 5, 1, 128, 64, 1), (37, 3, 1, 64, 32, 2), (65, 6, 3, 256, 64, 2), (9, 1, 1, 256, 256, 1)])
def test_vector_kernel_matches_the_oracle_and_the_warp_kernel(M, Hq, Hkv, D, rot, gap, norm, rotate):
    g = torch.Generator().manual_seed(M)
    nb, qhs = M // 16 + 2, gap * D
    width = Hq * qhs + 2 * Hkv * D
    wide = torch.randn(M, width + 8, generator=g).to(torch.bfloat16)           # rows 16 bytes longer than they need be
    pos = torch.randint(0, 500, (M,), generator=g, dtype=torch.int32)
    slots = torch.randperm(nb * 16, generator=g)[:M].to(torch.int64)
    if M > 3:
        slots[3] = -1
    kw = dict(Hq=Hq, Hkv=Hkv, D=D, q_head_stride=qhs)
    if norm:
        kw.update(q_norm_w=(torch.randn(D, generator=g) * 0.1 + 1).to(torch.bfloat16), k_norm_w=(torch.randn(D, generator=g) * 0.1 + 1).to(torch.bfloat16))
    if rotate:
        kw["cos"], kw["sin"] = ref.rope_tables(512, rot, 1e6)

    def run(dev, qkv):
        t = {k: v.to(dev) if torch.is_tensor(v) else v for k, v in kw.items()}
        kc, vc = (torch.zeros(nb, 16, Hkv, D, dtype=torch.bfloat16, device=dev) for _ in range(2))
        return ops.qk_norm_rope_kvwrite(qkv, positions=pos.to(dev), slots=slots.to(dev), k_cache=kc, v_cache=vc, **t), kc, vc
    want = run("cpu", wide[:, :width])
    on = wide.to(DEV)
    got = run(DEV, on[:, :width])
    odd = torch.empty(M, width + 1, dtype=torch.bfloat16, device=DEV)           # odd pitch: the warp-per-head kernel
    odd[:, :width] = on[:, :width]
    other = run(DEV, odd[:, :width])
    ops.check_status(DEV)
    for a, b, c in zip(got, other, want):
        # one bf16 ulp of the norm's rounding, carried through a rotation (|cos| + |sin| <= sqrt 2) and rounded again
        tol = 2.0 ** -7 * c.float().abs().clamp(min=2.0 ** -7).amax()
        assert (a.float() - b.float()).abs().max() <= tol and (a.cpu().float() - c.float()).abs().max() <= tol
        assert (a != b).float().mean() < 0.02
