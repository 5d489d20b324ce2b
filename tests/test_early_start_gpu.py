"""Rotation and decode attention that come up under the kernel in front of them (`early`) give the bits that they give behind it, when
inputs change in the same buffers from step to step and the step's own cache rows hold something else before."""
import pytest
import torch

from metrale_inference_alpha_b200 import ops
from metrale_inference_alpha_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# new tokens that begin on and off an edge of 16 and of 32 tokens, alone or behind partitions; one to five of a sequence
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("D,Hq,Hkv,news,pasts", [
    (128, 10, 2, [1, 1, 1, 1], [31, 32, 47, 0]), (128, 10, 2, [2, 5, 1, 3], [30, 29, 1023, 1024]), (128, 40, 8, [4] * 6, [44, 60, 61, 700, 2044, 3]),
    (128, 40, 8, [1] * 40, [37 * i + 1 for i in range(40)]), (256, 16, 2, [1, 2, 1], [15, 14, 1500])])
def test_early_launches_give_the_same_bits(fp8, D, Hq, Hkv, news, pasts):
    g = torch.Generator(device=DEV).manual_seed(len(news) + D)
    bs, T, S, hidden = 16, sum(news), len(news), 2048
    need = [(n + p + bs - 1) // bs for n, p in zip(news, pasts)]
    order = torch.randperm(sum(need), generator=g, device=DEV).int() + 1
    bt = torch.zeros(S, max(need), dtype=torch.int32, device=DEV)
    at, slots, pos = 0, [], []
    for s, k in enumerate(need):
        bt[s, :k] = order[at:at + k]
        for t in range(pasts[s], pasts[s] + news[s]):
            slots.append(int(order[at + t // bs]) * bs + t % bs)
            pos.append(t)
        at += k
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    slots, pos, q_len, ctx = torch.tensor(slots, device=DEV), i32(pos), i32(news), i32([n + p for n, p in zip(news, pasts)])
    q_start = (torch.cumsum(q_len, 0) - q_len).int()
    shape, dt, nan = (sum(need) + 1, bs, Hkv, D), torch.uint8 if fp8 else torch.bfloat16, 0x7f if fp8 else float("nan")
    kv = [torch.randn(shape, generator=g, device=DEV).bfloat16() for _ in range(2)]
    kv = [x.to(torch.float8_e4m3fn).view(dt) if fp8 else x for x in kv]
    one = torch.ones(1, device=DEV)
    w = ops.make_weight(torch.randn((Hq + 2 * Hkv) * D, hidden, generator=g, device=DEV).cpu() * 0.02, "bf16").to(DEV)
    ln, qn = (torch.ones(n, device=DEV).bfloat16() for n in (hidden, D))
    cos, sin = (t.to(DEV) for t in ref.rope_tables(8192, D, 1e6))
    x = torch.empty(T, hidden, dtype=torch.bfloat16, device=DEV)

    def step(early):
        for c in kv:
            c.view(-1, Hkv, D).index_fill_(0, slots, nan)                      # what is read too soon shows
        a = ops.row_op(x, "bf16", ops.IN_RMSNORM, w=ln)[0]
        q = ops.qk_norm_rope_kvwrite(ops.linear(a, w), Hq=Hq, Hkv=Hkv, D=D, positions=pos, slots=slots, k_cache=kv[0], v_cache=kv[1], q_norm_w=qn,
                                     k_norm_w=qn, cos=cos, sin=sin, k_scale=one, v_scale=one, early=early)
        o = ops.paged_attention(q, *kv, bt, q_start, q_len, ctx, max_q_len=max(news), max_ctx=4096, scale=D ** -0.5, k_scale=one, v_scale=one, early=early)
        return [q, o] + [c.view(-1, Hkv, D)[slots] for c in kv]

    x.normal_(generator=g)
    step(True)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        replayed = step(True)
    for _ in range(40):
        x.normal_(generator=g)
        want = [t.clone() for t in step(False)]
        got = [t.clone() for t in step(True)]
        graph.replay()
        for a, b, c in zip(want, got, replayed):
            assert not a.float().isnan().any() or a.dtype == torch.uint8
            assert torch.equal(a, b) and torch.equal(a, c)
    ops.check_status(DEV)
