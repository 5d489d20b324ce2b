"""The native call of a dense NVFP4 layer issues the launches that the blocks issue one by one: the same bits."""
import pytest
import torch

from metrale_inference_alpha_b200 import ops
from metrale_inference_alpha_b200.config.model_config import preset
from metrale_inference_alpha_b200.engine.batch import ForwardBatch
from metrale_inference_alpha_b200.engine.llm_engine import EngineArgs, LLMEngine
from metrale_inference_alpha_b200.ops import dense_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inter", [2048, 9728])                          # SwiGLU quantised behind the GEMM, and inside it at any size
@pytest.mark.parametrize("lens", [[(1, 700), (1, 30), (1, 0)], [(5, 40), (2, 1500)], [(40, 0), (100, 9)], [(200, 0), (1, 3), (133, 300)]])
def test_native_layer_is_the_blocks(inter, lens, monkeypatch):
    cfg = preset("dense-27b-nvfp4", num_layers=2, hidden_size=512, num_heads=8, num_kv_heads=2, intermediate_size=inter, vocab_size=512, mtp_layers=0,
                 max_position=4096)
    r = LLMEngine(EngineArgs(model=cfg, device="cuda:0", max_model_len=2048, num_kv_blocks=256)).runner
    seqs, at = [], 1
    for n, past in lens:
        k = (n + past + 15) // 16
        seqs.append(dict(tokens=[(7 * i + 3) % 512 for i in range(n)], start_pos=past, blocks=list(range(at, at + k)), state_slot=0, logits="last"))
        at += k
    batch = ForwardBatch.build(seqs, 16, device="cuda:0")
    g = torch.Generator(device="cuda:0").manual_seed(1)
    start = [torch.randn(t.shape, generator=g, device="cuda:0").to(torch.float8_e4m3fn).view(torch.uint8) for t in r.kv.k + r.kv.v]
    calls, seen = [], []
    real = dense_layer.dense_layer
    monkeypatch.setattr(dense_layer, "dense_layer", lambda *a, **k: calls.append(1) or real(*a, **k))
    for single in (False, True):
        monkeypatch.setattr(dense_layer, "observed", lambda: single)
        for t, s in zip(r.kv.k + r.kv.v, start):
            t.copy_(s)
        n0 = ops.launch_count
        logits, hidden = r.decoder.forward(batch, r.caches)
        ops.check_status("cuda:0")
        seen.append((ops.launch_count - n0, [logits, hidden] + [t.clone() for t in r.kv.k + r.kv.v]))
        assert len(calls) == 2                                           # both layers, in the first pass only
    assert seen[0][0] == seen[1][0]
    assert all(torch.equal(a, b) for a, b in zip(seen[0][1], seen[1][1]))
