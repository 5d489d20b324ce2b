"""The rows that logits are wanted of (``ForwardBatch.logit_rows``), in every form that indexing takes and none that it refuses."""
import pytest
import torch

from metrale_inference_alpha_b200.config.model_config import preset
from metrale_inference_alpha_b200.engine.batch import ForwardBatch
from metrale_inference_alpha_b200.engine.llm_engine import EngineArgs, LLMEngine


def _forward(device):
    cfg = preset("dense-27b-nvfp4", num_layers=1, hidden_size=256, num_heads=2, num_kv_heads=1, head_dim=128, intermediate_size=512, vocab_size=256,
                 mtp_layers=0, max_position=256, weight_format="bf16", kv_dtype="bf16")
    r = LLMEngine(EngineArgs(model=cfg, device=device, max_model_len=128, num_kv_blocks=16)).runner
    batch = ForwardBatch.build([dict(tokens=[(7 * i + 3) % 256 for i in range(9)], start_pos=0, blocks=[1], state_slot=0, logits="all")], 16, device=device)

    def run(rows):
        batch.logit_rows = rows
        return r.decoder.forward(batch, r.caches)
    return run


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda:0", marks=pytest.mark.gpu)])
def test_rows_are_taken_in_every_form_of_an_index(device):
    run = _forward(device)
    every = [t.clone() for t in run(torch.arange(9, device=device))]
    want = [5, 0, 5, 8]
    pair = torch.tensor([[5, 1], [0, 2], [5, 3], [8, 4]], device=device)
    for dtype in (torch.int32, torch.int64):
        for rows in (torch.tensor(want, dtype=dtype, device=device), pair.to(dtype)[:, 0]):          # whole and strided
            got = run(rows)
            assert torch.equal(got[1], every[1][want])
            assert (got[0].float() - every[0][want].float()).abs().max() <= 2.0 ** -7 * every[0].float().abs().max()
    for rows in (pair, torch.tensor(want, dtype=torch.int16, device=device), torch.tensor([True, False], device=device)):
        with pytest.raises((IndexError, RuntimeError)):
            run(rows)


def test_rows_that_are_not_there_are_refused_on_the_cpu():
    run = _forward("cpu")
    for row in (-1, 9):
        with pytest.raises((IndexError, RuntimeError)):
            run(torch.tensor([0, row]))
