"""A norm that takes its rows from a table by index, against taking them first."""
import pytest
import torch

from metrale_inference_alpha_b200 import ops
from metrale_inference_alpha_b200.models.stream import TableRows


def _check(dev, K, fmt, wide, rows, ids):
    g = torch.Generator().manual_seed(K)
    table, w = (torch.randn(rows, K, generator=g) * 2).bfloat16().to(dev), (torch.randn(K, generator=g) * 0.1).bfloat16().to(dev)
    idx = torch.tensor(ids, dtype=torch.int64 if wide else torch.int32, device=dev)
    lazy = TableRows(table, idx)
    act = lazy.reduce_norm(lazy, w, fmt, plus_one=True, also_bf16=True)
    want_rows = table[idx.long()]
    want = ops.row_op(want_rows, fmt, ops.IN_RMSNORM, w=w, plus_one=True, also_bf16=True)[0]
    assert torch.equal(lazy.resolve(), want_rows) and torch.equal(act.bf16, want.bf16) and torch.equal(act.data, want.data)
    for a, b in ((act.scale, want.scale), (act.sf, want.sf)):
        if a is not None and fmt != "bf16":
            if fmt == "fp8_g128":                            # columns past the rows are not written
                a, b = a[:, :len(ids)], b[:, :len(ids)]
            if a.dim() > 1 or a.dtype == torch.float32:
                assert torch.equal(a, b)


@pytest.mark.parametrize("wide", [False, True])
def test_rows_of_a_table_cpu(wide):
    _check("cpu", 64, "bf16", wide, 9, [3, 0, 8, 3])


@pytest.mark.gpu
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("K,fmt", [(100, "bf16"), (272, "bf16"), (2048, "fp8_g128"), (5120, "nvfp4"), (5120, "fp8_row"), (16384, "bf16")])
def test_rows_of_a_table(K, fmt, wide):
    _check("cuda:0", K, fmt, wide, 37, [36, 0, 5, 5, 17] * 3)


@pytest.mark.gpu
@pytest.mark.parametrize("K", [100, 256])
def test_rows_outside_the_table_are_zeros_and_reported(K):
    table, w = torch.ones(4, K, dtype=torch.bfloat16, device="cuda:0"), torch.ones(K, dtype=torch.bfloat16, device="cuda:0")
    act, rows = ops.row_op(table, "bf16", ops.IN_RMSNORM, w=w, gather=torch.tensor([1, -1, 4, 3], device="cuda:0"))
    assert rows[:, 0].tolist() == [1, 0, 0, 1] and act.data[:, 0].tolist() == [1, 0, 0, 1]
    with pytest.raises(ops._native.KernelError, match="bounds"):
        ops.check_status("cuda:0")
