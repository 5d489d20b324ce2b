"""Operands of the chunked gated delta rule's products (csrc/gdn_chunked.cu) are rounded to TF32's 11 significant bits to the nearest,
half way cases away from zero. One written token makes the rounding visible: from an empty state, with a decay and a write strength
of one and a key along one axis, the state's row of that axis is the rounded value row, exactly (a product with 1, a sum with zeros)."""
import numpy as np
import pytest
import torch

from metrale_inference_alpha_b200.ops import recurrent as rec
from types import SimpleNamespace

pytestmark = pytest.mark.gpu


def nearest_tf32(x: np.ndarray) -> np.ndarray:
    """11 significant bits, ties away from zero, in integers; numbers that round beyond the largest become infinite."""
    b = x.view(np.uint32).astype(np.uint64)
    mag = (b & 0x7fffffff) + 0x1000 & 0xffffe000
    out = ((b & 0x80000000) | np.minimum(mag, 0x7f800000)).astype(np.uint32)
    return np.where(np.isnan(x), np.float32(np.nan), out.view(np.float32))


def values(n: int, kind: str) -> np.ndarray:
    r = np.random.default_rng(11)
    m = r.integers(0, 1 << 23, n, dtype=np.uint32)
    sign = r.integers(0, 2, n, dtype=np.uint32) << 31
    e = {"ordinary": r.integers(110, 140, n), "ties": 8 + np.arange(n) % 240, "large": r.integers(235, 255, n), "special": r.integers(8, 255, n)}[kind]
    if kind == "ties":
        m = (m & 0x7fe000) | 0x1000
    x = (sign | e.astype(np.uint32) << 23 | m).view(np.float32).copy()
    if kind == "special":
        x[0::5], x[1::5], x[2::5], x[3::5] = np.inf, -np.inf, np.nan, np.finfo(np.float32).max
        x[4::10] = np.uint32(0x7f800001).view(np.float32)                  # a NaN whose payload lies below the 11 bits
    return x


@pytest.mark.parametrize("kind", ["ordinary", "ties", "large", "special"])
def test_written_values_are_rounded_to_the_nearest_with_ties_away_from_zero(kind):
    T, kh, vh, D, dev = 64, 4, 16, 128, "cuda"
    v = values(vh * D, kind)
    conv = torch.zeros(T, 2 * kh * D + vh * D, device=dev)
    conv[T - 1, kh * D + torch.arange(kh) * D + 5] = 1.0                   # the last token's key, axis 5
    conv[T - 1, 2 * kh * D:] = torch.from_numpy(v).to(dev)
    ba = torch.cat([torch.full((T, vh), 1000.0), torch.full((T, vh), -1000.0)], 1).to(dev)      # write strength 1, decay 1
    state = torch.full((2, vh, D, D), 7.0, device=dev)                     # an earlier sequence's: position 0 starts from zero
    i32 = lambda *x: torch.tensor(x, dtype=torch.int32, device=dev)
    batch = SimpleNamespace(q_start=i32(0), q_len=i32(T), positions=torch.arange(T, dtype=torch.int32, device=dev), state_slots=i32(1),
                            max_q_len=T)
    out = rec._gdn_chunked_cuda(conv, ba, torch.zeros(vh, device=dev), torch.zeros(vh, device=dev), state, batch, kh, vh, True)
    assert out is not None
    got = state[1, :, 5].flatten().cpu().numpy()
    want = nearest_tf32(v)
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got[~nan].view(np.uint32), want[~nan].view(np.uint32))
    if np.isfinite(want).all():
        rest = torch.cat([state[1, :, :5], state[1, :, 6:]], 1)
        assert not rest.any()


@pytest.mark.parametrize("where", ["key", "state"])
def test_a_nan_reaches_the_state(where):
    """Of either sign: rounding keeps it."""
    T, kh, vh, D, dev = 64, 1, 1, 128, "cuda"
    g = torch.Generator(device=dev).manual_seed(0)
    conv = torch.randn(T, 2 * kh * D + vh * D, generator=g, device=dev)
    state = torch.randn(2, vh, D, D, generator=g, device=dev)
    nan = torch.tensor([-1], dtype=torch.int32, device=dev).view(torch.float32)
    (conv[40, kh * D + 3:kh * D + 4] if where == "key" else state[1, 0, 3, 7:8]).copy_(nan)
    i32 = lambda *x: torch.tensor(x, dtype=torch.int32, device=dev)
    batch = SimpleNamespace(q_start=i32(0), q_len=i32(T), positions=torch.arange(9, 9 + T, dtype=torch.int32, device=dev), state_slots=i32(1),
                            max_q_len=T)
    out = rec._gdn_chunked_cuda(conv, torch.randn(T, 2 * vh, generator=g, device=dev), torch.zeros(vh, device=dev), torch.zeros(vh, device=dev),
                                state, batch, kh, vh, True)
    if where == "key":
        assert state[1].isnan().all() and out[40:].isnan().all()
    else:                                                                  # one value column, which every later row reads
        assert state[1, 0, :, 7].isnan().all() and out[:, 7].isnan().all() and int(state[1].isnan().sum()) == D and int(out.isnan().sum()) == T
