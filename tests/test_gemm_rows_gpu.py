"""GEMMs of many token rows (csrc/gemm_rows.cu): pairs of CTAs for bf16, fp8 per row and NVFP4, 128 x 128 tiles for fp8 blocks,
at the edges of their tiles, against the one-tile-per-CTA kernel (the same products in the same order: equal bits) and the oracle."""
import pytest
import torch

from metrale_inference_alpha_b200 import ops
from metrale_inference_alpha_b200.ops import moe_cuda, reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _operands(fmt, M, N, K, seed=0):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(M, K, generator=g).to(torch.bfloat16)
    w = ops.make_weight(torch.randn(N, K, generator=g) * 0.05, fmt)
    return x, w, ops.quantize_act(x.to(DEV), ops.ACT_FOR_WEIGHT[fmt]), w.to(DEV)


def _oracle(x, w, fmt):
    return ops.encode_act_ref(x.float(), ops.ACT_FOR_WEIGHT[fmt]).data.double() @ w.dequant().double().t()


# one row past a tile, a whole pair tile, one row short of and past it; features short of, at and past 128 and 256; few k blocks
# (fewer than the ring's stages), a ragged last one, and enough for the ring to come round; N = 9600 makes 256-feature tiles
@pytest.mark.parametrize("M,N,K", [(129, 128, 512), (255, 384, 768), (256, 256, 256), (257, 512, 1280), (300, 9600, 512),
                                   (520, 1152, 2816), (4100, 1024, 512)])
@pytest.mark.parametrize("fmt", ["bf16", "fp8_row", "nvfp4"])
def test_pair_kernel_matches_the_one_tile_kernel_and_the_oracle(fmt, M, N, K):
    x, w_cpu, act, w = _operands(fmt, M, N, K)
    res = torch.randn(M, N, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).to(DEV)
    got = ops.linear(act, w, out_f32=True)
    if fmt != "bf16" or M > 256:                           # bf16 of one token tile stays with a tile per CTA, in splits of K
        assert torch.equal(ops.linear(act, w, residual=res), ops.linear(act, w, residual=res, one_tile_per_cta=True, force_splits=1))
        assert torch.equal(got, ops.linear(act, w, out_f32=True, one_tile_per_cta=True, force_splits=1))
    ops.check_status(DEV)
    # fp32 sums of K products of the encoded operands: K ulps of the largest partial sum, far below this
    want = _oracle(x, w_cpu, fmt)
    assert (got.cpu().double() - want).norm() <= 1e-5 * want.norm() * max(1.0, K / 1024)


@pytest.mark.parametrize("N,K", [(200, 264), (72, 64), (9608, 320)])
def test_pair_kernel_ragged_features_and_depth(N, K):
    """bf16 only: NVFP4 weights come in whole 128-row tiles. Rows that are not whole vectors take single stores."""
    x, w_cpu, act, w = _operands("bf16", 261, N, K, 3)
    got = ops.linear(act, w, out_f32=True)
    ops.check_status(DEV)
    want = _oracle(x, w_cpu, "bf16")
    assert (got.cpu().double() - want).norm() <= 1e-5 * want.norm()
    wide = torch.full((261, N + 3), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.linear(act, w, out=wide[:, :N])
    assert torch.equal(wide[:, :N], got.to(torch.bfloat16)) and bool((wide[:, N:] == 7).all())


@pytest.mark.parametrize("fmt", ["bf16", "fp8_row", "nvfp4", "fp8_block"])
@pytest.mark.parametrize("M,N", [(257, 257), (300, 1030), (389, 4099)])
def test_rows_that_are_not_whole_vectors(fmt, M, N):
    """Odd and even row lengths; a last row block of one row, of part of a warp, of whole warps: the same sums as a tile per CTA."""
    x, w_cpu, act, w = _operands(fmt, M, N, 512, 11)
    res = torch.randn(M, N, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).to(DEV)
    one = dict(one_tile_per_cta=True, force_splits=1)
    got = ops.linear(act, w, out_f32=True)
    assert torch.equal(got, ops.linear(act, w, out_f32=True, **one))
    want = ops.linear(act, w, residual=res, **one)
    assert torch.equal(ops.linear(act, w, residual=res), want)
    wide = torch.full((M, N + 3), 7.0, dtype=torch.bfloat16, device=DEV)
    wide[:, :N] = res
    ops.linear(act, w, residual=wide[:, :N], out=wide[:, :N])                   # in place, rows of a wider matrix
    assert torch.equal(wide[:, :N], want) and bool((wide[:, N:] == 7).all())
    if N % 2 == 0 and fmt != "fp8_block":
        glu, other = ops.linear(act, w, swiglu=True), ops.linear(act, w, swiglu=True, **one)
        assert glu.shape[1] == N // 2 and (glu.float() - other.float()).abs().max() <= 2.0 ** -7 * other.float().abs().max()
    ops.check_status(DEV)
    exact = _oracle(x, w_cpu, fmt)
    assert (got.cpu().double() - exact).norm() <= 1e-5 * exact.norm()


@pytest.mark.parametrize("M", [129, 300])
def test_pair_kernel_epilogues(M):
    N, K = 9600, 256
    x, w_cpu, act, w = _operands("bf16", M, N, K, 5)
    bias = torch.randn(N, generator=torch.Generator().manual_seed(2))
    cpu = ops.encode_act_ref(x.float(), "bf16")
    for kw in (dict(swiglu=True), dict(geglu=True), dict(clamp_glu=(1.7, 0.4)), dict(silu_cols=1000), dict(relu2=True), dict(bias=bias),
               dict(log_sigmoid=(bias, 0.5)), dict(sigmoid=(bias, 2.0))):
        on = {k: v.to(DEV) if torch.is_tensor(v) else (v[0].to(DEV), v[1]) if isinstance(v, tuple) and torch.is_tensor(v[0]) else v
              for k, v in kw.items()}
        got, want = ops.linear(act, w, **on), ops.linear(cpu, w_cpu, out_f32=True, **kw)
        # bf16 results: half an ulp is 2^-9 of the value; the rest are the epilogue's approximate functions
        assert (got.cpu().float() - want).abs().max() <= 2.0 ** -8 * want.abs().max(), kw
    ops.check_status(DEV)


@pytest.mark.parametrize("fmt", ["nvfp4", "bf16"])
@pytest.mark.parametrize("M,N", [(129, 512), (300, 1024), (257, 10240)])
def test_pair_kernel_quantises_the_swiglu_result(fmt, M, N):
    """Against the row kernel on the same fp32-close values: the encoded rows differ only where a value sits on a rounding edge,
    so the decoded matrices agree to the bf16 rounding that the row kernel's input went through (2^-8 of an e2m1 step's range)."""
    x, w_cpu, act, w = _operands(fmt, M, N, 512, 7)
    y = ops.linear(act, w, swiglu=True)
    gs = 2 * float(y.float().abs().max()) / 2688
    got, want = ops.linear(act, w, swiglu=True, quant_out=gs), ops.quantize_act(y, "nvfp4", static_scale=gs)
    ops.check_status(DEV)

    def values(a):
        sf = ref.tiled_to_sf(a.sf.cpu().view(-1, a.sf_k64, 512), M, a.K // 16)
        return ref.dequantize_nvfp4(a.data.cpu(), sf, a.scale[:M].cpu())
    g, v = values(got), values(want)
    assert (g != v).float().mean() < 0.02
    exact = ops.linear(ops.encode_act_ref(x.float(), ops.ACT_FOR_WEIGHT[fmt]), w_cpu, swiglu=True, out_f32=True)
    assert (g - exact).norm() <= 1.01 * (v - exact).norm()


@pytest.mark.parametrize("M,N,K", [(65, 128, 128), (127, 256, 384), (128, 384, 1024), (129, 136, 1024), (300, 1024, 640), (5000, 256, 256),
                                   (5000, 2176, 384), (5000, 2100, 256)])       # the last two: 256 features a tile, a last half and a last row block missing
def test_block_kernel_matches_the_one_tile_kernel_and_the_oracle(M, N, K):
    x, w_cpu, act, w = _operands("fp8_block", M, N, K, 9)
    res = torch.randn(M, N, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).to(DEV)
    got = ops.linear(act, w, out_f32=True)
    assert torch.equal(got, ops.linear(act, w, out_f32=True, one_tile_per_cta=True, force_splits=1))
    assert torch.equal(ops.linear(act, w, residual=res), ops.linear(act, w, residual=res, one_tile_per_cta=True, force_splits=1))
    ops.check_status(DEV)
    want = _oracle(x, w_cpu, "fp8_block")
    assert (got.cpu().double() - want).norm() <= 1e-5 * want.norm()


@pytest.mark.parametrize("tile_rows", [16, 32, 64, 128])
def test_block_kernel_over_a_work_list_of_experts(tile_rows):
    """Experts with no row, one row, a whole tile, one more than a tile; pairs of experts that are not here."""
    E, N, K = 6, 384, 512
    g = torch.Generator().manual_seed(tile_rows)
    counts = [0, 1, tile_rows, tile_rows + 1, 3 * tile_rows - 1, 5]
    ids = torch.cat([torch.full((n,), e) for e, n in enumerate(counts)] + [torch.full((7,), -1)])
    ids = ids[torch.randperm(len(ids), generator=g)].to(torch.int32)
    T = len(ids)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16)
    w = ops.make_weight(torch.randn(E * N, K, generator=g) * 0.05, "fp8_block")
    act = ops.quantize_act(x.to(DEV), "fp8_g128")
    sp = moe_cuda.SortedPairs(ids.to(DEV).view(T, 1), 0, E, tile_rows)
    y = ops.linear(moe_cuda.gather_act(act, sp), w.to(DEV), out_f32=True, grouped=(sp.tile_expert, sp.tile_row0, sp.tile_nrows, N, sp.max_tiles, tile_rows))
    ops.check_status(DEV)
    a, d, at = ops.encode_act_ref(x.float(), "fp8_g128").data.double(), w.dequant().double(), sp.pair_row.cpu()
    for i in range(T):
        e = int(ids[i])
        assert (int(at[i]) < 0) == (e < 0)
        if e >= 0:
            want = d[e * N:(e + 1) * N] @ a[i]
            assert (y[int(at[i])].cpu().double() - want).norm() <= 1e-5 * want.norm()
