"""What the launchers refuse before they touch a device, called through the library's C entry points."""
import ctypes as C

import pytest
import torch

from metrale_inference_alpha_b200 import ops
from metrale_inference_alpha_b200.ops import _native

BAD_ARG, UNSUPPORTED = -1, -2


@pytest.fixture(scope="module")
def lib():
    if not _native.LIB_PATH.exists():
        pytest.skip("kernel library not built")
    L = C.CDLL(str(_native.LIB_PATH))
    L.mb_gemm.argtypes, L.mb_gemm.restype = [C.POINTER(_native.GemmArgs), C.c_void_p], C.c_int
    return L


@pytest.mark.parametrize("fmt,rows", [("bf16", 128), ("fp8_row", 128), ("fp8_block", 128)])
@pytest.mark.parametrize("flags,no_cluster,epilogue", [(ops.GEMM_ONE_TILE_PER_CTA, 0, 0), (ops.GEMM_DECODE_TILE_ORDER, 0, 0), (0, 1, 0),
                                                       (0, 0, ops.EPI_SWIGLU)])
def test_a_work_list_entry_has_no_more_rows_than_the_tile(lib, fmt, rows, flags, no_cluster, epilogue):
    buf = torch.zeros(1 << 20, dtype=torch.uint8)
    p = buf.data_ptr()
    a = _native.GemmArgs()
    a.kind, a.M, a.N, a.K, a.ldo, a.a_ld = ops.KIND[fmt], 512, 1024, 128, 256, 512 + rows
    a.W = a.X = a.out = a.w_scale = a.a_scale = a.tile_expert = a.tile_row0 = a.tile_nrows = p
    a.alpha, a.n_per_expert, a.max_tiles, a.force_tn, a.sm_count = 1.0, 256, 8, rows, 148
    a.flags, a.no_cluster, a.epilogue = flags | ops.GEMM_PERSISTENT_PREFILL, no_cluster, epilogue
    assert lib.mb_gemm(C.byref(a), None) == UNSUPPORTED


def test_splits_of_k_keep_their_clusters_resident(lib):
    """No cluster beyond what the chip holds at once (measured: 74, 45, 33, 26, 22, 15, 15 of 2 to 8 CTAs), no split without four k blocks."""
    lib.mb_gemm_auto_splits.argtypes, lib.mb_gemm_auto_splits.restype = [C.c_int, C.c_int, C.c_int, C.c_bool], C.c_int
    held = {1: 148, 2: 74, 3: 45, 4: 33, 5: 26, 6: 22, 7: 15, 8: 15}
    for tiles in range(1, 200):
        for num_kb in (1, 4, 11, 20, 80):
            s = lib.mb_gemm_auto_splits(tiles, num_kb, 148, True)
            want = max((n for n in held if tiles <= held[n] and n * tiles <= 148 and (n == 1 or 4 * n <= num_kb)), default=1)
            assert s == want, (tiles, num_kb)
            assert lib.mb_gemm_auto_splits(tiles, num_kb, 148, False) == max(1, min(148 // tiles, num_kb // 4))


@pytest.mark.parametrize("D,most", [(128, 3), (256, 1)])
def test_decode_attention_launches_only_resident_ctas(lib, D, most):
    """Shared memory beside the ring grows with rows and batch: 228 KB an SM, a kilobyte of it a block's own."""
    lib.mb_attn_decode_per_sm.argtypes, lib.mb_attn_decode_per_sm.restype = [C.c_int] * 4 + [C.POINTER(C.c_size_t)], C.c_int
    seen = set()
    for fp8 in (0, 1):
        for rows in range(1, 33 if D == 128 else 17):
            for seqs in (1, 64, 128, 512, 1024):
                smem = C.c_size_t()
                n = lib.mb_attn_decode_per_sm(D, fp8, rows, seqs, C.byref(smem))
                assert n * (smem.value + 1024 + 256) <= 228 * 1024 and smem.value <= 220 * 1024, (fp8, rows, seqs)
                assert n == (2 if rows > 16 else most) or (n + 1) * (smem.value + 1024) > 227 * 1024, (fp8, rows, seqs)
                seen.add(n)
    assert seen == ({1, 2, 3} if D == 128 else {1})
