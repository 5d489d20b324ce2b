"""Sorting up to 1024 pairs by expert, one a thread: at the line and on both sides of it."""
import pytest

from test_expert_sort_gpu import test_pairs_sorted_by_expert as _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,K", [(2, 1), (128, 8), (205, 5), (114, 9)])      # 2, 1024, 1025 and 1026 pairs
@pytest.mark.parametrize("align,tile_rows,lo,E", [(1, 64, 0, 257), (128, 32, 3, 64)])
def test_few_pairs_sorted_by_expert(T, K, align, tile_rows, lo, E):
    _check(T, K, align, tile_rows, lo, E)
