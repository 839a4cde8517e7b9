"""Counting sort of routed rows on both sides of the line between one CTA and a cluster."""
import pytest

from tests import test_gpu_sort_rows as rows_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [4080, 4095, 4096, 4097, 4113])
@pytest.mark.parametrize("experts", [8, 1500])
@pytest.mark.parametrize("bad", [False, True])
def test_sorted_order(gpu_ctx, rows, experts, bad):
    rows_of.test_sorted_order(gpu_ctx, rows, experts, 64, bad)
