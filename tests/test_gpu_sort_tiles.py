"""The one-launch radix sort where every block has at most a tile of pairs (read once per pass and ranked without a histogram
step; the blocks of a cluster exchange their counts), around the sizes where the number of blocks or the form changes; keys of
one, two and three passes.  Same checks as the sort's other sizes: exact scatter sums, and the sequential insert's state."""
import pytest

from test_gpu_sort_edges import test_insert_meets_ids_in_batch_order as _insert
from test_gpu_sort_edges import test_scatter_sums_every_row as _scatter

pytestmark = pytest.mark.gpu
SIZES = [2, 511, 513, 2048, 2049, 4095, 8191, 8193, 16385, 32767, 32768, 32769]


@pytest.mark.parametrize("hash_rows", [2, 300, 60_000, 1_200_000])
@pytest.mark.parametrize("n", SIZES)
def test_scatter_sums(n, hash_rows):
    _scatter(n, hash_rows)


@pytest.mark.parametrize("lim", [40, 3000, 200_000])
@pytest.mark.parametrize("n", [513, 2048, 2049, 4096, 16385, 32769])
def test_insert_order(n, lim):
    _insert(n, lim)
