"""The batched radix sort at the edges of its forms: one pair, part of a warp, a tile and one more, the largest batch of the
one-launch form and one more, several tiles per block; key ranges of one, two and three passes.  Checked through what it
is for: the SGD scatter (gradients are small whole numbers and lr is 1, so every sum is exact whatever its order) and the
sketch insert (which meets the ids of a bucket in batch order, or ends in another state than the sequential oracle)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SIZES = [1, 31, 33, 4096, 4097, 131072, 131073, 1300001]


@pytest.mark.parametrize("hash_rows", [300, 60_000, 1_200_000])
@pytest.mark.parametrize("n", SIZES)
def test_scatter_sums_every_row(n, hash_rows):
    import torch
    from cafe_b200 import HotSketch
    from cafe_b200.sk_embedding_bag import _FieldSet
    D, hot = 16, 500
    g = torch.Generator(device="cuda").manual_seed(n + hash_rows)
    high = torch.zeros(hot, D, device="cuda")
    cold = torch.zeros(hash_rows, D, device="cuda")
    sk = HotSketch(hot, max_lookups=n)
    fs = _FieldSet(sk, high, [cold], [0], [hash_rows], D)
    # a third of the lookups in a few hot rows, the others spread over all hash rows
    pick = torch.rand(n, device="cuda", generator=g)
    row = torch.randint(0, hash_rows, (n,), device="cuda", generator=g, dtype=torch.int32)
    row = torch.where(pick < 0.33, -torch.randint(1, hot, (n,), device="cuda", generator=g, dtype=torch.int32) // 50 - 1, row)
    grad = torch.randint(-3, 4, (n, D), device="cuda", generator=g).float()
    fs.scatter_sgd(grad, 0, D, row, n, 1.0)
    want_h, want_c = torch.zeros_like(high), torch.zeros_like(cold)
    want_h.index_add_(0, torch.where(row < 0, -row, 0).long(), torch.where(row[:, None] < 0, -grad, 0 * grad))
    want_c.index_add_(0, torch.where(row < 0, 0, row).long(), torch.where(row[:, None] < 0, 0 * grad, -grad))
    assert torch.equal(high, want_h) and torch.equal(cold, want_c)


@pytest.mark.parametrize("lim", [40, 3000, 200_000])
@pytest.mark.parametrize("n", [1, 33, 4097, 131073])
def test_insert_meets_ids_in_batch_order(n, lim):
    from sketch_driver import drive
    from test_gpu_sketch import GpuSketch
    drive(lambda lim, thr, adj, alpha, cap, par: GpuSketch(lim, thr, adj, alpha, cap, par), lim, 1, 1.0000005, 2, n, max(20, 2 * lim), 1)
