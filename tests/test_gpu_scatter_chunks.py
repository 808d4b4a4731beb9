"""The SGD scatter at the edges of its chunks and of the fix-up: calls of less than a chunk, around a multiple of it, the largest
call that takes short chunks and one more; rows that end with a chunk, go on for one, for as many as one group adds up and
one more, and one row for the whole call.  Gradients are small whole numbers and lr is 1, so every sum is exact whatever
its order (below 2^24)."""
import pytest

pytestmark = pytest.mark.gpu


def _run_lengths(kind, n, gen):
    import torch
    if kind == "one":
        return [n]
    if kind == "edges":     # lengths around multiples of 8 and 32, up to more than 16 chunks of 32
        want = [1, 7, 8, 9, 31, 32, 33, 120, 128, 129, 136, 137, 512, 544, 545, 576, 577, 2]
    else:                   # a head of long rows, then short ones
        want = [n // 3, n // 7, n // 20] + torch.randint(1, 40, (n,), generator=gen).tolist()
    out, left, i = [], n, 0
    while left > 0:
        k = max(1, min(left, want[i % len(want)]))
        out.append(k)
        left -= k
        i += 1
    return out


@pytest.mark.parametrize("D", [16, 32, 64, 128])
@pytest.mark.parametrize("kind", ["one", "edges", "heads"])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 257, 5000, 131072, 131073])
def test_sums_of_rows_of_every_length(n, kind, D):
    import torch
    from cafe_b200 import HotSketch
    from cafe_b200.sk_embedding_bag import _FieldSet
    gen = torch.Generator().manual_seed(n + D)
    lengths = _run_lengths(kind, n, gen)
    rows = len(lengths)
    hot = 4
    row = torch.repeat_interleave(torch.arange(rows), torch.tensor(lengths))[torch.randperm(n, generator=gen)].to(torch.int32).cuda()
    row = torch.where(row < hot - 1, -(row + 1), row)     # the first three rows are hot rows 1..3
    grad = torch.randint(-3, 4, (n, D), generator=gen).float().cuda()
    cold = torch.zeros(max(rows, 1), D, device="cuda")
    sk = HotSketch(500, max_lookups=n)
    high = torch.zeros(500, D, device="cuda")
    _FieldSet(sk, high, [cold], [0], [max(rows, 1)], D).scatter_sgd(grad, 0, D, row, n, 1.0)
    want_h, want_c = torch.zeros_like(high), torch.zeros_like(cold)
    is_hot = row < 0
    want_h.index_add_(0, -row[is_hot].long(), -grad[is_hot])
    want_c.index_add_(0, row[~is_hot].long(), -grad[~is_hot])
    assert torch.equal(high, want_h) and torch.equal(cold, want_c)


def test_small_handles_hold_little_memory():
    """Workspaces are sized for the calls a handle was made for: sketches of 1000 rows and 2048 lookups, whose arrays add up to
    about 1 MB (one-stage: 0.2 MB), take no more than one of the driver's granules of 2 MiB each (one-stage sketches share them)."""
    import torch
    from cafe_b200 import HotSketch
    from cafe_b200.sigmod import SigmodSketch
    for make, granules in ((lambda: HotSketch(1000, max_lookups=2048), 32), (lambda: SigmodSketch(1000, 1, max_lookups=2048), 8)):
        first = make()
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        held = [make() for _ in range(32)]
        torch.cuda.synchronize()
        assert before - torch.cuda.mem_get_info()[0] <= granules * 2**21
        del held, first
