"""The tiled interaction kernels at the edges of their tiles and in every form the entry points take: vector counts around
multiples of seven, dimensions that fill the lanes partly, field-major and padded layouts, rows that are not on 16-byte
boundaries (which take the general kernels), partial last groups.  Oracle: the same sums in fp64.  A sum of n fp32 products
added in any order is off by at most n * 2^-23 times the sum of the products' magnitudes (n roundings of half an ulp, and
the product's own), which is the bound used, element by element."""
import pytest

pytestmark = pytest.mark.gpu


def _strided(B, F, D, layout, shift, gen):
    """[B, F, D] values in a buffer of the given layout; returns the values, the buffer, its address and both strides."""
    import torch
    v = torch.randn(B, F, D, device="cuda", generator=gen)
    fs, ss = {"sample": (D, F * D), "field": (B * D, D), "padded": (D + 4, F * (D + 4) + 8)}[layout]
    buf = torch.full((shift + (B - 1) * ss + (F - 1) * fs + D + 8,), float("nan"), device="cuda")
    buf[shift:].as_strided((B, F, D), (ss, fs, 1)).copy_(v)
    return v, buf, buf.data_ptr() + 4 * shift, fs, ss


@pytest.mark.parametrize("layout,shift", [("sample", 0), ("field", 0), ("padded", 0), ("sample", 1)])
@pytest.mark.parametrize("B,F,D,dense,itself", [
    (1, 1, 4, True, 0), (3, 6, 16, True, 1), (150, 7, 16, False, 0), (149, 13, 32, True, 0), (5, 14, 12, False, 1),
    (600, 20, 64, True, 0), (31, 26, 128, True, 1), (450, 27, 128, False, 0), (9, 32, 100, True, 0), (70, 63, 64, True, 0),
    (4, 62, 128, True, 0), (33, 26, 20, True, 0), (1000, 3, 16, True, 0), (77, 2, 36, False, 0), (1, 26, 17, True, 0)])
def test_every_form_against_fp64(B, F, D, dense, itself, layout, shift):
    import torch
    from cafe_b200 import _lib
    lib = _lib.load()
    gen = torch.Generator(device="cuda").manual_seed(B * 31 + F * 7 + D)
    emb, ebuf, ep, fs, ss = _strided(B, F, D, layout, shift, gen)
    x = torch.randn(B, D, device="cuda", generator=gen) if dense else None
    T = (emb if x is None else torch.cat([x.unsqueeze(1), emb], 1)).double()
    nv = T.shape[1]
    lead = D if dense else 0
    li, lj = torch.tril_indices(nv, nv, offset=0 if itself else -1, device="cuda")
    n = li.numel()
    stride = lead + n + 3
    st = torch.cuda.current_stream().cuda_stream
    xp = None if x is None else x.data_ptr()
    out = torch.full((B, stride), 7.0, device="cuda")
    _lib.check(lib.cafe_dot_interaction_forward(xp, ep, fs, ss, B, F, D, itself, out.data_ptr(), stride, st), "forward")
    want = torch.bmm(T, T.transpose(1, 2))[:, li, lj]
    room = torch.bmm(T.abs(), T.abs().transpose(1, 2))[:, li, lj] * D * 2.0 ** -23
    assert bool(((out[:, lead:lead + n].double() - want).abs() <= room).all())
    assert bool((out[:, lead + n:] == 7.0).all())
    if dense:
        assert torch.equal(out[:, :D], x)
    # backward: every vector's gradient is the incoming row, as a symmetric matrix with a doubled diagonal, times the vectors
    g = torch.randn(B, stride, device="cuda", generator=gen)
    gbuf = torch.full_like(ebuf, 3.0)
    gx = None if x is None else torch.full_like(x, 3.0)
    _lib.check(lib.cafe_dot_interaction_backward(xp, ep, fs, ss, B, F, D, itself, g.data_ptr(), stride,
                                                 None if gx is None else gx.data_ptr(), gbuf.data_ptr() + 4 * shift, fs, ss, st), "backward")
    W = torch.zeros(B, nv, nv, device="cuda", dtype=torch.float64)
    W[:, li, lj] = g[:, lead:lead + n].double()
    W = W + W.transpose(1, 2)
    want = torch.bmm(W, T)
    size = torch.bmm(W.abs(), T.abs())
    if dense:
        want[:, 0] += g[:, :D].double()
        size[:, 0] += g[:, :D].double().abs()
    room = size * (nv + 1) * 2.0 ** -23
    view = gbuf[shift:].as_strided((B, F, D), (ss, fs, 1))
    assert bool(((view.double() - want[:, nv - F:]).abs() <= room[:, nv - F:]).all())
    if dense:
        assert bool(((gx.double() - want[:, 0]).abs() <= room[:, 0]).all())
    written = torch.zeros_like(gbuf)
    written[shift:].as_strided((B, F, D), (ss, fs, 1)).fill_(1.0)
    assert bool((gbuf[written == 0] == 3.0).all())      # nothing beside the rows


@pytest.mark.parametrize("backward", [False, True])
def test_threads_with_different_sizes(backward):
    """Threads whose calls share a kernel but want different amounts of shared memory, all above the default limit: every call
    is taken, and the results are those of the same calls made alone."""
    import threading
    import torch
    from cafe_b200 import _lib
    lib = _lib.load()
    B, D, rounds, workers = 1, 128, 10_000, 8
    calls, alone = [], []
    for k in range(workers):
        F = (50, 40)[k % 2] if backward else (62, 45)[k % 2]
        gen = torch.Generator(device="cuda").manual_seed(k)
        x, emb, g = (torch.randn(*s, device="cuda", generator=gen) for s in ((B, D), (B, F, D), (B, D + (F + 1) * F // 2)))
        out = [torch.empty_like(x), torch.empty_like(emb)] if backward else [torch.empty_like(g)]
        args = (x.data_ptr(), emb.data_ptr(), D, F * D, B, F, D, 0)
        if backward:
            fn, args = lib.cafe_dot_interaction_backward, args + (g.data_ptr(), g.shape[1], out[0].data_ptr(), out[1].data_ptr(), D, F * D)
        else:
            fn, args = lib.cafe_dot_interaction_forward, args + (out[0].data_ptr(), g.shape[1])
        calls.append((fn, args, out, (x, emb, g)))
        _lib.check(fn(*args, torch.cuda.current_stream().cuda_stream), "alone")
        alone.append([t.clone() for t in out])
        for t in out:
            t.zero_()
    torch.cuda.synchronize()
    refused = [0] * workers

    def work(k):
        stream = torch.cuda.Stream()
        fn, args, _, _ = calls[k]
        for _ in range(rounds):
            refused[k] += fn(*args, stream.cuda_stream) != _lib.OK
        stream.synchronize()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(workers)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert refused == [0] * workers
    for k in range(workers):
        assert all(torch.equal(u, v) for u, v in zip(alone[k], calls[k][2]))
