"""or_and operands packed to FP4: tile edges, and closures whose delta steps pack again only what changed."""

import pytest
import torch

import simd2_b200 as s2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (31, 129, 33), (130, 255, 257), (256, 128, 256), (300, 127, 511)])
@pytest.mark.parametrize("dtype", [torch.uint8, torch.int32])
def test_products_at_tile_edges(cuda, shape, dtype):
    m, n, k = shape
    g = torch.Generator(device=cuda).manual_seed(m + n + k)
    a = (torch.rand((m, k), generator=g, device=cuda) < 0.03).to(dtype) * 5
    b = (torch.rand((k, n), generator=g, device=cuda) < 0.03).to(dtype) * 3
    want = ((a != 0).float() @ (b != 0).float() > 0).to(dtype)
    got = s2.srgemm("or_and", a, b, do_epilogue=False)
    assert torch.equal(got, want)
    # one matrix as both operands, and a view whose rows are not 16-byte aligned
    sq = torch.zeros((k + 1, k + 1), dtype=dtype, device=cuda)
    sq[1:, 1:] = (torch.rand((k, k), generator=g, device=cuda) < 0.03).to(dtype)
    for x in (sq, sq[1:, 1:]):
        want = ((x != 0).float() @ (x != 0).float() > 0).to(dtype)
        assert torch.equal(s2.srgemm("or_and", x, x, do_epilogue=False), want)


@pytest.mark.parametrize("n", [2000, 2048, 3137])
@pytest.mark.parametrize("tail", [0, 40, 300])
def test_closure_delta_steps(cuda, n, tail):
    """A dense part that settles early and a path that keeps a few tiles changing:
    the closure is that of the whole graph, from the same number of steps."""
    g = torch.Generator(device=cuda).manual_seed(n + tail)
    x = torch.zeros((n, n), dtype=torch.uint8, device=cuda)
    h = n // 2
    x[:h, :h] = torch.rand((h, h), generator=g, device=cuda) < 4.0 / h
    at = torch.arange(n - max(tail, 1), n - 1, device=cuda)
    x[at, at + 1] = 1
    x.fill_diagonal_(1)
    want, steps = x.clone(), 0
    while True:
        f = want.half()
        y = ((f @ f > 0) | (want != 0)).to(torch.uint8)
        steps += 1
        if torch.equal(y, want):
            break
        want = y
    got = x.clone()
    it = s2.closure("or_and", got)
    assert torch.equal(got, want) and it == steps


@pytest.mark.parametrize("max_iter", [3, 8, 9, 500])
@pytest.mark.parametrize("n,ld,shift", [(1, 1, 0), (150, 150, 0), (700, 707, 3), (2100, 2112, 1)])
def test_closure_in_place_and_chunked(cuda, n, ld, shift, max_iter):
    """or_and closures squared in place, their steps enqueued in chunks of eight: a
    chain takes more steps than a chunk holds; the step limit inside, at and past a
    chunk's end; pitched and unaligned rows, single-SM and SM-pair kernel."""
    buf = torch.full((n * ld + 16,), 7, dtype=torch.uint8, device=cuda)
    X = buf[shift:shift + n * ld].view(n, ld)[:, :n]
    X.zero_()
    i = torch.arange(n - 1, device=cuda)
    X[i, i + 1] = 1
    want, steps, changed = X.float(), 0, True
    while changed and steps < max_iter:
        nxt = torch.maximum(want, (want @ want > 0).float())
        changed = not torch.equal(nxt, want)
        want, steps = nxt, steps + 1
    if changed:
        with pytest.raises(s2.Simd2Error):
            s2.closure("or_and", X, max_iter=max_iter)
    else:
        assert s2.closure("or_and", X, max_iter=max_iter) == steps
    assert torch.equal(X, want.to(torch.uint8))
    pad = buf[shift:shift + n * ld].view(n, ld)[:, n:]
    assert bool((pad == 7).all()) and bool((buf[shift + n * ld:] == 7).all())
    assert s2.device_status() == 0
