"""Several threads closing graphs on streams of their own at once: small closures
(one cooperative launch each, page-locked words lent out), batches and products,
each against the same call made alone."""
import threading

import pytest
import torch

import simd2_b200 as s2

pytestmark = pytest.mark.gpu


def graph(n, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randint(1, 101, (n, n), generator=gen, device="cuda").float()
    x = torch.where(torch.rand((n, n), generator=gen, device="cuda") < 8.0 / n, w, torch.full_like(w, float("inf")))
    return x.fill_diagonal_(0.0)


def run(jobs, rounds):
    """Each job (its own thread and stream) is run `rounds` times; returns the errors."""
    errors = []

    def loop(job):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for _ in range(rounds):
                    job()
                stream.synchronize()
        except Exception as e:  # shown by the caller
            errors.append(repr(e))

    threads = [threading.Thread(target=loop, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return errors


def closing(n, seed):
    x = graph(n, seed)
    want = x.clone()
    steps = s2.closure("min_plus", want)
    torch.cuda.synchronize()

    def job():
        X = x.clone()
        assert s2.closure("min_plus", X) == steps
        assert torch.equal(X, want)

    return job


def test_small_closures(cuda):
    sizes = [512, 1000, 300, 64, 1400]
    assert run([closing(n, i) for i, n in enumerate(sizes)], 25) == []
    assert s2.device_status() == 0


def test_closures_batches_and_products(cuda):
    mats = [graph(n, 50 + n) for n in (40, 200, 300, 700, 90, 128)]
    want = [m.clone() for m in mats]
    steps = [s2.closure("min_plus", w) for w in want]
    a, b = graph(900, 1), graph(900, 2)
    prod = s2.srgemm("min_plus", a, b)
    torch.cuda.synchronize()

    def batch():
        X = [m.clone() for m in mats]
        assert list(s2.closure_batched("min_plus", X)) == steps
        assert all(torch.equal(x, w) for x, w in zip(X, want))

    def product():
        assert torch.equal(s2.srgemm("min_plus", a, b), prod)

    assert run([closing(512, 7), batch, product, closing(900, 8)], 25) == []
    assert s2.device_status() == 0
