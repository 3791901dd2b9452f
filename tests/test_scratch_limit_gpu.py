"""Products and closures on a device that has no room for the 16-bit codes beside
the FP32 operand copies: they run without codes, with the same bits."""
import pytest
import torch

import simd2_b200 as s2

pytestmark = pytest.mark.gpu


@pytest.fixture
def leave(cuda):
    """leave(bytes): takes device memory until about that much is free."""
    held = []

    def take(free):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        assert s2.lib().simd2_release_workspaces() == 0
        held.append(torch.empty(max(0, torch.cuda.mem_get_info()[0] - free), dtype=torch.uint8, device="cuda"))

    yield take
    held.clear()
    torch.cuda.empty_cache()
    assert s2.lib().simd2_release_workspaces() == 0


def graph(n, gen):
    x = torch.where(torch.rand((n, n), generator=gen, device="cuda") < 0.002,
                    torch.randint(1, 101, (n, n), generator=gen, device="cuda").float(),
                    torch.full((), float("inf"), device="cuda"))
    return x.fill_diagonal_(0.0)


@pytest.mark.parametrize("op", ["min_plus", "max_min"])
def test_product(leave, op):
    n = 8192  # FP32 copy of B 256 MiB, codes of A and B 128 MiB each
    gen = torch.Generator(device="cuda").manual_seed(1)
    a, b = (torch.randint(0, 1000, (n, n), generator=gen, device="cuda").float() for _ in range(2))
    want = s2.srgemm(op, a, b)
    got = torch.empty_like(want)
    tuned = torch.empty_like(want)
    leave(430 << 20)
    s2.srgemm(op, a, b, D=got)
    s2.lib().simd2_release_workspaces()
    s2.srgemm_tuned(op, a, b, config=0, D=tuned)
    assert torch.equal(got, want) and torch.equal(tuned, want)
    assert s2.device_status() == 0


@pytest.mark.parametrize("kw", [{"dispatch": "dense"}, {"dispatch": "rules", "config": 4}])
def test_closure(leave, kw):
    n = 6144  # FP32 copy of B and the other X 144 MiB each, codes as much together
    gen = torch.Generator(device="cuda").manual_seed(2)
    x = graph(n, gen)
    want, got = x.clone(), x.clone()
    steps = s2.closure_ex("min_plus", want, **kw)
    if kw["dispatch"] == "rules":  # the sparse opening's store, of the same size, stays out of it
        kw = {**kw, "conv": "tol"}
    leave(400 << 20)
    assert s2.closure_ex("min_plus", got, **kw) == steps
    assert torch.equal(got, want)
    assert s2.device_status() == 0
