"""plus_mul and minus_square on the tensor cores (N-major B, tile widths 64..256,
single SMs and SM pairs, FP32 and float16 operands) and or_and on float16, at the
edges of tiles, k-tiles and alignment, against the FP64 oracle.

Bounds.  FP32 operands: the BF16 hi / lo split's, |D - D64| <= (4 * 2^-16 +
2 K 2^-24) S with S the sum of the terms' magnitudes.  Float16 operands: every
product is exact in FP32, so only the FP32 sums round: at most one rounding of
2^-24 a term and the accumulator, (2 K + 8) * 2^-24 S (8 for the norms, the final
combination and C).
"""
import numpy as np
import pytest
import torch

import oracle
import simd2_b200 as s2

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24
SHAPES = [(1, 1, 1), (128, 64, 64), (129, 65, 65), (127, 191, 63), (300, 193, 130), (70, 700, 17), (1000, 800, 200),
          (64, 4100, 96), (2100, 2049, 70)]


def operands(m, n, k, dtype, seed, offset=0):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def place(r, c, dt):
        x = torch.randn((r, c), generator=g, device="cuda").to(dt)
        buf = torch.full((r, c + offset + (offset and 5)), float("nan"), device="cuda", dtype=dt)
        buf[:, offset:offset + c] = x
        return buf[:, offset:offset + c]
    return place(m, k, dtype), place(k, n, dtype), place(m, n, torch.float32)


def check(op, a, b, c, got, half):
    a64, b64 = a.double().cpu().numpy(), b.double().cpu().numpy()
    want = oracle.srgemm_f64(op, a64.astype(np.float32), b64.astype(np.float32), c.cpu().numpy(), do_epilogue=True)
    if op == "plus_mul":
        s = np.abs(a64) @ np.abs(b64)
    else:
        s = 2 * (a64 ** 2).sum(1)[:, None] + 2 * (b64 ** 2).sum(0)[None, :]
    s = s + np.abs(c.double().cpu().numpy())
    k = a.shape[1]
    rel = (2 * k + 8) * EPS if half else 4 * 2.0 ** -16 + 2 * k * EPS
    err = np.abs(got.double().cpu().numpy() - want)
    assert np.all(err <= rel * s + 1e-30), f"{op}: worst ratio {(err / (rel * s + 1e-30)).max():.3f}"


@pytest.mark.parametrize("op", ["plus_mul", "minus_square"])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("half", [False, True])
def test_shapes(cuda, op, shape, half):
    m, n, k = shape
    for offset in (0, 1):  # rows on the 16-byte grid where the size allows, and off it
        a, b, c = operands(m, n, k, torch.float16 if half else torch.float32, m + n + k, offset)
        f = s2.srgemm_f16 if half else s2.srgemm
        check(op, a, b, c, f(op, a, b, c, do_epilogue=True), half)
    assert s2.device_status() == 0


@pytest.mark.parametrize("half", [False, True])
def test_near_duplicate_points(cuda, half):
    """Distances in the cancellation band are recomputed from the operands: equal
    points give exactly 0, a change of one unit in one coordinate its square."""
    g = torch.Generator(device="cuda").manual_seed(4)
    a = torch.randint(-8, 9, (200, 96), generator=g, device="cuda").float() + 30.0
    b = a.t().contiguous()
    b[5, 7] += 1.0
    dt = torch.float16 if half else torch.float32
    f = s2.srgemm_f16 if half else s2.srgemm
    d = f("minus_square", a.to(dt), b.to(dt))
    diag = torch.diagonal(d)
    assert diag[7] == 1.0
    assert torch.all(diag[torch.arange(200, device="cuda") != 7] == 0.0)


@pytest.mark.parametrize("shape", [(1, 1, 1), (130, 225, 257), (100, 448, 31), (2050, 2300, 100)])
@pytest.mark.parametrize("offset", [0, 1])
def test_or_and_f16(cuda, shape, offset):
    m, n, k = shape
    a, b, c = operands(m, n, k, torch.float16, 3, offset)
    for x, keep in ((a, 0.05), (b, 0.05), (c, 0.02)):
        x[torch.rand(x.shape, device="cuda") >= keep] = -0.0  # a negative zero is false
    got = s2.srgemm_f16("or_and", a, b, c, do_epilogue=True)
    want = ((a != 0).float() @ (b != 0).float() > 0) | (c != 0)
    assert torch.equal(got, want.float())


@pytest.mark.parametrize("op", ["min_plus", "max_plus", "max_min", "min_max", "max_mul", "min_mul"])
@pytest.mark.parametrize("offset", [0, 1])
def test_minmax_f16(cuda, op, offset):
    """Integers (coded) and fractions (FP32) through the float16 entry."""
    m, n, k = 130, 77, 100
    g = torch.Generator(device="cuda").manual_seed(5)
    for scale in (1.0, 0.25 if op.endswith("plus") else 1.0 / 1024):
        a, b, c = operands(m, n, k, torch.float16, 6, offset)
        a.copy_(torch.randint(1, 1001, a.shape, generator=g, device="cuda").float() * scale)
        b.copy_(torch.randint(1, 1001, b.shape, generator=g, device="cuda").float() * scale)
        got = s2.srgemm_f16(op, a, b, c, do_epilogue=True).cpu().numpy()
        want = oracle.srgemm(op, a.float().cpu().numpy(), b.float().cpu().numpy(), c.contiguous().cpu().numpy(),
                             do_epilogue=True)
        np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("op", ["plus_mul", "minus_square"])
@pytest.mark.parametrize("shape", [(64, 64, 128), (65, 63, 129), (1, 1, 2500), (200, 201, 1000), (500, 500, 2000),
                                   (1000, 131, 700), (63, 1030, 5000), (1000, 800, 900)])
@pytest.mark.parametrize("half", [False, True])
def test_split_k(cuda, op, shape, half):
    """Few tiles: the CTAs of a cluster share a tile's k.  Some rows of A are columns
    of B, whose distances lie in the cancellation band."""
    m, n, k = shape
    for offset in (0, 1):
        a, b, c = operands(m, n, k, torch.float16 if half else torch.float32, m + n + k, offset)
        a[::9] = b[:, : len(a[::9])].T[: len(a[::9])] if n >= len(a[::9]) else b[:, :1].T
        f = s2.srgemm_f16 if half else s2.srgemm
        check(op, a, b, c, f(op, a, b, c, do_epilogue=True), half)
        if not offset:
            assert torch.equal(f(op, a, b, c, do_epilogue=True), f(op, a, b, c, do_epilogue=True))
    assert s2.device_status() == 0
