"""The persistent CUDA-core srgemm (srgemm_sk.cuh): tile sizes, split tiles and
the 16-bit codes against the CPU oracle, bit for bit.

The shapes lie on either side of each rule: 64 x 64 and 128 x 128 tiles, fewer
tiles than SMs (several CTAs per tile, evenly or by units), more tiles than SMs
with a remainder, K below, at and past a k-tile.  The values lie on either side
of the codes' range: 16383 is the largest coded integer, its sum with itself
the largest finite sum; one entry outside the range anywhere sends the call to
the FP32 operands.
"""
import numpy as np
import pytest
import torch

import oracle
import simd2_b200 as s2
from simd2_b200 import datagen

pytestmark = pytest.mark.gpu
CODED = ["min_plus", "max_plus", "max_min", "min_max"]
SHAPES = [(1, 1, 1), (63, 65, 7), (64, 64, 64), (65, 129, 72), (100, 100, 100), (30, 30, 3000), (200, 300, 640),
          (257, 255, 129), (700, 690, 66), (900, 905, 70), (1300, 1701, 33), (1030, 2050, 64)]


def same(got, want, msg=""):
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32), err_msg=msg)


def call(op, a, b, c=None, dev="cuda", **kw):
    A, B = (torch.from_numpy(np.ascontiguousarray(x)).to(dev) for x in (a, b))
    C = None if c is None else torch.from_numpy(np.ascontiguousarray(c)).to(dev)
    D = s2.srgemm(op, A, B, C, do_epilogue=c is not None, **kw)
    torch.cuda.synchronize()
    return D.cpu().numpy()


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("op", CODED + ["max_mul"])
def test_shapes(cuda, op, shape):
    m, n, k = shape
    a, b, c = datagen.semiring_operands(op, m, n, k, seed=m + 3 * n + 7 * k)
    same(call(op, a, b, c), oracle.srgemm(op, a, b, c, do_epilogue=True, threads=8), f"{op} {shape}")
    if op in CODED:  # fractions have no code: the FP32 operands
        a2 = a + np.float32(0.3)
        same(call(op, a2, b), oracle.srgemm(op, a2, b, threads=8), f"{op} {shape} fractions")
    assert s2.device_status() == 0


@pytest.mark.parametrize("op", CODED)
@pytest.mark.parametrize("value", [16383.0, 16384.0, 65504.0, 1e30, -3.0, 0.5, np.inf, -np.inf])
def test_code_range(cuda, op, value):
    """One value of the range's edge or beyond it, alone in A, alone in B, and
    everywhere."""
    m, n, k = 130, 70, 90
    rng = np.random.default_rng(5)
    ident = np.float32(np.inf if op.startswith("min") else -np.inf)
    if op.endswith("plus") and np.isinf(value) and np.float32(value) != ident:
        pytest.skip("inf - inf")
    a = rng.integers(0, 2000, size=(m, k)).astype(np.float32)
    b = rng.integers(0, 2000, size=(k, n)).astype(np.float32)
    a[rng.random((m, k)) < 0.2] = ident
    b[rng.random((k, n)) < 0.2] = ident
    v = np.float32(value)
    a1, b1 = a.copy(), b.copy()
    a1[m - 1, k - 1] = v
    b1[k - 1, n - 1] = v
    for x, y in ((a1, b), (a, b1), (np.full_like(a, v), np.full_like(b, v))):
        same(call(op, x, y), oracle.srgemm(op, x, y), f"{op} {value}")


@pytest.mark.parametrize("op", ["min_plus", "max_min"])
def test_strided_unaligned_and_in_place(cuda, op):
    """Rows off the 16-byte grid, wide pitches, and D written over C."""
    m, n, k = 150, 203, 77
    a, b, c = datagen.semiring_operands(op, m, n, k, seed=9)
    want = oracle.srgemm(op, a, b, c, do_epilogue=True)
    for off, extra in ((0, 0), (1, 3), (3, 8)):
        def place(x):
            buf = torch.full((x.shape[0], x.shape[1] + off + extra), float("nan"), device=cuda)
            view = buf[:, off:off + x.shape[1]]
            view.copy_(torch.from_numpy(x))
            return view
        A, B, C = place(a), place(b), place(c)
        s2.srgemm(op, A, B, C, do_epilogue=True, D=C)
        torch.cuda.synchronize()
        same(C.cpu().numpy(), want, f"{op} offset {off}")


@pytest.mark.parametrize("op", ["min_plus", "max_plus", "max_min", "max_mul", "min_mul", "min_max"])
@pytest.mark.parametrize("shape", [(1, 1, 1), (31, 33, 31), (32, 32, 32), (33, 32, 33), (5, 300, 65), (100, 100, 100),
                                   (383, 130, 64), (1000, 900, 5)])
def test_small_products(cuda, op, shape):
    """Sizes of the one-launch kernel (srgemm_small.cuh), float32 and float16, rows on
    and off the 16-byte grid, with and without C."""
    m, n, k = shape
    a, b, c = datagen.semiring_operands(op, m, n, k, seed=m + n + k)
    for off in (0, 1):
        def place(x, dt=torch.float32):
            buf = torch.full((x.shape[0], x.shape[1] + 2 * off), float("nan"), device=cuda, dtype=dt)
            view = buf[:, off:off + x.shape[1]]
            view.copy_(torch.from_numpy(x))
            return view
        for epi in (False, True):
            got = s2.srgemm(op, place(a), place(b), place(c) if epi else None, do_epilogue=epi)
            same(got.cpu().numpy(), oracle.srgemm(op, a, b, c, do_epilogue=epi), f"{op} {shape} {off} {epi}")
        ah, bh = (x.astype(np.float16) for x in (a, b))
        got = s2.srgemm_f16(op, place(ah, torch.float16), place(bh, torch.float16))
        same(got.cpu().numpy(), oracle.srgemm(op, ah.astype(np.float32), bh.astype(np.float32)), f"{op} {shape} f16")


@pytest.mark.parametrize("op", CODED)
@pytest.mark.parametrize("shape", [(1500, 1540, 960), (1500, 1540, 1030), (1153, 1409, 1285)])
def test_pair_of_launches(cuda, op, shape):
    """Sizes on either side of the line from which a product gets a launch for its
    codes and one for FP32: coded operands, fractions, and one entry without a code
    in the last row; a pair is timed as one launch."""
    m, n, k = shape
    a, b, c = datagen.semiring_operands(op, m, n, k, seed=m + k)
    same(call(op, a, b, c), oracle.srgemm(op, a, b, c, do_epilogue=True, threads=8), f"{op} {shape}")
    a2 = a + np.float32(0.3)
    same(call(op, a2, b), oracle.srgemm(op, a2, b, threads=8), f"{op} {shape} fractions")
    b[k - 1, n - 1] = 0.3
    with s2.KernelTimer() as t:
        got = call(op, a, b)
    same(got, oracle.srgemm(op, a, b, threads=8), f"{op} {shape} one fraction")
    assert (t.launches, t.ops) == (1, 2 * m * n * k)
    assert s2.device_status() == 0


@pytest.mark.parametrize("op", ["min_plus", "max_mul"])
@pytest.mark.parametrize("shape", [(1990, 2000, 64), (1990, 2000, 100), (2000, 2000, 130), (1600, 1601, 96), (2100, 1500, 48)])
def test_more_tiles_than_sms(cuda, op, shape):
    """Products of few k-tiles on either side of the line from which the last tiles
    are split, coded and not."""
    m, n, k = shape
    a, b, c = datagen.semiring_operands(op, m, n, k, seed=m + k)
    same(call(op, a, b, c), oracle.srgemm(op, a, b, c, do_epilogue=True, threads=8), f"{op} {shape}")
    a2 = (a * np.float32(1.3)).astype(np.float32)
    same(call(op, a2, b), oracle.srgemm(op, a2, b, threads=8), f"{op} {shape} fractions")
    assert s2.device_status() == 0
