"""Small closures as one cooperative launch (closure_coop.cuh) against the oracle,
bit for bit: sizes around the 64-wide tiles and the split of tiles between CTAs,
entries and results without a 16-bit code (the launch-per-step path takes over),
the step limit, the change tests, and rows with a pitch."""
import os
import subprocess

import numpy as np
import pytest
import torch

import oracle
import simd2_b200 as s2
from simd2_b200 import datagen

pytestmark = pytest.mark.gpu


def same(got, want, msg=""):
    np.testing.assert_array_equal(got.cpu().numpy().view(np.uint32), np.ascontiguousarray(want).view(np.uint32),
                                  err_msg=msg)


def graph(op, n, p, seed):
    x = datagen.closure_graph("min_plus" if op.startswith("min") else "max_min", n, p, seed)
    if op == "max_plus":
        x = np.where(np.triu(np.ones((n, n), bool), 1), x, np.float32(-np.inf)).astype(np.float32)
    return x


@pytest.mark.parametrize("op", ["min_plus", "max_plus", "max_min", "min_max"])
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 130, 257, 500, 769])
def test_sizes(cuda, op, n):
    x = graph(op, n, min(1.0, 8.0 / n), n)
    want, steps = oracle.closure(op, x)
    X = torch.from_numpy(x.copy()).cuda()
    assert s2.closure(op, X) == steps
    same(X, want, f"{op} {n}")
    wide = torch.full((n, n + 7), 3.0, device=cuda)  # rows off the 16-byte grid
    wide[:, 3:3 + n] = torch.from_numpy(x).cuda()
    assert s2.closure(op, wide[:, 3:3 + n]) == steps
    same(wide[:, 3:3 + n].contiguous(), want, f"{op} {n} pitched")
    assert torch.all(wide[:, :3] == 3.0) and torch.all(wide[:, 3 + n:] == 3.0)
    assert s2.device_status() == 0


@pytest.mark.parametrize("case", ["entry", "result", "fraction"])
def test_without_codes(cuda, case):
    n = 200
    x = np.full((n, n), np.inf, np.float32)
    np.fill_diagonal(x, 0.0)
    x[np.arange(n - 1), np.arange(1, n)] = {"entry": 16384.0, "result": 5000.0, "fraction": 0.5}[case]
    want, steps = oracle.closure("min_plus", x)
    X = torch.from_numpy(x.copy()).cuda()
    assert s2.closure("min_plus", X) == steps
    same(X, want, case)


@pytest.mark.parametrize("op", ["min_plus", "max_min"])
@pytest.mark.parametrize("n", [130, 700])
def test_entry_without_code_goes_on_in_fp32(cuda, op, n):
    """One fraction, then all fractions; on either side of the tile sizes."""
    x = graph(op, n, 8.0 / n, n)
    for x in (np.where(np.arange(n * n).reshape(n, n) == 2, np.float32(0.3), x), x + np.float32(0.3)):
        want, steps = oracle.closure(op, x)
        X = torch.from_numpy(x.copy()).cuda()
        assert s2.closure(op, X) == steps
        same(X, want, f"{op} {n}")
    assert s2.device_status() == 0


@pytest.mark.parametrize("op", ["min_plus", "max_plus"])
@pytest.mark.parametrize("n", [90, 200, 500, 1100])
def test_first_squaring_outgrows_codes(cuda, op, n):
    """Sums of two entries already have no code, found by CTAs that leave the grid
    barrier of the coding pass at different times; on one tile and on many."""
    x = np.full((n, n), np.inf if op == "min_plus" else -np.inf, np.float32)
    np.fill_diagonal(x, 0.0)
    for i in range(0, n - 1, 3):  # paths of three vertices
        x[i, i + 1] = 9000.0 + i
        if i + 2 < n:
            x[i + 1, i + 2] = 8200.0 + i
    want, steps = oracle.closure(op, x)
    assert np.isfinite(want).sum() > np.isfinite(x).sum()
    for _ in range(10):
        X = torch.from_numpy(x.copy()).cuda()
        assert s2.closure(op, X) == steps
        same(X, want, f"{op} {n}")
    assert s2.device_status() == 0


@pytest.mark.parametrize("op", ["min_plus", "max_min"])
@pytest.mark.parametrize("steps", [1, 2, 3])
def test_step_limit(cuda, op, steps):
    x = graph(op, 300, 0.01, 5)
    want = x
    for _ in range(steps):
        want = oracle.srgemm(op, want, want, want, do_epilogue=True, threads=8)
    X = torch.from_numpy(x.copy()).cuda()
    with pytest.raises(s2.NotConverged):
        s2.closure(op, X, max_iter=steps)
    same(X, want)


@pytest.mark.parametrize("op", ["min_plus", "max_min"])
def test_tolerance_change_test(cuda, op):
    x = graph(op, 150, 0.05, 6)
    if op == "max_min":
        x = (x / 1024.0).astype(np.float32)  # FP16 fractions, some steps move by less than the tolerance
        x[np.isinf(x)] = -np.inf
    want, steps = oracle.closure(op, x, tol_mode=1)
    X = torch.from_numpy(x.copy()).cuda()
    assert s2.closure(op, X, conv="tol") == steps
    same(X, want)


def test_failed_wait_reaches_every_cta(cuda, tmp_path):
    """A CTA whose bounded wait ran out may not leave the others to finish on its
    data: after the grid barrier all of them know."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    exe = tmp_path / "coop_barrier"
    res = subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1",
                          os.path.join(root, "tests", "device", "coop_barrier.cu"), "-o", str(exe)],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0, (res.returncode, res.stdout)


def test_profiled(cuda):
    """The one launch of a small closure is timed, and counts every step's
    operations; one that falls back adds its discarded launch's time alone."""
    n = 300
    x = graph("min_plus", n, 0.03, 7)
    with s2.KernelTimer() as t:
        steps = s2.closure("min_plus", torch.from_numpy(x).cuda())
    assert steps > 1 and t.launches == 1
    assert t.ops == 2 * n ** 3 * steps
    assert t.kernel_ms > 0.0
    assert t.by_kind["simt"][1:] == (1, t.ops)
    with s2.KernelTimer() as t:
        steps = s2.closure("min_plus", torch.from_numpy(x + np.float32(0.25)).cuda())
    assert t.launches > steps and t.ops >= 2 * n ** 3 * steps
