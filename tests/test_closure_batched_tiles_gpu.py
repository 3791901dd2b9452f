"""The batched closure's tile scheduling, code range and restarts against the
oracle, bit for bit: graphs of one and of several tiles in one batch, few large
graphs among many small ones, results that outgrow the 16-bit codes in the
middle of a closure, and more steps than the entry list holds."""
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


def check(op, graphs, **kw):
    mats = [torch.from_numpy(g.copy()).cuda() for g in graphs]
    iters = s2.closure_batched(op, mats, **kw)
    for g, m, it in zip(graphs, mats, iters):
        want, want_it = oracle.closure(op, g)
        assert it == want_it, (op, g.shape, it, want_it)
        same(m, want, f"{op} n={g.shape[0]}")
    assert s2.device_status() == 0


@pytest.mark.parametrize("op", ["min_plus", "max_plus", "max_min", "min_mul"])
def test_mixed_sizes(cuda, op):
    """One large graph, some of a few tiles, many of one."""
    rng = np.random.default_rng(3)
    sizes = [640, 300, 257, 256, 129, 130, 191, 193] + [int(v) for v in rng.integers(1, 129, 30)]
    graphs = []
    for i, n in enumerate(sizes):
        x = datagen.closure_graph("min_plus" if op in ("min_plus", "min_mul") else "max_min", n, 0.05, seed=i)
        if op == "max_plus":  # a DAG, so longest paths exist
            x = np.where(np.triu(np.ones((n, n), bool), 1), x, np.float32(-np.inf)).astype(np.float32)
        if op == "min_mul":
            x = np.where(np.isinf(x), x, 1.0 + x / 128.0).astype(np.float32)
            np.fill_diagonal(x, 1.0)
        graphs.append(x)
    check(op, graphs)


def test_steps_of_more_tiles_than_threads(cuda):
    """A step of 576 tiles is published by every warp of the CTA that opens it, in
    two rounds; beside it steps of 36 tiles (two warps).  A disjoint union of small
    graphs, so the oracle closes it by parts."""
    part, parts = 48, 63
    n = part * parts
    graphs = [datagen.er_graph(part, 0.06, seed=i) for i in range(parts)]
    x = np.full((n, n), np.inf, np.float32)
    want = x.copy()
    steps = 0
    for i, g in enumerate(graphs):
        w, it = oracle.closure("min_plus", g)
        x[i * part:(i + 1) * part, i * part:(i + 1) * part] = g
        want[i * part:(i + 1) * part, i * part:(i + 1) * part] = w
        steps = max(steps, it)
    mid = datagen.er_graph(700, 0.02, seed=9)
    want_mid, it_mid = oracle.closure("min_plus", mid)
    for _ in range(3):
        mats = [torch.from_numpy(g.copy()).cuda() for g in (x, mid, mid)]
        assert list(s2.closure_batched("min_plus", mats)) == [steps, it_mid, it_mid]
        same(mats[0], want)
        same(mats[1], want_mid)
        same(mats[2], want_mid)
    assert s2.device_status() == 0


@pytest.mark.parametrize("op", ["min_plus", "max_min", "max_mul"])
@pytest.mark.parametrize("sizes", [(0,), (0, 0, 0), (0, 40, 0, 300, 128, 0)])
def test_empty_graphs(cuda, op, sizes):
    """A graph without vertices takes one unchanged step and no tile."""
    graphs = []
    for i, n in enumerate(sizes):
        x = datagen.closure_graph("max_min" if op == "max_min" else "min_plus", max(n, 1), 0.1, seed=i)[:n, :n]
        if op == "max_mul":  # weights in (0, 1], no edge 0
            x = np.where(np.isinf(x), np.float32(0.0), 1.0 / (1.0 + x)).astype(np.float32)
        graphs.append(np.ascontiguousarray(x))
    mats = [torch.from_numpy(g.copy()).cuda() for g in graphs]
    plan = s2.BatchedClosure(op, mats)
    for _ in range(2):
        for g, m in zip(graphs, mats):
            m.copy_(torch.from_numpy(g))
        plan.run()
        torch.cuda.synchronize()
        its, not_converged = plan.iters()
        assert not_converged == 0
        for g, m, it in zip(graphs, mats, its):
            want, want_it = oracle.closure(op, g) if g.shape[0] else (g, 1)
            assert it == want_it
            same(m, want)
    plan.close()
    assert s2.device_status() == 0


@pytest.mark.parametrize("n", [100, 300])
def test_outgrows_codes(cuda, n):
    """A path of heavy edges: distances pass 16383 in the second squaring, so the
    graph starts again on FP32; its neighbours in the batch stay coded."""
    chain = np.full((n, n), np.inf, np.float32)
    np.fill_diagonal(chain, 0.0)
    for i in range(n - 1):
        chain[i, i + 1] = 6000.0 + i
    big = datagen.er_graph(n, 0.1, seed=1)
    big[3, 5] = 16384.0  # no code from the start
    frac = datagen.er_graph(n, 0.1, seed=2) + np.float32(0.25)
    check("min_plus", [chain, datagen.er_graph(n, 0.1, seed=3), big, frac, datagen.er_graph(40, 0.1, seed=4)])


@pytest.mark.parametrize("n", [45, 113, 300])
def test_runs_of_one_plan_take_turns(cuda, n):
    """Codes and FP32 operands share their memory: one plan run on graphs that stay
    on codes, that outgrow them, that have none, and on codes again."""
    coded = datagen.er_graph(n, 0.1, seed=n)
    heavy = np.full((n, n), np.inf, np.float32)
    np.fill_diagonal(heavy, 0.0)
    heavy[np.arange(n - 1), np.arange(1, n)] = 6000.0
    frac = coded + np.float32(0.25)
    first, second = torch.empty((n, n), device=cuda), torch.empty((n, n), device=cuda)
    plan = s2.BatchedClosure("min_plus", [first, second])
    graphs = {id(g): (g,) + oracle.closure("min_plus", g) for g in (coded, heavy, frac)}
    for a, b in ((coded, frac), (heavy, coded), (frac, heavy), (coded, coded), (heavy, frac)):
        first.copy_(torch.from_numpy(a))
        second.copy_(torch.from_numpy(b))
        plan.run()
        torch.cuda.synchronize()
        its, not_converged = plan.iters()
        assert not_converged == 0
        for m, g, it in ((first, a, its[0]), (second, b, its[1])):
            _, want, steps = graphs[id(g)]
            assert it == steps
            same(m, want)
    plan.close()
    assert s2.device_status() == 0


@pytest.mark.parametrize("op", ["max_plus", "max_min"])
def test_aplp_change_test(cuda, op):
    """The change test that writes -FLT_MAX keeps a plan on FP32 from the start."""
    graphs = []
    for n in (45, 130, 300):
        x = datagen.closure_graph("max_min", n, 6.0 / n, seed=n)
        x = np.where(np.isinf(x), np.float32(-3.4028234663852886e38), x).astype(np.float32)
        if op == "max_plus":  # a DAG, so longest paths exist
            x = np.where(np.triu(np.ones((n, n), bool), 1), x, np.float32(-3.4028234663852886e38)).astype(np.float32)
        graphs.append(x)
    mats = [torch.from_numpy(g.copy()).cuda() for g in graphs]
    its = s2.closure_batched(op, mats, conv="aplp")
    for g, m, it in zip(graphs, mats, its):
        want, steps = oracle.closure(op, g, tol_mode=2)
        assert it == steps
        same(m, want)
    assert s2.device_status() == 0


@pytest.mark.parametrize("op", ["min_plus", "max_min", "max_mul"])
def test_plan_memory(cuda, op):
    """Both operand layouts of X, twice: 16 bytes an element, codes or not."""
    n = 8192
    X = torch.zeros((n, n), device=cuda)
    s2.closure_batched(op, [torch.ones((130, 130), device=cuda)], max_iter=1)  # kernels loaded
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    plan = s2.BatchedClosure(op, [X])
    used = before - torch.cuda.mem_get_info()[0]
    plan.close()
    assert used <= 16.25 * n * n


def test_more_steps_than_entries(cuda):
    """Longest paths around a cycle never settle: every step changes X, past the
    codes' range and past the steps the entry list has room for."""
    n, steps = 150, 90
    rng = np.random.default_rng(8)
    x = np.full((n, n), -np.inf, np.float32)
    x[rng.random((n, n)) < 0.03] = 1.0
    x[np.arange(n), (np.arange(n) + 1) % n] = 1.0
    graphs = [x, np.roll(x, 1, 0), datagen.closure_graph("max_min", 200, 0.1, seed=2)]
    mats = [torch.from_numpy(g.copy()).cuda() for g in graphs]
    plan = s2.BatchedClosure("max_plus", mats, max_iter=steps)
    plan.run()
    torch.cuda.synchronize()
    its, not_converged = plan.iters()
    for g, m, it in zip(graphs, mats, its):
        want, cur = g, g
        done = 0
        while done < steps:
            cur = oracle.srgemm("max_plus", want, want, want, do_epilogue=True, threads=8)
            done += 1
            stop = np.array_equal(cur.view(np.uint32), want.view(np.uint32))
            want = cur
            if stop:
                break
        assert it == done
        same(m, want)
    assert not_converged >= 2
    plan.close()
    assert s2.device_status() == 0
