"""Performance cases: what a program that uses simd2_b200 has it do.

Each case is one call (or, for the in-place closures, one copy of the input
and one call) of a public entry point on inputs that lie in device memory.
Kinds of case and the ranges `draw` takes them from:

  srgemm    srgemm of the nine semirings, float32 (or_and: int32 or uint8),
            any M, N, K in 16..4096, with and without the C term
  f16       srgemm_f16 (float16 A and B, float32 C and D), 16..2048
  closure   closure of one dense graph, 32..2048 vertices
  gtc       or_and closure (transitive closure) of a sparse graph, 512..16384
  batched   one launch over 16..512 graphs of uneven size, 32..1024 vertices
  knn       k nearest neighbours: 64..16384 queries, 256..65536 references,
            2..300 dimensions, k 1..32
  rmat      closure_ex with a dispatch policy on an R-MAT graph, average degree
            4..1024, 2048 or 4096 vertices (the generator needs a power of two)
"""
import math
import os
import random

import torch

import simd2_b200 as s2
from simd2_b200 import costmodel, datagen

INF = float("inf")
OPS = s2.OPS
FLOAT_OPS = tuple(op for op in OPS if op != "or_and")
CLOSURE_OPS = ("min_plus", "max_plus", "max_min", "min_max", "max_mul", "min_mul")
WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(s2.__file__)), "costmodel_weights.json")


def listed():
    return [
        # The smallest calls: one small product, bound by the call itself.
        {"name": "srgemm_small", "kind": "srgemm", "op": "min_plus", "dtype": "f32", "m": 100, "n": 100, "k": 100, "c": False},
        # An ordinary product of odd sizes with the C term (a capacity update).
        {"name": "srgemm_ragged", "kind": "srgemm", "op": "max_min", "dtype": "f32", "m": 1000, "n": 1203, "k": 1501, "c": True},
        # The sweep's size for the shortest-path semiring, accumulating into C.
        {"name": "srgemm_min_plus", "kind": "srgemm", "op": "min_plus", "dtype": "f32", "m": 4096, "n": 4096, "k": 4096, "c": True},
        # The largest dense contraction of the tests and the benchmark.
        {"name": "srgemm_plus_mul", "kind": "srgemm", "op": "plus_mul", "dtype": "f32", "m": 8192, "n": 8192, "k": 8192, "c": False},
        # Pairwise squared distances between two ordinary point sets.
        {"name": "srgemm_minus_square", "kind": "srgemm", "op": "minus_square", "dtype": "f32", "m": 1500, "n": 2100, "k": 300, "c": False},
        # The int32 Boolean surface, as the reference's gtc app calls it.
        {"name": "srgemm_or_and", "kind": "srgemm", "op": "or_and", "dtype": "i32", "m": 3000, "n": 2500, "k": 2000, "c": True},
        # The float16 entry that stands behind tensor_srgemm.
        {"name": "f16_plus_mul", "kind": "f16", "op": "plus_mul", "m": 2048, "n": 2048, "k": 2048, "c": True},
        # All-pairs shortest paths of a 512-vertex random graph: a chain of
        # short steps with a change test after each.
        {"name": "closure_512", "kind": "closure", "op": "min_plus", "n": 512, "p": 0.05},
        # Transitive closure of a large sparse graph.
        {"name": "gtc_16384", "kind": "gtc", "n": 16384, "degree": 2.0},
        # Many graphs of uneven size through a kept plan.
        {"name": "batched_512", "kind": "batched", "op": "min_plus", "count": 512, "nmin": 32, "nmax": 1024},
        # The nearest-neighbour search of the tests and the benchmark.
        {"name": "knn_16384", "kind": "knn", "q": 16384, "r": 65536, "d": 128, "k": 16},
        # A mixed-density graph closed under the learned dispatch.
        {"name": "rmat_4096", "kind": "rmat", "dispatch": "learned", "n": 4096, "degree": 32.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("srgemm", "srgemm", "srgemm", "f16", "closure", "gtc", "batched", "knn", "rmat"))
    if kind == "srgemm":
        op = rng.choice(OPS)
        dtype = rng.choice(("i32", "u8")) if op == "or_and" else "f32"
        m, n, k = (_log(rng, 16, 4096) for _ in range(3))
        return {"kind": kind, "op": op, "dtype": dtype, "m": m, "n": n, "k": k, "c": rng.random() < 0.5}
    if kind == "f16":
        m, n, k = (_log(rng, 16, 2048) for _ in range(3))
        return {"kind": kind, "op": rng.choice(OPS), "m": m, "n": n, "k": k, "c": rng.random() < 0.5}
    if kind == "closure":
        return {"kind": kind, "op": rng.choice(CLOSURE_OPS), "n": _log(rng, 32, 2048), "p": round(rng.uniform(0.01, 0.3), 3)}
    if kind == "gtc":
        return {"kind": kind, "n": _log(rng, 512, 16384), "degree": round(rng.uniform(1.5, 8.0), 2)}
    if kind == "batched":
        nmax = _log(rng, 64, 1024)
        return {"kind": kind, "op": rng.choice(CLOSURE_OPS), "count": _log(rng, 16, 512), "nmin": 32, "nmax": nmax}
    if kind == "knn":
        return {"kind": kind, "q": _log(rng, 64, 16384), "r": _log(rng, 256, 65536), "d": _log(rng, 2, 300), "k": rng.randint(1, 32)}
    return {"kind": kind, "dispatch": rng.choice(("dense", "rules", "learned")), "n": rng.choice((2048, 4096)),
            "degree": float(_log(rng, 4, 1024))}


# ---------------------------------------------------------------------------
# inputs: the value distributions of simd2_b200.datagen, drawn on the GPU
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _values(op, rows, cols, g):
    """Operand values of the nine-semiring sweep."""
    shape = (rows, cols)
    if op in ("plus_mul", "minus_square"):
        return torch.randn(shape, generator=g, device="cuda")
    if op in ("max_mul", "min_mul"):
        return 1.0 - torch.rand(shape, generator=g, device="cuda")
    x = torch.randint(1, 1001, shape, generator=g, device="cuda").float()
    x[torch.rand(shape, generator=g, device="cuda") < 0.2] = _identity(op)
    return x


def _identity(op):
    return -INF if op.startswith("max") else INF


def _bits(rows, cols, g, density=0.01):
    return torch.rand((rows, cols), generator=g, device="cuda") < density


def _graph(op, n, p, g):
    """Edge weights of a random graph with the reference apps' fill values."""
    if op in ("max_mul", "min_mul"):
        w = 1.0 - torch.rand((n, n), generator=g, device="cuda")
    else:
        w = torch.randint(1, 101, (n, n), generator=g, device="cuda").float()
    fill = torch.full((), _identity(op), device="cuda")
    x = torch.where(torch.rand((n, n), generator=g, device="cuda") < p, w, fill)
    if op == "max_plus":  # longest paths: edges only from lower to higher vertices
        x = torch.where(torch.ones((n, n), dtype=torch.bool, device="cuda").triu(1), x, fill)
    else:
        x.fill_diagonal_({"min_plus": 0.0, "max_mul": 1.0, "min_mul": 1.0}.get(op, _identity(op)))
    return x


def _batched_sizes(case):
    """Sizes (log-uniform) and edge probabilities of a batched case."""
    r = random.Random(3)
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
    sizes = [int(round(math.exp(r.uniform(lo, hi)))) for _ in range(case["count"])]
    return sizes, [r.uniform(0.01, 0.3) for _ in sizes]


def _square_views(flat, sizes):
    out, at = [], 0
    for n in sizes:
        out.append(flat[at:at + n * n].view(n, n))
        at += n * n
    return out


def _batched_flat(case, g):
    sizes, probs = _batched_sizes(case)
    flat = torch.empty(sum(n * n for n in sizes), device="cuda")
    for x, p in zip(_square_views(flat, sizes), probs):
        x.copy_(_graph(case["op"], x.shape[0], p, g))
    return flat, sizes


def _points(case, g):
    """N(0,1) points; a share of the queries nearly duplicates a reference."""
    q, r, d = case["q"], case["r"], case["d"]
    ref = torch.randn((r, d), generator=g, device="cuda")
    query = torch.randn((q, d), generator=g, device="cuda")
    dup = q // 20
    at = torch.randint(0, r, (dup,), generator=g, device="cuda")
    query[:dup] = ref[at] + 1e-3 * torch.randn((dup, d), generator=g, device="cuda")
    return query, ref


def _inputs(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind in ("srgemm", "f16"):
        m, n, k, op = case["m"], case["n"], case["k"], case["op"]
        shapes = [(m, k), (k, n)] + ([(m, n)] if case["c"] else [])
        if op == "or_and":
            ts = [_bits(*s, g) for s in shapes]
            if kind == "f16":
                ts = [t.float() for t in ts]
            else:
                ts = [t.to(torch.int32 if case["dtype"] == "i32" else torch.uint8) for t in ts]
        else:
            ts = [_values(op, *s, g) for s in shapes]
        if kind == "f16":
            ts[:2] = [t.half() for t in ts[:2]]
        return ts + [None] * (3 - len(ts))
    if kind == "closure":
        return [_graph(case["op"], case["n"], case["p"], g)]
    if kind == "gtc":
        return [_bits(case["n"], case["n"], g, case["degree"] / case["n"]).to(torch.uint8)]
    if kind == "batched":
        return [_batched_flat(case, g)[0]]
    if kind == "knn":
        return list(_points(case, g))
    return [datagen.rmat_graph_device(case["n"], case["degree"], seed, "cuda")]


def prepare(case, seed):
    state = {"case": case, "in": _inputs(case, seed)}
    kind = case["kind"]
    if kind in ("closure", "gtc", "rmat", "batched"):
        state["x"] = torch.empty_like(state["in"][0])  # closed in place
    if kind == "batched":
        state["plan"] = s2.BatchedClosure(case["op"], _square_views(state["x"], _batched_sizes(case)[0]))
    if kind == "rmat":
        state["mlp"] = costmodel.load(WEIGHTS) if case["dispatch"] == "learned" else None
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("srgemm", "f16"):
        a, b, c = state["in"]
        call = s2.srgemm if kind == "srgemm" else s2.srgemm_f16
        return call(case["op"], a, b, c, do_epilogue=case["c"])
    if kind == "knn":
        dist, idx = s2.knn(*state["in"], case["k"])
        return {"dist": dist, "idx": idx}
    x = state["x"]
    x.copy_(state["in"][0])
    if kind == "batched":
        state["plan"].run()
        return x
    if kind == "rmat":
        steps = s2.closure_ex("min_plus", x, dispatch=case["dispatch"], mlp_params=state["mlp"])
    else:
        steps = s2.closure("or_and" if kind == "gtc" else case["op"], x)
    return {"x": x, "steps": steps}


def work(case):
    """Inputs read once and outputs written once; two operations per (x), (+)
    pair of a product.  A closure is counted as one all-pairs pass (n^3 pairs,
    as Floyd-Warshall makes): the number of squarings depends on the values."""
    kind = case["kind"]
    if kind in ("srgemm", "f16"):
        m, n, k = case["m"], case["n"], case["k"]
        ab = 2 if kind == "f16" else 1 if case["dtype"] == "u8" else 4
        cd = 4 if kind == "f16" else ab
        return {"bytes": ab * (m * k + k * n) + cd * m * n * (2 if case["c"] else 1), "flops": 2 * m * n * k}
    if kind == "knn":
        q, r, d, k = case["q"], case["r"], case["d"], case["k"]
        return {"bytes": 4 * (q + r) * d + 8 * q * k, "flops": 2 * q * r * d}
    if kind == "batched":
        sizes = _batched_sizes(case)[0]
        return {"bytes": 8 * sum(n * n for n in sizes), "flops": 2 * sum(n ** 3 for n in sizes)}
    n = case["n"]
    return {"bytes": (2 if kind == "gtc" else 8) * n * n, "flops": 2 * n ** 3}


# ---------------------------------------------------------------------------
# the same results in 64 bits, with torch alone
# ---------------------------------------------------------------------------
_TIMES = {"plus": torch.add, "mul": torch.mul, "min": torch.minimum, "max": torch.maximum}


def _product64(op, a, b):
    """id (+) A(x)B in 64 bits."""
    if op == "plus_mul":
        return a @ b
    if op == "minus_square":
        return (a * a).sum(1, keepdim=True) + (b * b).sum(0, keepdim=True) - 2.0 * (a @ b)
    plus, times = op.split("_")
    times = _TIMES[times]
    out = torch.empty((a.shape[0], b.shape[1]), dtype=torch.float64, device=a.device)
    rows = max(1, (1 << 27) // max(1, b.numel()))
    for i in range(0, a.shape[0], rows):
        t = times(a[i:i + rows, :, None], b[None])
        out[i:i + rows] = t.amin(1) if plus == "min" else t.amax(1)
    return out


def _plus64(op, x, y):
    if op in ("plus_mul", "minus_square"):
        return x + y
    return torch.minimum(x, y) if op.startswith("min") else torch.maximum(x, y)


def _closure64(op, x):
    x = x.double()
    while True:
        y = _plus64(op, _product64(op, x, x), x)
        if torch.equal(x, y):
            return x
        x = y


def exact(case, seed):
    ins = _inputs(case, seed)
    kind = case["kind"]
    if kind in ("srgemm", "f16"):
        a, b, c = ins
        if case["op"] == "or_and":
            if kind == "srgemm":
                return None  # whole numbers
            d = ((a.double() @ b.double()) > 0).double()
            return torch.maximum(d, (c != 0).double()) if c is not None else d
        d = _product64(case["op"], a.double(), b.double())
        return _plus64(case["op"], d, c.double()) if c is not None else d
    if kind == "closure":
        if case["op"] in ("max_mul", "min_mul", "max_plus"):
            return None  # rounding of repeated products depends on the step that forms them
        return {"x": _closure64(case["op"], ins[0]), "steps": None}
    if kind == "rmat":
        return {"x": _closure64("min_plus", ins[0]), "steps": None}
    if kind == "batched":
        if case["op"] in ("max_mul", "min_mul", "max_plus"):
            return None
        views = _square_views(ins[0], _batched_sizes(case)[0])
        return torch.cat([_closure64(case["op"], x).reshape(-1) for x in views])
    if kind == "knn":
        q, r = (t.double() for t in ins)
        rt = r.t().contiguous()
        rows = max(1, (1 << 27) // r.shape[0])
        best = []
        for i in range(0, q.shape[0], rows):
            sq = _product64("minus_square", q[i:i + rows], rt).clamp_min_(0.0)
            best.append(sq.topk(min(case["k"], r.shape[0]), dim=1, largest=False).values.sqrt())
        return {"dist": torch.cat(best), "idx": None}
    return None
