"""The work a user of this package has it do, as cases to be timed: searches for single goals,
precomputed databases, refills of a planned database, and lookups. All sizes are those of the
command line (`morello matmul <n>`, `precompute <size>`), of bench.py and of the tests.

A case is a dict of plain values; `op` says which entry points a pass goes through:

  search      top_down_many of a goal Spec (and the same Spec with its operands in faster memories)
              under `queries` memory budgets, the filled table left on the device, then get_impl of the
              goal (what the command line does with a Spec: search, print the implementation)
  search_noalloc   the same search through top_down_many_noalloc, by a host whose tables hold all of HBM
  precompute  precompute(size, through, dtypes), the whole table to the host (export_all, what a page
              writer consumes) and get_many of `queries` Specs
  fill        fill() of a planned and uploaded database, the table left on the device, and get_many
              of `queries` Specs
  lookup      get_many of `queries` (Spec, limits) pairs in a filled database

A seed decides the memory budgets and which Specs are asked for; the Spec space itself is generated
from the sizes alone, so every seed of a case is the same amount of work.
"""
import functools
import itertools
import math
import random

import numpy as np
import torch

import morello_b200 as m

DTYPES = {"u32": (m.DTYPE_U32,), "f32": (m.DTYPE_F32,), "both": (m.DTYPE_U32, m.DTYPE_F32)}
KINDS = {"move": m.KIND_MOVE, "zero": m.KIND_FILL_ZERO, "accum": m.KIND_MATMUL_ACCUM, "matmul": m.KIND_MATMUL}
THROUGH = {"move": m.THROUGH_MOVE, "zero": m.THROUGH_ZERO, "matmul": m.THROUGH_MATMUL}


def listed():
    return [
        # The smallest search there is (the smoke test's): all launch and call overhead.
        {"name": "search_matmul_1x1x1", "op": "search", "kind": "matmul", "shape": "1x1x1x1", "dtypes": "u32", "queries": 16},
        # `morello matmul 2`, the command line's own example: 86 stages of a few Specs each.
        {"name": "search_matmul_2x2x2", "op": "search", "kind": "matmul", "shape": "1x2x2x2", "dtypes": "u32", "queries": 16},
        # A middling goal, ragged, in both dtypes at once, under many budgets.
        {"name": "search_matmul_2x8x4", "op": "search", "kind": "matmul", "shape": "1x2x8x4", "dtypes": "both", "queries": 64},
        # The largest Matmul goal of the tests: half a million Specs, as much planning as solving.
        {"name": "search_matmul_8x8x8", "op": "search", "kind": "matmul", "shape": "1x8x8x8", "dtypes": "f32", "queries": 64},
        # A relayout of a matrix: few Specs with many actions each, deep same-stage dependencies.
        {"name": "search_move_16x16", "op": "search", "kind": "move", "shape": "16x16", "dtypes": "f32", "queries": 16},
        # A search by a host that may not allocate on the device.
        {"name": "search_noalloc_matmul_2x2x2", "op": "search_noalloc", "kind": "matmul", "shape": "1x2x2x2", "dtypes": "f32", "queries": 16},
        # `precompute 2`, the size the reference's own checks run.
        {"name": "precompute_2", "op": "precompute", "size": 2, "through": "matmul", "dtypes": "both", "queries": 256},
        # `precompute 4`: an ordinary database, 0.6 M Specs.
        {"name": "precompute_4", "op": "precompute", "size": 4, "through": "matmul", "dtypes": "both", "queries": 256},
        # The Move and Zero phases of `precompute 8` in one dtype, as a first part of a database.
        {"name": "precompute_8_zero", "op": "precompute", "size": 8, "through": "zero", "dtypes": "f32", "queries": 256},
        # bench.py's headline table in one dtype: 7.3 M Specs, 200 M candidate records, throughput.
        {"name": "fill_8", "op": "fill", "size": 8, "through": "matmul", "dtypes": "u32", "queries": 256},
        # A search's own use of a finished database: a Spec and its neighbours at a few limits.
        {"name": "lookup_16", "op": "lookup", "size": 4, "through": "matmul", "dtypes": "both", "queries": 16},
        # A sweep over a database, as the parity tests make it.
        {"name": "lookup_16384", "op": "lookup", "size": 4, "through": "matmul", "dtypes": "both", "queries": 16384},
    ]


def draw(rng):
    op = rng.choice(["search", "search", "search", "search_noalloc", "precompute", "fill", "lookup"])
    dtypes = rng.choice(["u32", "f32", "both"])
    if op in ("search", "search_noalloc"):
        kind = rng.choice(["move", "zero", "accum", "matmul", "matmul"])
        # dims are powers of two (the only tile scale); all of a shape's dims multiply to at most
        # 2^most. The fixed device array of the no-allocation entry point holds the small ones.
        most = 3 if op == "search_noalloc" else (8 if kind in ("move", "zero") else (6 if dtypes == "both" else 8))
        left, dims = rng.randint(1, most), []
        rank = rng.randint(1, 3) if kind in ("move", "zero") else 3
        for _ in range(rank - 1):
            dims.append(rng.randint(0, min(left, 4)))
            left -= dims[-1]
        dims.append(min(left, 4) if rank > 1 else left)
        rng.shuffle(dims)
        shape = [1 << d for d in dims]
        if kind in ("accum", "matmul"):
            shape = [1] + shape
        return {"op": op, "kind": kind, "shape": "x".join(map(str, shape)), "dtypes": dtypes,
                "queries": round(2 ** rng.uniform(4, 7))}
    size = rng.choice([1, 2, 4, 8] if op == "precompute" else ([2, 4, 8] if op == "fill" else [2, 4]))
    through = rng.choice(["move", "zero"] if size == 8 else ["move", "zero", "matmul", "matmul"])
    queries = round(2 ** rng.uniform(3, 14)) if op == "lookup" else round(2 ** rng.uniform(5, 9))
    return {"op": op, "size": size, "through": through, "dtypes": dtypes, "queries": queries}


# ---- inputs ------------------------------------------------------------------------------

def _limits(rng):
    """A memory budget: any point of the limits lattice (registers by count, caches by powers of two)."""
    return (rng.randint(0, m.MAX_MEM[0]), rng.randint(0, m.MAX_MEM[1]), (1 << rng.randint(0, 11)) >> 1,
            (1 << rng.randint(0, 26)) >> 1)


def _goals(case, memory=m.GL):
    shape = [int(d) for d in case["shape"].split("x")]
    return [m.simple_spec(KINDS[case["kind"]], dt, shape, memory) for dt in DTYPES[case["dtypes"]]]


def _simple_queries(case, rng):
    """Row-major Specs of a precomputed space, at random limits (half of them with everything available)."""
    specs, limits = [], []
    logs = range(case["size"].bit_length())
    for _ in range(case["queries"]):
        kind = rng.choice(["move", "zero", "accum", "matmul"][:{"move": 1, "zero": 2, "matmul": 4}[case["through"]]])
        rank = 3 if kind in ("accum", "matmul") else rng.randint(1, 3)
        shape = ([1] if kind in ("accum", "matmul") else []) + [1 << rng.choice(logs) for _ in range(rank)]
        specs.append(m.simple_spec(KINDS[kind], rng.choice(DTYPES[case["dtypes"]]), shape, m.GL))
        limits.append(m.MAX_MEM if rng.random() < 0.5 else _limits(rng))
    return specs, limits


class _State:
    pass


def prepare(case, seed):
    rng = random.Random(seed)
    s = _State()
    s.case = case
    s.db = m.SynthesisDatabase(device=0)
    if case["op"] in ("search", "search_noalloc"):
        goals = _goals(case)
        s.goal = goals[0]
        # the goal itself with everything available, then the same Spec with its operands in any of
        # the scalar memories (Specs its own search meets too) under any budget
        s.specs, s.limits = list(goals), [m.MAX_MEM] * len(goals)
        while len(s.specs) < case["queries"]:
            s.specs.append(rng.choice(_goals(case, rng.choice([m.GL, m.L1, m.RF]))))
            s.limits.append(m.MAX_MEM if rng.random() < 0.5 else _limits(rng))
        return s
    s.args = (case["size"], THROUGH[case["through"]], DTYPES[case["dtypes"]])
    if case["op"] == "lookup":
        s.db.precompute(*s.args)
        n = s.db.num_specs()
        s.specs = [s.db.spec_blob(rng.randrange(n)) for _ in range(case["queries"])]
        s.limits = [_limits(rng) for _ in range(case["queries"])]
        return s
    s.specs, s.limits = _simple_queries(case, rng)
    if case["op"] == "fill":
        s.db.plan_precompute(*s.args)
        s.db.upload()
    return s


# ---- one pass ----------------------------------------------------------------------------

def _array(decisions):
    flat = itertools.chain.from_iterable((d.found, d.action, d.main_cost, d.depth) + d.peaks for d in decisions)
    return np.fromiter(flat, dtype=np.int64, count=8 * len(decisions)).reshape(-1, 8)


class _DeviceRows:
    """The finished table where it lies on the device, for torch to look at; keeps its database alive."""

    def __init__(self, db):
        self.db = db
        pointer, rows = db.device_rows()
        self.__cuda_array_interface__ = {"shape": (rows, 4), "typestr": "<i4", "data": (pointer, False), "strides": None,
                                         "version": 3}


def _device_rows(db):
    return torch.as_tensor(_DeviceRows(db), device=torch.device("cuda", 0))


def run(state):
    db, op = state.db, state.case["op"]
    if op == "search":
        got = db.top_down_many(state.specs, state.limits)
        impl = np.frombuffer(db.get_impl(state.goal).encode(), dtype=np.uint8)
        return {"decisions": _array(got), "impl": impl, "rows": _device_rows(db)}
    if op == "search_noalloc":
        return {"decisions": _array(db.top_down_many_noalloc(state.specs, state.limits))}
    if op == "precompute":
        db.precompute(*state.args)
        masks, first, rows = db.export_all()
        return {"masks": masks.view(np.int32), "first": first.view(np.int64), "rows": rows.view(np.int32),
                "decisions": _array(db.get_many(state.specs, state.limits))}
    if op == "fill":
        db.fill()
        return {"rows": _device_rows(db), "decisions": _array(db.get_many(state.specs, state.limits))}
    return {"decisions": _array(db.get_many(state.specs, state.limits))}


# ---- what a pass cannot do without -------------------------------------------------------

# (Specs, candidate records, table rows, bytes of records and child rows its rows are the combination of)
_FILL_8 = (7333498, 200375197, 267945719, 3.1e11)


@functools.lru_cache(maxsize=None)
def _counts(key):
    """(Specs, candidate records, table rows, combined bytes) of a search's or precompute's table."""
    case = dict(key)
    if case.get("size") == 8 and case["through"] == "matmul":
        return _FILL_8
    db = m.SynthesisDatabase(device=0)
    if "size" in case:
        st = db.precompute(case["size"], THROUGH[case["through"]], DTYPES[case["dtypes"]])
    else:
        db.top_down_many(_goals(case))
        st = db.stats()
    db.close()
    return st["n_specs"], st["n_candidates"], st["n_rows"], st["algorithmic_bytes"]


def work(case):
    """bytes: every candidate record (32) and Spec header (32) read once, every table row (16)
    written once, every query's Spec, limits and decision (about 150). flops: 8 integer operations
    per 16 bytes of record or child row that the finished rows are the combination of."""
    queries = 150 * case["queries"]
    if case["op"] == "lookup":
        # about 4 dependent reads per lookup: id table, Spec, header, row
        return {"bytes": queries + 4 * 32 * case["queries"], "flops": 0}
    specs, records, rows, combined = _counts(tuple(sorted((k, v) for k, v in case.items() if k in ("kind", "shape", "size", "through", "dtypes"))))
    return {"bytes": 32 * records + 32 * specs + 16 * rows + queries, "flops": math.ceil(combined / 2)}


def tolerance(case):
    return "exact"   # decisions and tables are whole numbers
