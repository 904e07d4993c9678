"""Measured workloads of the query path, each one pass through the public Python entry points.

A partition (rhydb_gpu.Table on the host, rhydb_gpu.Device in HBM) is opened once and then serves
every query, so the partitions here come from the seeded generator with a fixed seed and are shared
by the states that use them; what a new seed brings is the queries (filter trees, filters, query
sequences, samples). Partitions follow the synthetic data set of the benchmark: a 29,903-nt genome,
0 or 12 amino-acid genes, date, country and lineage columns, optionally null sequences.

Every output is a whole number (counts, row sets, count tables, row ids), except the proportion of
a Mutations row (one quotient of two counts) and the planner network's numbers.
"""
import ctypes
import math
import sys
from collections import OrderedDict
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path.cwd() / "lapis-silo_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import rhydb_gpu as R  # noqa: E402
import workloads  # noqa: E402

GENOME = 29903
MIN_PROPORTION = 0.05
TABLE_SEED = 42


def listed():
    return [
        # one Aggregated count over a small instance: an interactive request, all latency
        {"name": "count_100k", "kind": "count", "rows": 100_000, "genes": 0, "nulls": 0.0, "calls": 1, "leaves": 0},
        # row sets of filters over the full data set (what the table scans of other actions consume)
        {"name": "rowsets_2m", "kind": "rowset", "rows": 2_000_000, "genes": 12, "nulls": 0.0, "calls": 8, "leaves": 0},
        # one Mutations table over the small instance
        {"name": "mutations_100k", "kind": "mutations", "rows": 100_000, "genes": 0, "nulls": 0.0, "calls": 1,
         "column": 0},
        # Mutations tables of the nucleotide column, one query per call, over the full data set
        {"name": "mutations_2m", "kind": "mutations", "rows": 2_000_000, "genes": 12, "nulls": 0.0, "calls": 4,
         "column": 0},
        # the Mutations pass of a caller that holds its filter and its counts in device memory
        {"name": "resident_2m", "kind": "resident", "rows": 2_000_000, "genes": 12, "nulls": 0.0, "column": 0,
         "density": 0.2},
        # a micro-batch: the requests of a few milliseconds, a ragged partition with null sequences
        {"name": "microbatch_500k", "kind": "batch_rows", "rows": 500_009, "genes": 12, "nulls": 0.002, "queries": 47,
         "mut_every": 4},
        # the benchmark's batch: 1,536 counts and 512 Mutations queries planned and run in one call
        {"name": "batch_2m", "kind": "batch_rows", "rows": 2_000_000, "genes": 12, "nulls": 0.0, "queries": 2048,
         "mut_every": 4},
        # the batching workload's trees: 1 to 64 leaves, NOf of up to 64 children, counts
        {"name": "trees_2m", "kind": "batch", "rows": 2_000_000, "genes": 12, "nulls": 0.0, "queries": 4096,
         "leaves": 64},
        # rows near a query sequence, at the distances a user tries
        {"name": "profile_2m", "kind": "profile", "rows": 2_000_000, "genes": 12, "nulls": 0.0, "calls": 4,
         "substitutions": 20},
        # counts grouped by a nucleotide position and a metadata column
        {"name": "aggregate_2m", "kind": "aggregate", "rows": 2_000_000, "genes": 12, "nulls": 0.0},
        # the serving loop: counts, Mutations and Details requests that arrive together
        {"name": "serve_2m", "kind": "serve", "rows": 2_000_000, "genes": 12, "nulls": 0.0, "requests": 256},
        # the planner network: gradient of a set of samples (forward and backward) and a prediction
        {"name": "planner_30k", "kind": "planner", "rows": 30_000, "genes": 0, "nulls": 0.0, "samples": 30_011},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["count", "rowset", "mutations", "mutations", "resident", "resident", "batch_rows", "batch_rows",
                       "batch", "profile", "aggregate", "serve", "planner"])
    # sizes log-uniform over the range of the listed partitions, most of them ragged in the last chunk
    case = {"kind": kind, "rows": _log_uniform(rng, 30_000, 2_000_000), "genes": rng.choice([0, 12]),
            "nulls": rng.choice([0.0, 0.002])}
    column = 0 if case["genes"] == 0 or rng.random() < 0.6 else rng.randint(1, 12)
    if kind in ("count", "rowset"):
        case.update(calls=rng.randint(1, 8), leaves=rng.choice([0, 0, 16]))
    elif kind == "mutations":
        case.update(calls=rng.randint(1, 4), column=column)
    elif kind == "resident":
        case.update(column=column, density=round(math.exp(rng.uniform(math.log(1e-4), math.log(0.9))), 6))
    elif kind == "batch_rows":
        case.update(queries=_log_uniform(rng, 8, 2048), mut_every=rng.choice([2, 4, 4, 8]))
    elif kind == "batch":
        case.update(queries=_log_uniform(rng, 32, 4096), leaves=rng.choice([8, 64]))
    elif kind == "profile":
        case.update(calls=rng.randint(1, 4), substitutions=rng.randint(0, 60))
    elif kind == "serve":
        case.update(requests=_log_uniform(rng, 16, 256))
    elif kind == "planner":
        case.update(rows=30_000, genes=0, nulls=0.0, samples=_log_uniform(rng, 128, 100_000))
    return case


# ---- partitions ----

_partitions = OrderedDict()  # the partitions opened last, as a service keeps them open


def _partition(case):
    key = (case["rows"], case["genes"], case["nulls"])
    if key not in _partitions:
        while len(_partitions) >= 3:
            _partitions.popitem(last=False)
        table = R.Table.generate(case["rows"], seed=TABLE_SEED, genome_len=GENOME, n_aa_genes=case["genes"],
                                 null_fraction=case["nulls"])
        _partitions[key] = (table, R.Device(table, 0))
    _partitions.move_to_end(key)
    return _partitions[key]


def _queries(table, n, seed, genes, leaves=0):
    if leaves:
        return table.queries(n, seed=seed, max_depth=4, max_nof_children=max(8, leaves), max_leaves=leaves,
                             use_aa=genes > 0, use_metadata=True)
    return table.queries(n, seed=seed, use_aa=genes > 0, use_metadata=True)


# ---- states ----

def prepare(case, seed):
    kind, qseed = case["kind"], 1000 + seed
    table, dev = _partition(case)
    s = {"kind": kind, "table": table, "dev": dev, "column": case.get("column", 0)}
    rng = np.random.default_rng([seed, 7])
    if kind in ("count", "rowset", "mutations"):
        # trees that select some of the rows, not none or all (about 70% of the generated ones do)
        n = case["calls"]
        found = _queries(table, 16 + 8 * n, qseed, case["genes"], case.get("leaves", 0))
        s["queries"] = [q for q in found if 0 < dev.count(q) < table.n_rows][:n]
    elif kind == "resident":
        rows = np.zeros(table.n_chunks * R.CHUNK_ROWS, np.uint8)
        rows[:table.n_rows] = rng.random(table.n_rows) < case["density"]
        col = table.columns[s["column"]]
        bits = np.packbits(rows, bitorder="little").view(np.int32)
        s["filter"] = torch.from_numpy(bits.copy()).cuda()
        s["cardinality"] = torch.tensor([int(rows.sum())], dtype=torch.int64, device="cuda")
        s["counts"] = torch.empty(col.n_symbols, col.L, dtype=torch.int32, device="cuda")
        s["status"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    elif kind == "batch_rows":
        n, every = case["queries"], case["mut_every"]
        s["queries"] = _queries(table, n, qseed, case["genes"])
        s["actions"] = np.array([1 if i % every == every - 1 else 0 for i in range(n)], np.int32)
        s["columns"] = np.zeros(n, np.uint32)
        s["min_props"] = np.full(n, MIN_PROPORTION)
        s["rows"] = np.zeros(ROWS_PER_QUERY * max(1, int(s["actions"].sum())), R.Device.ROW_DTYPE)
    elif kind == "batch":
        s["queries"] = _queries(table, case["queries"], qseed, case["genes"], case["leaves"])
    elif kind == "profile":
        row = int(rng.integers(table.n_rows))
        seq = workloads.profile_query_sequence(table, row=row, substitutions=case["substitutions"], seed=seed)
        s["queries"] = [f"MutProfile(main,{d},{seq})" for d in (200, 50, 5, 0)[:case["calls"]]]
    elif kind == "aggregate":
        s["queries"] = _queries(table, 4, qseed, case["genes"])
        # a filter of a good part of the rows: a span of dates or a random tree
        s["queries"].append("DateBetween(date,18300,%d)" % (18400 + 10 * int(rng.integers(40))))
        s["queries"] = [q.encode() for q in s["queries"]]
        s["dims"] = (R.AggDimension * 2)(R.AggDimension(0, 0, 1 + int(rng.integers(GENOME))), R.AggDimension(1, 0, 0))
        s["groups"] = np.zeros((len(s["queries"]), GROUPS, 2), np.int32)
        s["counts"] = np.zeros((len(s["queries"]), GROUPS), np.uint64)
        s["n"] = np.zeros((len(s["queries"]), 2), np.int64)
    elif kind == "serve":
        n = case["requests"]
        s["queries"] = _queries(table, n, qseed, case["genes"])
        s["mix"] = rng.permutation(([0] * 14 + [1] * 5 + [2]) * (n // 20 + 1))[:n].tolist()
        s["rows"] = np.zeros(ROWS_PER_QUERY * n, R.Device.ROW_DTYPE)
        s["ids"] = np.zeros(1000 * n, np.uint32)
        s["server"] = R.Server(dev, max_batch=512, streams=3)
    elif kind == "planner":
        s.update(_samples(case["samples"], seed))
        model = R.PlannerModel()
        model.weights[:] = s["w"].tolist()
        model.feature_mean[:] = [0.0] * R.PLANNER_FEATURES
        model.feature_std[:] = [1.0] * R.PLANNER_FEATURES
        model.target_std[:] = [1.0, 1.0]
        model.accepted = 1
        s["dev"] = R.Device(table, 0)  # a handle of its own: it keeps this state's weights
        s["dev"].planner_import(model)
    else:
        raise ValueError(kind)
    return s


def _samples(n, seed):
    """Weights as the network is initialised (He-normal, small biases) and normalised samples."""
    rng = np.random.default_rng([seed, 11])
    w = np.concatenate([rng.normal(0, math.sqrt(2 / 24), 64 * 24), rng.normal(0, 0.1, 64),
                        rng.normal(0, math.sqrt(2 / 64), 64 * 64), rng.normal(0, 0.1, 64),
                        rng.normal(0, math.sqrt(1 / 64), 2 * 64), rng.normal(0, 0.1, 2)]).astype(np.float32)
    return {"w": w, "x": rng.normal(size=(n, 24)).astype(np.float32), "t": rng.normal(size=(n, 2)).astype(np.float32)}


# The caller's result buffers hold this many Mutations rows a query and groups an aggregation.
ROWS_PER_QUERY, GROUPS = 1000, 17 * 201


def _keep(buffer, values):
    buffer[:len(values)] = values
    return len(values)


def _row_fields(rows):
    return {"position": rows["position"], "from": rows["from_"].view(np.uint8), "to": rows["to"].view(np.uint8),
            "count": rows["count"], "coverage": rows["coverage"], "proportion": rows["proportion"]}


def run(s):
    dev, kind = s["dev"], s["kind"]
    if kind == "count":
        return np.array([dev.count(q) for q in s["queries"]], np.int64)
    if kind == "rowset":
        return [dev.compute_filter(q) for q in s["queries"]]
    if kind == "mutations":
        return [dev.mutations(q, s["column"]) for q in s["queries"]]
    if kind == "resident":
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        dev.mutations_noalloc(s["column"], s["filter"].data_ptr(), s["cardinality"].data_ptr(), s["counts"].data_ptr(),
                              s["status"].data_ptr(), stream)
        return s["counts"], s["status"]
    if kind == "batch_rows":
        counts, rows, begin, count = dev.batch_rows(s["queries"], s["actions"], s["columns"], s["min_props"])
        return counts, _keep(s["rows"], rows), _row_fields(s["rows"]), begin, count
    if kind == "batch":
        return dev.batch(s["queries"])[0]
    if kind == "profile":
        return np.array([dev.count(q) for q in s["queries"]], np.int64)
    if kind == "aggregate":
        # the C-ABI call into the caller's buffers: groups (symbol and value ids) and their counts
        n, filtered = ctypes.c_size_t(), ctypes.c_uint64()
        for i, q in enumerate(s["queries"]):
            rc = R.lib().rhy_aggregate(dev._h, q, s["dims"], 2, None, s["groups"][i].ctypes.data,
                                       s["counts"][i].ctypes.data, GROUPS, ctypes.byref(n), ctypes.byref(filtered))
            if rc:
                raise R.RhyError(rc, R.lib().rhy_last_error().decode())
            s["n"][i] = n.value, filtered.value
        return s["n"], s["groups"], s["counts"]
    if kind == "serve":
        srv = s["server"]
        ids = [srv.submit(q, a, 0, MIN_PROPORTION, 1000) for q, a in zip(s["queries"], s["mix"])]
        got = [srv.result(i) for i in ids]
        _keep(s["rows"], np.concatenate([g["rows"] for g in got]))
        _keep(s["ids"], np.concatenate([g["ids"] for g in got]))
        return {"counts": np.array([(g["count"], len(g["rows"]), len(g["ids"])) for g in got], np.int64),
                "rows": _row_fields(s["rows"]), "ids": s["ids"]}
    if kind == "planner":
        grad, loss, y = dev.mlp_gradient(s["w"], s["x"], s["t"])
        selectivity, cost = dev.planner_predict(s["x"])
        return {"grad": grad, "loss": loss, "y": y, "selectivity": selectivity, "cost": cost}
    raise ValueError(kind)


# ---- what a pass cannot do without ----

# stored bytes of the nucleotide column per row: container payloads, boundary events of the covered
# regions and missing intervals, and the row index (substitutions and boundaries, 4 bytes each)
ROW_PAYLOAD, ROW_EVENTS, ROW_INDEX = 46, 16, 130
LEAF = 0.16        # payload bytes per row of a generated tree's mean leaf
LEAVES = 10        # leaves of a mean generated tree
AA_PAYLOAD = 20    # all amino-acid columns together


def work(case):
    kind, rows = case["kind"], case["rows"]
    column = ROW_PAYLOAD + ROW_EVENTS
    table = 16 * GENOME * 4
    image = rows * (column + (AA_PAYLOAD if case["genes"] else 0))
    tree = rows * LEAF * (case.get("leaves") or LEAVES)
    flops = 0
    if kind == "count":
        nbytes = case["calls"] * (tree + 8)
    elif kind == "rowset":
        nbytes = case["calls"] * (tree + rows / 8)
    elif kind == "mutations":  # about half of the filters take few rows
        share = 0.5 if case["column"] == 0 else 0.05
        nbytes = case["calls"] * (share * rows * column + table * share * 2)
    elif kind == "resident":
        share = 1.0 if case["column"] == 0 else 0.1
        nbytes = share * (min(rows * column, rows * case["density"] * ROW_INDEX) + table) + rows / 8
    elif kind == "batch_rows":
        nbytes = image + case["queries"] * 400
    elif kind == "batch":
        nbytes = min(image, case["queries"] * tree) + case["queries"] * 8
    elif kind == "profile":
        nbytes = case["calls"] * rows * (ROW_INDEX + 4 + 1 / 8)
    elif kind == "aggregate":
        nbytes = 5 * (tree / 2 + 0.3 * rows * ROW_INDEX)
    elif kind == "serve":
        nbytes = image + case["requests"] * 400
    else:
        nbytes = case["samples"] * (24 + 2 + 2) * 4
        flops = case["samples"] * 2 * 5760 * 4  # gradient: three products per layer; prediction: one
    return {"bytes": nbytes, "flops": flops}


# ---- 64-bit results of the planner network ----

def _bf16(w):
    u = w.view(np.uint32).astype(np.uint64)
    return ((u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32).astype(np.float64)


def exact(case, seed):
    """The network with BF16 weights in float64; every other workload's outputs are whole numbers
    (and quotients of two of them, which a plain evaluation of the filters would take too long for)."""
    if case["kind"] != "planner":
        return None
    s = _samples(case["samples"], seed)
    w, x, t = _bf16(s["w"]), s["x"].astype(np.float64), s["t"].astype(np.float64)
    w1, b1, w2 = w[:1536].reshape(64, 24), w[1536:1600], w[1600:5696].reshape(64, 64)
    b2, w3, b3 = w[5696:5760], w[5760:5888].reshape(2, 64), w[5888:]
    h1 = np.maximum(x @ w1.T + b1, 0)
    h2 = np.maximum(h1 @ w2.T + b2, 0)
    y = h2 @ w3.T + b3
    n = len(x)
    d3 = 2 * (y - t) / n
    d2 = (d3 @ w3) * (h2 > 0)
    d1 = (d2 @ w2) * (h1 > 0)
    grad = np.concatenate([(d1.T @ x).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), (d3.T @ h2).ravel(),
                           d3.sum(0)])
    # the selectivity starts from a rule estimate in the features: no value here
    return {"grad": grad, "loss": float(((y - t) ** 2).sum() / n), "y": y, "selectivity": None,
            "cost": np.exp(y[:, 1])}
