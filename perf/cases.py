"""Performance cases of the hash map and of the DOK tensor on one GPU: small calls, ordinary ones and the largest.

Each case is one unit of work of a program that uses the package through its public entry points, with the sizes of
`bench_configs.py`, of the benchmark's per-GPU shard, or generic ones.  A case is a dict of plain values:

  kind "lookup"   one `get` batch
       "churn"    `get`, `set` and drop-in `remove` of one batch of Zipf-distributed ids, table at a steady load
       "stream"   `set`, `get` and `remove_rows` of batches without equal keys, load stationary
       "build"    a new table: `set` of all rows, `get`, `remove` of a quarter, `get` again
       "grow"     a default-sized table that batches of new rows make grow (rehash)
       "gather"   `t[I, J]` on a 2-D tensor
       "assign"   `t[I, J] = v` and the selection read back
       "block"    `t[i0, :m, i2, mask]` on a 4-D tensor
       "lines"    a row read, a column written and read back on a small 2-D tensor
       "convert"  `from_dense` and `to_dense`
       "host"     `get`, `set` and `remove_rows` on pinned host buffers through `HostBatch`

Outputs are copies of stored bytes, flags and counts, so everything is compared exactly."""
import math

import numpy as np
import torch

from doksparse_b200 import CudaClosedHashmap, SparseDOKTensor
from doksparse_b200.host_batch import HostBatch

DEVICE = "cuda:0"
DTYPES = {"i64": torch.int64, "i32": torch.int32, "i16": torch.int16, "u8": torch.uint8, "f64": torch.float64,
          "f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
BYTES = {"i64": 8, "i32": 4, "i16": 2, "u8": 1, "f64": 8, "f32": 4, "f16": 2, "bf16": 2}


def listed():
    return [
        # a service that looks a request's few ids up: launch and host latency are all there is
        {"name": "lookup_1k", "kind": "lookup", "rows": 1000, "buckets": 65536, "load": 0.5, "hits": 0.9,
         "key": "i64", "key_cols": 1, "value": "f32", "value_cols": 2},
        # the same service updating its table between requests
        {"name": "churn_2k", "kind": "churn", "rows": 2000, "buckets": 65536, "load": 0.6, "threshold": 0.75,
         "value": "f32", "value_cols": 4},
        # cache-like churn at a high load: 64 M operations a batch, 70 % get, 20 % set, 10 % remove, 2^28 buckets
        {"name": "churn_64m_load09", "kind": "churn", "rows": 64000000, "buckets": 1 << 28, "load": 0.9, "threshold": 0.95,
         "value": "f32", "value_cols": 4},
        # one GPU's shard of the sharded 2^31-key table with its share of a 2^28-row batch
        {"name": "stream_32m_shard", "kind": "stream", "rows": 1 << 25, "keys": 1 << 28, "load": 0.6, "hits": 0.8,
         "key": "i64", "key_cols": 1, "value": "f32", "value_cols": 2},
        # points with float coordinates and a wide payload, built, queried and thinned out once
        {"name": "build_1m_f32x3", "kind": "build", "rows": 1000000, "buckets": 1 << 21, "hits": 0.5,
         "key": "f32", "key_cols": 3, "value": "i64", "value_cols": 5},
        # a vocabulary that is filled batch by batch, its size not known beforehand
        {"name": "grow_300k", "kind": "grow", "rows": 300000, "batches": 8, "key": "i64", "key_cols": 1,
         "value": "f32", "value_cols": 1},
        # 10 M stored elements in 10^5 x 10^5: a batch of pairs, nearly all of them misses
        {"name": "gather_4m_2d", "kind": "gather", "extent": 100000, "nnz": 10000000, "rows": 4000000, "hits": 0.001,
         "value": "f32"},
        # a batch of updates of the same tensor
        {"name": "assign_4m_2d", "kind": "assign", "extent": 100000, "nnz": 10000000, "rows": 4000000, "hits": 0.25,
         "value": "f32", "scalar": False},
        # advanced indexing of a 4-D tensor with slice and mask
        {"name": "block_4d_50m", "kind": "block", "d0": 4096, "d1": 2048, "d2": 512, "d3": 8, "nnz": 50000000,
         "n0": 256, "m1": 64, "n2": 128, "value": "f32"},
        # interactive work on a small matrix
        {"name": "lines_1000", "kind": "lines", "height": 1000, "width": 1000, "nnz": 20000, "value": "f32"},
        # a pruned weight matrix into the dictionary form and back
        {"name": "convert_8192", "kind": "convert", "height": 8192, "width": 8192, "density": 0.01, "value": "f32"},
        # a data pipeline whose keys and results live in host memory
        {"name": "host_4m", "kind": "host", "rows": 1 << 22, "keys": 1 << 24, "load": 0.6, "hits": 0.8,
         "value": "f32", "value_cols": 2},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm; odd more often than round."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["lookup", "churn", "stream", "build", "grow", "gather", "assign", "block", "lines", "convert", "host"])
    case = {"kind": kind}
    if kind in ("lookup", "stream", "build", "grow"):
        key, cols = rng.choice([("i64", 1), ("i64", 1), ("i64", 2), ("i64", 3), ("i32", 1), ("i32", 2), ("i32", 4), ("f32", 3), ("f32", 4)])
        value, width = rng.choice([("f32", 1), ("f32", 2), ("f32", 4), ("i64", 1), ("i64", 5), ("f16", 1), ("f16", 8), ("bf16", 3), ("f64", 2), ("i32", 3), ("u8", 5)])
        case.update(key=key, key_cols=cols, value=value, value_cols=width)
    if kind == "lookup":
        rows = _spread(rng, 1, 8000000)
        case.update(rows=rows, buckets=_spread(rng, 1 << 14, 1 << 26), load=round(rng.uniform(0.2, 0.85), 3), hits=round(rng.uniform(0, 1), 3))
    elif kind == "churn":
        rows = _spread(rng, 500, 16000000)
        load = round(rng.uniform(0.3, 0.7), 3)
        case.update(rows=rows, buckets=_spread(rng, max(1 << 14, rows), 1 << 26), load=load, threshold=0.75,
                    value=rng.choice(["f32", "f16", "i64"]), value_cols=rng.choice([1, 2, 4]))
    elif kind == "stream":
        keys = _spread(rng, 1 << 16, 1 << 27)
        case.update(rows=_spread(rng, 1 << 12, max(1 << 13, keys // 8)), keys=keys, load=round(rng.uniform(0.3, 0.65), 3), hits=round(rng.uniform(0.5, 0.95), 3))
    elif kind == "build":
        rows = _spread(rng, 2000, 4000000)
        case.update(rows=rows, buckets=int(rows / rng.uniform(0.2, 0.7)), hits=round(rng.uniform(0.1, 0.9), 3))
    elif kind == "grow":
        case.update(rows=_spread(rng, 5000, 4000000), batches=rng.randint(3, 12))
    elif kind in ("gather", "assign"):
        extent = _spread(rng, 1000, 1000000)
        nnz = _spread(rng, 1000, min(20000000, extent * extent // 4))
        case.update(extent=extent, nnz=nnz, rows=_spread(rng, 16, 8000000), hits=round(rng.uniform(0, 0.9), 3), value=rng.choice(["f32", "f32", "f16", "i64", "f64"]))
        if kind == "assign":
            case["scalar"] = rng.random() < 0.3
    elif kind == "block":
        d = [_spread(rng, 16, 4096), _spread(rng, 8, 2048), _spread(rng, 8, 512), _spread(rng, 2, 8)]
        case.update(d0=d[0], d1=d[1], d2=d[2], d3=d[3], nnz=_spread(rng, 500, max(501, min(20000000, math.prod(d) // 8))),
                    n0=_spread(rng, 1, 256), m1=rng.randint(1, min(64, d[1])), n2=_spread(rng, 1, 128), value=rng.choice(["f32", "f16", "i64"]))
    elif kind == "lines":
        h, w = _spread(rng, 50, 20000), _spread(rng, 50, 20000)
        case.update(height=h, width=w, nnz=_spread(rng, 100, min(2000000, h * w // 4)), value=rng.choice(["f32", "f16", "i64"]))
    elif kind == "convert":
        case.update(height=_spread(rng, 16, 8192), width=_spread(rng, 16, 8192), density=round(10 ** rng.uniform(-3, -1), 4), value=rng.choice(["f32", "f16", "bf16", "f64", "i32"]))
    else:
        case.update(rows=_spread(rng, 1 << 12, 1 << 22), keys=_spread(rng, 1 << 18, 1 << 25), load=round(rng.uniform(0.3, 0.65), 3),
                    hits=round(rng.uniform(0.5, 0.95), 3), value="f32", value_cols=rng.choice([1, 2, 4]))
    return case


# ---------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------

def _mix(x, bits):
    """A bijection of [0, 2^bits): different counters give different, scattered ids."""
    mask, half = (1 << bits) - 1, bits // 2
    x = (x * 0x2545F4914F6CDD1D) & mask
    x = x ^ (x >> half)
    x = (x * 0x1B03738712FAD5C9) & mask
    return x ^ (x >> (half + 1))


def _keys(counter, dtype, cols):
    """Key rows of the given counters: pairwise different for different counters.  Float columns hold whole numbers below
    2^24, as coordinates on a grid do (the map converts key elements by value)."""
    bits = {("i32", 1): 31}.get((dtype, cols), 62)
    m = _mix(counter, bits)
    if cols == 1:
        return m[:, None].to(DTYPES[dtype]).contiguous()
    width = -(-bits // cols)
    return torch.stack([(m >> (width * j)) & ((1 << width) - 1) for j in range(cols)], dim=1).to(DTYPES[dtype]).contiguous()


def _values(gen, n, dtype, cols):
    dt = DTYPES[dtype]
    if dt.is_floating_point:
        return torch.randn(n, cols, generator=gen, device=DEVICE, dtype=torch.float32).to(dt)
    return torch.randint(0, 100 if dtype == "u8" else 1 << 30, (n, cols), generator=gen, device=DEVICE).to(dt)


def _generator(seed):
    np.random.seed(seed & 0x7FFFFFFF)          # the map draws its hash parameters from numpy's global state
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _zipf(gen, n, support, s=0.99):
    """n ids in [0, support) with P(k) about (k + 1)^-s, by the inverse of the continuous distribution."""
    u = torch.rand(n, generator=gen, device=DEVICE, dtype=torch.float64)
    top = (support + 1.0) ** (1 - s)
    return ((1 + u * (top - 1)).pow_(1 / (1 - s)) - 1).long().clamp_(0, support - 1)


def _sample(gen, below, n):
    """n different counters below `below`: every `step`-th one from a random start."""
    step = 7919
    while math.gcd(step, below) != 1:
        step += 2
    start = int(torch.randint(0, below, (1,), generator=gen, device=DEVICE))
    return (torch.arange(n, device=DEVICE) * step + start) % below


def _filled(gen, buckets, n, key, key_cols, value, value_cols, threshold=0.75):
    """A table of `buckets` buckets that stores the keys of the counters 0 .. n - 1."""
    table = CudaClosedHashmap(n_buckets=buckets, device=DEVICE, rehash_threshold=threshold)
    for lo in range(0, n, 1 << 25):
        m = min(1 << 25, n - lo)
        table.set(_keys(torch.arange(lo, lo + m, device=DEVICE), key, key_cols), _values(gen, m, value, value_cols), assume_unique=True)
    return table


def _queries(gen, n, hits, stored):
    """n counters in random order, a share `hits` of them below `stored` and the others absent."""
    counters = torch.randint(0, stored, (n,), generator=gen, device=DEVICE)
    absent = torch.rand(n, generator=gen, device=DEVICE) >= hits
    return counters + absent * (1 << 29)


def _positions(gen, extents, n):
    return [torch.randint(0, e, (n,), generator=gen, device=DEVICE) for e in extents]


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    state = {"kind": kind}
    if kind in ("lookup", "build", "grow", "stream"):
        key, value = (case["key"], case["key_cols"]), (case["value"], case["value_cols"])
    if kind == "lookup":
        n = max(1, int(case["load"] * case["buckets"]))
        state["table"] = _filled(gen, case["buckets"], n, *key, *value, threshold=0.9)
        state["keys"] = _keys(_queries(gen, case["rows"], case["hits"], n), *key)
    elif kind == "churn":
        n, rows, value = int(case["load"] * case["buckets"]), case["rows"], (case["value"], case["value_cols"])
        state["table"] = _filled(gen, case["buckets"], n, "i64", 1, *value, threshold=case["threshold"])
        ids = _zipf(gen, rows, 8 * n)           # the most popular ids are the stored ones
        get, put = int(0.7 * rows), int(0.9 * rows)
        gone = _sample(gen, n, max(1, min(n, (rows - put) // 2)))
        gone = torch.cat([gone, gone])[:rows - put][torch.randperm(min(rows - put, 2 * gone.numel()), generator=gen, device=DEVICE)]
        state["get"], state["set"], state["remove"] = (_keys(part, "i64", 1) for part in (ids[:get], ids[get:put], gone))
        state["values"] = _values(gen, put - get, *value)
    elif kind == "stream":
        n, rows = case["keys"], case["rows"]
        state["table"] = _filled(gen, int(n / case["load"]), n, *key, *value)
        new = rows // 5
        inserted = n + torch.arange(new, device=DEVICE)
        order = torch.randperm(rows, generator=gen, device=DEVICE)
        state["set"] = _keys(torch.cat([_sample(gen, n, rows - new), inserted])[order], *key)
        state["values"] = _values(gen, rows, *value)
        state["get"] = _keys(_queries(gen, rows, case["hits"], n + new), *key)
        state["remove"] = _keys(inserted, *key)
    elif kind == "build":
        rows = case["rows"]
        state["buckets"] = case["buckets"]
        state["keys"], state["values"] = _keys(torch.arange(rows, device=DEVICE), *key), _values(gen, rows, *value)
        state["get"] = _keys(_queries(gen, rows, case["hits"], rows), *key)
        state["remove"] = _keys(_sample(gen, rows, rows // 4), *key)
    elif kind == "grow":
        keys = _keys(torch.randperm(case["rows"], generator=gen, device=DEVICE), *key)
        values = _values(gen, case["rows"], *value)
        state["batches"] = list(zip(keys.chunk(case["batches"]), values.chunk(case["batches"])))
        state["keys"] = keys
    elif kind in ("gather", "assign"):
        extents = (case["extent"], case["extent"])
        stored = _positions(gen, extents, case["nnz"])
        state["tensor"] = SparseDOKTensor(extents, torch.stack(stored), _values(gen, case["nnz"], case["value"], 1)[:, 0], device=DEVICE)
        known = torch.randint(0, case["nnz"], (case["rows"],), generator=gen, device=DEVICE)
        hit = torch.rand(case["rows"], generator=gen, device=DEVICE) < case["hits"]
        state["at"] = tuple(torch.where(hit, s[known], p) for s, p in zip(stored, _positions(gen, extents, case["rows"])))
        if kind == "assign":
            state["values"] = 1.0 if case["scalar"] else _values(gen, case["rows"], case["value"], 1)[:, 0]
    elif kind == "block":
        extents = (case["d0"], case["d1"], case["d2"], case["d3"])
        stored = _positions(gen, extents, case["nnz"])
        stored[0] = _zipf(gen, case["nnz"], case["d0"], 1.1)
        state["tensor"] = SparseDOKTensor(extents, torch.stack(stored), _values(gen, case["nnz"], case["value"], 1)[:, 0], device=DEVICE)
        i0, i2 = (torch.randint(0, e, (n,), generator=gen, device=DEVICE) for e, n in ((case["d0"], case["n0"]), (case["d2"], case["n2"])))
        mask = torch.zeros(case["d3"], dtype=torch.bool, device=DEVICE)
        mask[torch.randperm(case["d3"], generator=gen, device=DEVICE)[:(case["d3"] + 1) // 2]] = True
        state["at"] = (i0[:, None, None], slice(0, case["m1"]), i2[None, :, None], mask)
    elif kind == "lines":
        extents = (case["height"], case["width"])
        stored = _positions(gen, extents, case["nnz"])
        state["tensor"] = SparseDOKTensor(extents, torch.stack(stored), _values(gen, case["nnz"], case["value"], 1)[:, 0], device=DEVICE)
        state["row"], state["column"] = (int(torch.randint(0, e, (1,), generator=gen, device=DEVICE)) for e in extents)
        state["values"] = _values(gen, case["height"], case["value"], 1)[:, 0]
    elif kind == "convert":
        n, dt = case["height"] * case["width"], DTYPES[case["value"]]
        dense = _values(gen, n, case["value"], 1)[:, 0]
        dense *= (torch.rand(n, generator=gen, device=DEVICE) < case["density"]).to(dt)
        state["dense"] = dense.reshape(case["height"], case["width"])
    else:
        n, rows, value = case["keys"], case["rows"], (case["value"], case["value_cols"])
        table = _filled(gen, int(n / case["load"]), n, "i64", 1, *value, threshold=0.9)
        state["batch"] = HostBatch(table, DEVICE)
        new = min(rows, n) // 5
        inserted = n + torch.arange(new, device=DEVICE)
        put = torch.cat([_sample(gen, n, min(rows, n) - new), inserted])
        get = _queries(gen, rows, case["hits"], n + new)
        host = lambda x: x.cpu().pin_memory()
        found, values = torch.zeros(rows, dtype=torch.bool), torch.zeros(rows, case["value_cols"], dtype=DTYPES[case["value"]])
        state["out"] = (values.pin_memory(), found.pin_memory(), torch.zeros(new, dtype=torch.bool).pin_memory())
        values, found, removed = state["out"]
        state["operations"] = [("set", host(_keys(put, "i64", 1)), host(_values(gen, put.numel(), *value))),
                               ("get", host(_keys(get, "i64", 1)), values, found),
                               ("remove_rows", host(_keys(inserted, "i64", 1)), removed)]
    return state


# ---------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "lookup":
        return state["table"].get(state["keys"])
    if kind == "churn":
        table = state["table"]
        table.set(state["set"], state["values"])
        values, found = table.get(state["get"])
        return values, found, table.remove(state["remove"])
    if kind == "stream":
        table = state["table"]
        table.set(state["set"], state["values"])
        values, found = table.get(state["get"])
        return values, found, table.remove_rows(state["remove"])
    if kind == "build":
        table = CudaClosedHashmap(n_buckets=state["buckets"], device=DEVICE)
        table.set(state["keys"], state["values"])
        first = table.get(state["get"])
        removed = table.remove(state["remove"])
        return first, removed, table.get(state["get"]), table.n_elements
    if kind == "grow":
        table = CudaClosedHashmap(device=DEVICE)
        for keys, values in state["batches"]:
            table.set(keys, values)
        return table.get(state["keys"]), table.n_elements
    if kind in ("gather", "block"):
        return state["tensor"][state["at"]]
    if kind == "assign":
        state["tensor"][state["at"]] = state["values"]
        return state["tensor"][state["at"]]
    if kind == "lines":
        tensor = state["tensor"]
        row = tensor[state["row"]]
        tensor[:, state["column"]] = state["values"]
        return row, tensor[:, state["column"]]
    if kind == "convert":
        return SparseDOKTensor.from_dense(state["dense"]).to_dense()
    state["batch"].begin()
    state["batch"].run(state["operations"])
    state["batch"].join()
    torch.cuda.current_stream().synchronize()          # the results are used on the host
    return state["out"]


# ---------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------

TAG = 8          # bytes that identify a stored row


def work(case):
    """Batch rows read and written once, and per row the stored bytes it has to touch: the tag of the key, the value of a
    hit or of a written row, the key of an inserted one."""
    kind = case["kind"]
    v = BYTES[case["value"]] * case.get("value_cols", 1)
    k = BYTES[case["key"]] * case["key_cols"] if "key" in case else 8
    get = lambda n, hits, kb: n * (kb + TAG + hits * v + v + 1)
    put = lambda n, new, kb: n * (kb + v + TAG + v + new * kb)
    drop = lambda n, kb: n * (kb + TAG + TAG + 1)
    if kind == "lookup":
        total = get(case["rows"], case["hits"], k)
    elif kind == "churn":
        total = get(0.7 * case["rows"], 0.85, 8) + put(0.2 * case["rows"], 0.1, 8) + drop(0.1 * case["rows"], 8)
    elif kind in ("stream", "host"):
        rows = min(case["rows"], case["keys"]) if kind == "host" else case["rows"]
        total = get(case["rows"], case["hits"], k) + put(rows, 0.2, k) + drop(0.2 * rows, k)
    elif kind == "build":
        total = put(case["rows"], 1, k) + 2 * get(case["rows"], case["hits"], k) + drop(case["rows"] / 4, k)
    elif kind == "grow":
        total = put(case["rows"], 1, k) + get(case["rows"], 1, k)
    elif kind == "gather":
        total = case["rows"] * (16 + TAG + v + case["hits"] * v)
    elif kind == "assign":
        total = case["rows"] * (2 * (16 + TAG + v) + 2 * v)
    elif kind == "block":
        total = case["n0"] * case["m1"] * case["n2"] * ((case["d3"] + 1) // 2) * (TAG + v)
    elif kind == "lines":
        total = (2 * case["height"] + case["width"]) * (TAG + v) + 2 * case["height"] * v
    else:
        n = case["height"] * case["width"]
        total = 2 * n * v + 2 * case["density"] * n * (16 + TAG + v)
    return {"bytes": int(total), "flops": 0}


def tolerance(case):
    return "exact"
