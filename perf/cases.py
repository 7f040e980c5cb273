"""The work that a user of this library has it do, as timed cases: fused
filter-aggregate and join queries on bit-packed fact tables, decode of every
scheme to memory or fused with a sum, decode of other lane widths and of the
tile-based run-length format, encoding with a fixed scheme or with the learned
selector, and batched queries.  Sizes and distributions are those of the
benchmark and of the Star Schema Benchmark at its scale factors.

    listed()            the cases that stand for the ranges below
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs on the GPU, encoded columns, tables, weights
    run(state)          one pass through the public entry points
    work(case)          bytes that one pass cannot do without
    exact(case, seed)   the outputs computed with plain torch, where they are numbers
"""
import math

import numpy as np
import torch

from fastlanesgpu_b200 import (LAYOUT_TRANSPOSED, ORDER_ORIGINAL, ORDER_STORED, SCHEME_CONST, SCHEME_DELTA,
                               SCHEME_DICT, SCHEME_FOR, SCHEME_RLE, datagen, ops)
from fastlanesgpu_b200._lib import MLP_N_PARAMS, lib
from fastlanesgpu_b200.batch import Batch
from fastlanesgpu_b200.column import (DeviceUniformColumn, RforColumn, encode_column_gpu, encode_column_learned_gpu,
                                      n_vectors)

SCHEMES = {"for": SCHEME_FOR, "delta": SCHEME_DELTA, "rle": SCHEME_RLE, "dict": SCHEME_DICT}
FAMILY_SCHEME = {"uniform": SCHEME_FOR, "zipf": SCHEME_DICT, "sorted_gaps": SCHEME_DELTA, "geometric_runs": SCHEME_RLE}
DEV = "cuda"


def listed():
    return [
        # A dashboard's query on a small table: one call, latency and launches count.
        {"name": "filter_small", "kind": "filter", "n": 60175},
        # The headline scan: SSB Q1.1's shape on 2^27 rows.
        {"name": "filter_large", "kind": "filter", "n": 1 << 27},
        # A whole star join at scale factor 1: the three hash tables, then probe and group-by.
        {"name": "q21_sf1", "kind": "q21", "n": 6001171},
        # Three large dimension tables (kept by the program), 4375 groups, scale factor 10's rows.
        {"name": "q31_sf10", "kind": "q31", "n": 59986214},
        # A table loader unpacking a column of mixed widths, about a row group at a time.
        {"name": "decode_for", "kind": "decode", "scheme": "for", "n": (1 << 20) + 333, "order": "stored"},
        # Sorted keys back in their original order, a whole large column.
        {"name": "decode_delta", "kind": "decode", "scheme": "delta", "n": (1 << 26) + 777, "order": "original"},
        # An aggregate over a skewed dictionary column without writing it out.
        {"name": "sum_dict", "kind": "sum", "scheme": "dict", "n": 50000017},
        # A column that was written by the reference's tile-based run-length encoder.
        {"name": "rfor", "kind": "rfor", "n": (1 << 24) + 777, "out": "hbm"},
        # 16-bit measures (quantities, codes) unpacked for a consumer of 16-bit values.
        {"name": "width_16", "kind": "width", "bits": 16, "bw": 11, "n": (1 << 26) + 5, "out": "hbm"},
        # Ingest of one low-cardinality attribute column as a dictionary.
        {"name": "encode_dict", "kind": "encode", "scheme": "dict", "n": 6001171},
        # Ingest of a table of unlike columns, the scheme of every vector picked by the network.
        {"name": "learned", "kind": "learned", "n": (1 << 25) + 99},
        # Many small aggregates over columns of uneven length in one call.
        {"name": "batch", "kind": "batch", "cols": 24, "queries": 96, "lo_log": 14, "hi_log": 22},
    ]


def draw(rng):
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    kind = rng.choice(["filter", "q21", "q31", "q41", "decode", "sum", "rfor", "width", "encode", "learned", "batch"])
    if kind == "filter":
        return {"kind": kind, "n": size(20000, 1 << 27)}
    if kind in ("q21", "q31", "q41"):
        return {"kind": kind, "n": size(60000, 6e7)}
    if kind == "decode":
        return {"kind": kind, "scheme": rng.choice(["for", "uniform", "delta", "rle", "dict"]), "n": size(1 << 16, 1 << 26),
                "order": rng.choice(["stored", "original"])}
    if kind == "sum":
        return {"kind": kind, "scheme": rng.choice(["for", "uniform", "delta", "rle", "dict"]), "n": size(1 << 16, 1 << 26)}
    if kind == "rfor":
        return {"kind": kind, "n": size(1 << 16, 1 << 24), "out": rng.choice(["hbm", "sum"])}
    if kind == "width":
        bits = rng.choice([8, 16, 64])
        return {"kind": kind, "bits": bits, "bw": rng.randint(1, {8: 8, 16: 16, 64: 48}[bits]),
                "n": size(1 << 16, (1 << 27) // (bits // 8)), "out": rng.choice(["hbm", "sum"])}
    if kind == "encode":
        return {"kind": kind, "scheme": rng.choice(["for", "delta", "rle", "dict"]), "n": size(1 << 16, 1 << 25)}
    if kind == "learned":
        return {"kind": kind, "n": size(1 << 18, 1 << 25)}
    hi = rng.randint(18, 23)
    return {"kind": kind, "cols": rng.randint(4, 32), "queries": rng.randint(16, 128), "lo_log": rng.randint(13, 16),
            "hi_log": hi}


# ------------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _ints(g, lo, hi, n):
    return torch.randint(lo, hi, (n,), generator=g, device=DEV, dtype=torch.int32)


def _widths(seed, n):
    """Bit width and base of every vector of the mixed-width column."""
    g = datagen.rng(seed)
    nv = n_vectors(n)
    return g.choice(np.array([3, 7, 11, 16, 21]), size=nv), g.integers(0, 1 << 20, size=nv)


def _uniform_bw(seed):
    return 1 + seed % 20


def _column(scheme, n, seed):
    """Values of a column as its scheme meets them (int32, on the GPU)."""
    if scheme == "for":  # a width and a base of its own for every vector
        w, b = (torch.from_numpy(x).to(DEV) for x in _widths(seed, n))
        v = torch.randint(0, 1 << 31, (w.numel(), 1024), generator=_gen(seed), device=DEV, dtype=torch.int64)
        return ((v & ((1 << w) - 1)[:, None]) + b[:, None]).reshape(-1)[:n].to(torch.int32)
    if scheme == "uniform":  # one width for the whole column, the reference's format
        return _ints(_gen(seed), 0, 1 << _uniform_bw(seed), n)
    if scheme == "delta":
        return datagen.sorted_geometric_device(n, seed=seed, device=DEV)
    if scheme == "rle":
        return datagen.geometric_runs_device(n, seed=seed, device=DEV)
    return datagen.zipf_device(n, seed=seed, device=DEV)


def _low_cardinality(n, seed):
    """Attribute codes: 250 values spread over 2^16 (city codes)."""
    g = _gen(seed)
    codes = torch.randperm(1 << 16, generator=g, device=DEV)[:250].to(torch.int32)
    return codes[_ints(g, 0, 250, n).long()]


def _packed(values, bw, bits=32):
    """FastLanes packing of values in [0, 2^bw) with torch: row r of a lane
    starts at bit r * bw of its stream, word k of lane l at (1024 / bits) k + l."""
    lanes, nv = 1024 // bits, n_vectors(values.numel())
    out = torch.zeros(nv, bw, lanes, dtype=torch.int64, device=DEV)
    for v0 in range(0, nv, 1 << 14):
        part = values[v0 * 1024:(v0 + (1 << 14)) * 1024].to(torch.int64)
        part = torch.nn.functional.pad(part, (0, -part.numel() % 1024)).view(-1, bits, lanes)
        o = out[v0:v0 + (1 << 14)]
        for r in range(bits):
            k, s = divmod(r * bw, bits)
            o[:, k] |= part[:, r] << s
            if s + bw > bits:
                o[:, k + 1] |= part[:, r] >> (bits - s)
    return out.view(-1).to({8: torch.uint8, 16: torch.int16, 32: torch.int32, 64: torch.int64}[bits])


def _uniform(values, bw):
    return DeviceUniformColumn(_packed(values, bw), values.numel(), bw)


Q11 = [("date", 12), ("discount", 4), ("quantity", 6), ("price", 24)]


def _q11_table(n, seed):
    g = _gen(seed)
    return {"date": _ints(g, 0, datagen.N_DAYS, n), "discount": _ints(g, 0, 11, n), "quantity": _ints(g, 1, 51, n),
            "price": _ints(g, 90000, 10500001, n)}


def _q11_filters(seed):
    y = seed % 7  # one of the seven years
    f = datagen.Q11_FILTER
    return [(0, int(datagen.YEAR_START[y]), int(datagen.YEAR_START[y + 1]) - 1), (1, *f["discount"]), (2, *f["quantity"])]


JOIN_COLS = {"q21": ["supp", "part", "date", "revenue"], "q31": ["supp", "cust", "date", "revenue"],
             "q41": ["supp", "cust", "part", "date", "revenue", "cost"]}
JOIN_BITS = {"supp": 17, "cust": 18, "part": 19, "date": 12, "revenue": 24, "cost": 18}


def _join_tables(kind, n, seed):
    """Fact columns, and per dimension its filter column and its payload."""
    g = _gen(seed)
    ids = {"supp": 1 << 17, "cust": 1 << 18, "part": 1 << 19, "date": datagen.N_DAYS}
    fact = {c: _ints(g, 90000, 10500001, n) if c == "revenue" else _ints(g, 50000, 150000, n) if c == "cost" else
            _ints(g, 1, ids[c], n) for c in JOIN_COLS[kind]}  # keys from 1: a table's empty slot holds 0
    year = torch.from_numpy(datagen.year_of_day(np.arange(datagen.N_DAYS))).to(DEV)
    s_nation, c_nation = _ints(g, 0, 25, ids["supp"]), _ints(g, 0, 25, ids["cust"])
    category, brand = _ints(g, 0, 5, ids["part"]), _ints(g, 0, 1000, ids["part"])
    if kind == "q21":  # name: (filter column, its ranges, payload)
        dims = {"supp": (s_nation, [(1, 1)], None), "part": (category, [(1, 1)], brand), "date": (None, None, year)}
    elif kind == "q31":
        dims = {"supp": (s_nation // 5, [(1, 1)], s_nation), "cust": (c_nation // 5, [(1, 1)], c_nation),
                "date": (year, [(1992, 1997)], year)}
    else:
        dims = {"supp": (s_nation // 5, [(1, 1)], None), "cust": (c_nation // 5, [(1, 1)], c_nation),
                "part": (category, [(0, 1)], None), "date": (None, None, year)}
    keys = {c: torch.arange(ids[c], dtype=torch.int32, device=DEV) for c in dims}
    return fact, dims, keys


JOIN_ARGS = {
    "q31": dict(agg_col=3, keys=[(0, 175, 2), (1, 7, 1), (2, 1, 0)], group_sub=1992, n_groups=datagen.Q31_GROUPS,
                res_stride=6, sum_slot=4),
    "q41": dict(agg_col=4, keys=[(1, 7, 1), (3, 1, 0)], group_sub=1992, n_groups=datagen.Q41_GROUPS, res_stride=4,
                sum_slot=2, agg_sub_col=5)}


def _build_tables(dims, keys):
    probes = []
    for i, (c, (filt, ranges, vals)) in enumerate(dims.items()):
        n = keys[c].numel()
        ht = ops.build_pht(keys[c], n, vals=vals, filt=filt, ranges=ranges)
        probes.append((i, ht, n, 0, 1 if vals is None else 2))
    return probes


def _selector_weights():
    """Weights that score a scheme by its estimated words per vector, linear in
    the statistics; DICT's weighed by its slower decode as the labels are."""
    w1, w2, w3 = torch.zeros(64, 16), torch.zeros(64, 64), torch.zeros(5, 64)
    w1[range(16), range(16)] = 1.0
    w2[range(16), range(16)] = 1.0
    w3[SCHEME_FOR, 0] = 1024.0                                            # range bits
    w3[SCHEME_DELTA, 1], w3[SCHEME_DELTA, 15] = 1024.0, 32.0              # delta bits
    w3[SCHEME_RLE, 2], w3[SCHEME_RLE, 15] = 512.0, 48.0                   # runs
    w3[SCHEME_CONST, 15], w3[SCHEME_CONST, 12] = 2048.0, -2048.0          # constant vector
    w3[SCHEME_DICT, 7], w3[SCHEME_DICT, 6] = 1.105 * 512.0, 1.105 * 640.0  # distinct bits, distinct values
    p = torch.cat([w1.flatten(), torch.zeros(64), w2.flatten(), torch.zeros(64), (-0.1 * w3).flatten(), torch.zeros(5)])
    assert p.numel() == MLP_N_PARAMS
    return p.to(DEV)


def _learned_columns(n, seed):
    n4 = n // 4
    return [_column(s, n4 + 37 * i, seed + i) for i, s in enumerate(["uniform", "dict", "delta", "rle"])]


def _batch_inputs(case, seed):
    cols = datagen.mixed_columns(case["cols"], case["lo_log"], case["hi_log"], seed=seed, device=DEV)
    g = datagen.rng(seed)
    queries = []
    for q in range(case["queries"]):
        c = q % len(cols)
        v = cols[c][1]
        lo, hi = sorted(int(v[int(i)]) for i in g.integers(0, v.numel(), size=2))
        queries.append((c, lo, hi, c))
    return cols, queries


def _width_values(case, seed):
    return torch.randint(0, 1 << case["bw"], (case["n"],), generator=_gen(seed), device=DEV, dtype=torch.int64)


def prepare(case, seed):
    kind, n = case["kind"], case.get("n")
    if kind == "filter":
        t = _q11_table(n, seed)
        return kind, [_uniform(t[c], bw) for c, bw in Q11], _q11_filters(seed), _long(1)
    if kind == "q21":  # the tables are built in the pass
        fact, dims, keys = _join_tables(kind, n, seed)
        return kind, [_uniform(fact[c], JOIN_BITS[c]) for c in JOIN_COLS[kind]], dims, keys
    if kind in ("q31", "q41"):
        fact, dims, keys = _join_tables(kind, n, seed)
        return kind, [_uniform(fact[c], JOIN_BITS[c]) for c in JOIN_COLS[kind]], _build_tables(dims, keys)
    if kind in ("decode", "sum"):
        v = _column(case["scheme"], n, seed)
        col = _uniform(v, _uniform_bw(seed)) if case["scheme"] == "uniform" else encode_column_gpu(v, SCHEMES[case["scheme"]])
        if kind == "sum":
            return kind, col, _long(1)
        order = ORDER_ORIGINAL if case["order"] == "original" else ORDER_STORED
        return kind, col, order, torch.empty(n_vectors(n) * 1024, dtype=torch.int32, device=DEV)
    if kind == "rfor":
        col = RforColumn.encode(_column("rle", n, seed).cpu().numpy()).to_device(DEV)
        return kind, col, torch.empty(n, dtype=torch.int32, device=DEV) if case["out"] == "hbm" else None, _long(1)
    if kind == "width":
        bits = case["bits"]
        packed = _packed(_width_values(case, seed), case["bw"], bits)
        out = torch.empty(n_vectors(n) * 1024, dtype=packed.dtype, device=DEV) if case["out"] == "hbm" else None
        return kind, packed, n, bits, case["bw"], _width_base(case), out, None if case["out"] == "hbm" else _long(1)
    if kind == "encode":
        v = _low_cardinality(n, seed) if case["scheme"] == "dict" else _column(case["scheme"], n, seed)
        return kind, v, SCHEMES[case["scheme"]], _store(n)
    if kind == "learned":
        cols = _learned_columns(n, seed)
        return kind, cols, _selector_weights(), [_store(v.numel()) for v in cols]
    cols, queries = _batch_inputs(case, seed)
    return kind, Batch([encode_column_gpu(v, FAMILY_SCHEME[f]) for f, v in cols], queries)


def _store(n):
    """The loader's own store of a column's words, as large as any encoding of n values."""
    return torch.zeros(int(lib().fls_encode_bound_words(n)), dtype=torch.int32, device=DEV)


def _stored(col, store):
    store[:col.payload_words].copy_(col.data[:col.payload_words])
    return store, col.meta


def _long(n):
    return torch.zeros(n, dtype=torch.int64, device=DEV)


def _width_base(case):
    return 3 if case["bits"] == 8 else 1000


def run(state):
    kind = state[0]
    if kind == "filter":
        return ops.query_filter_agg(state[1], state[2], agg_a=3, agg_b=1, out=state[3])
    if kind == "q21":
        return ops.probe_groupby(state[1], _build_tables(state[2], state[3]), 3, 1, 2, 7, 1992, datagen.N_GROUPS)
    if kind in ("q31", "q41"):
        return ops.join_groupby(state[1], state[2], **JOIN_ARGS[kind])
    if kind == "decode":
        return ops.unpack_global(state[1], state[2], out=state[3])
    if kind == "sum":
        return ops.query_aggregate(state[1], out=state[2])
    if kind == "rfor":
        _, col, out, total = state
        return ops.rfor_decode_sum(col, out=total) if out is None else ops.rfor_decode(col, out=out)
    if kind == "width":
        ops.decode_width_into(*state[1:])
        return state[6] if state[6] is not None else state[7]
    if kind == "encode":
        return _stored(encode_column_gpu(state[1], state[2], compact=False), state[3])
    if kind == "learned":  # every column enqueued before the first result is read back
        pending = [encode_column_learned_gpu(v, state[2], kappa=0.03, compact=False, defer=True) for v in state[1]]
        done = [p.finish() for p in pending]
        return [(*_stored(col, store), schemes, fallback) for (col, schemes, fallback), store in zip(done, state[3])]
    return state[1].run()


# -------------------------------------------------------- bytes of one pass

def work(case):
    kind, n = case["kind"], case.get("n")
    nv = n_vectors(n) if n else 0
    mean_bits = {"for": 11.6, "uniform": 10.5, "delta": 6.0, "rle": 2.4, "dict": 20.0}  # of the encoded columns
    if kind == "filter":
        return {"bytes": nv * 128 * 46 + 8}
    if kind in ("q21", "q31", "q41"):
        _, table = {"q21": (0, 1 << 22), "q31": (0, 3 << 20), "q41": (0, 5 << 20)}[kind]
        return {"bytes": nv * 128 * sum(JOIN_BITS[c] for c in JOIN_COLS[kind]) + table}
    if kind in ("decode", "sum"):
        return {"bytes": nv * 128 * mean_bits[case["scheme"]] + (4096 * nv if kind == "decode" else 8)}
    if kind == "rfor":
        return {"bytes": n / 4 + (4 * n if case["out"] == "hbm" else 8)}
    if kind == "width":
        return {"bytes": nv * 128 * case["bw"] + (nv * 128 * case["bits"] if case["out"] == "hbm" else 8)}
    if kind == "encode":
        return {"bytes": 4 * n + nv * (16 + 128 * {"for": 11.6, "delta": 6.0, "rle": 2.4, "dict": 12.0}[case["scheme"]])}
    if kind == "learned":
        return {"bytes": 4 * n + nv * (16 + 128 * 10)}
    lo, hi = case["lo_log"], case["hi_log"]  # lengths log-uniform in [2^lo, 2^hi], one read per column
    mean = (2 ** hi - 2 ** lo) / ((hi - lo) * math.log(2))
    return {"bytes": min(case["cols"], case["queries"]) * mean * 10 / 8}


# ------------------------------------------------------------ plain results

def _stored_order(v, layout):
    """Values padded to whole vectors with the last one, in a column's stored order (transpose.cpp:4110)."""
    v = torch.cat([v, v[-1:].expand(-v.numel() % 1024)]).view(-1, 1024)
    if layout == LAYOUT_TRANSPOSED:
        lane, row = torch.arange(32), torch.arange(32)[:, None]
        chunk = ((lane & 15) << 1) | (lane >> 4)
        step = 8 * torch.tensor([0, 2, 1, 3])[row & 3] + (row >> 2)
        v = v[:, (32 * chunk + step).reshape(-1).to(DEV)]
    return v.reshape(-1)


def _exact_join(kind, n, seed):
    fact, dims, _ = _join_tables(kind, n, seed)
    spec = JOIN_ARGS.get(kind) or dict(agg_col=3, keys=[(1, 7, 1), (2, 1, 0)], group_sub=1992, n_groups=datagen.N_GROUPS,
                                       res_stride=4, sum_slot=2)
    mask = torch.ones(n, dtype=torch.bool, device=DEV)
    for c, (filt, ranges, _) in dims.items():
        if filt is not None:
            lo, hi = ranges[0]
            mask &= ((filt >= lo) & (filt <= hi))[fact[c].long()]
    names = list(dims)
    group = torch.full((int(mask.sum()),), -spec["group_sub"], dtype=torch.int64, device=DEV)
    parts = []
    for q, mul, slot in spec["keys"]:
        p = dims[names[q]][2][fact[names[q]][mask].long()].long()
        group += p * mul
        parts.append((slot, p))
    group %= spec["n_groups"]
    cols = JOIN_COLS[kind]
    m = fact[cols[spec["agg_col"]]][mask].long()
    if "agg_sub_col" in spec:
        m -= fact[cols[spec["agg_sub_col"]]][mask].long()
    res = torch.zeros(spec["n_groups"], spec["res_stride"], dtype=torch.int32, device=DEV)
    for slot, p in parts:
        res[group, slot] = p.to(torch.int32)
    sums = _long(spec["n_groups"]).index_add_(0, group, m)
    res[:, spec["sum_slot"]:spec["sum_slot"] + 2] = sums.view(torch.int32).view(-1, 2)
    return res.reshape(-1)


def exact(case, seed):
    kind, n = case["kind"], case.get("n")
    if kind == "filter":
        t = _q11_table(n, seed)
        mask = torch.ones(n, dtype=torch.bool, device=DEV)
        for c, lo, hi in _q11_filters(seed):
            mask &= (t[Q11[c][0]] >= lo) & (t[Q11[c][0]] <= hi)
        return (t["price"][mask].long() * t["discount"][mask].long()).sum().view(1)
    if kind in JOIN_COLS:
        return _exact_join(kind, n, seed)
    if kind == "decode":
        v = _column(case["scheme"], n, seed)
        if case["scheme"] == "uniform":  # packed here, zeros past the last value
            return torch.nn.functional.pad(v, (0, -n % 1024))
        return _stored_order(v, None if case["order"] == "original" else LAYOUT_TRANSPOSED)
    if kind == "sum":
        return _column(case["scheme"], n, seed).sum(dtype=torch.int64).view(1)
    if kind == "rfor":
        v = _column("rle", n, seed)
        return v if case["out"] == "hbm" else v.sum(dtype=torch.int64).view(1)
    if kind == "width":
        bits = case["bits"]
        v = (_width_values(case, seed) + _width_base(case)) & ((1 << bits) - 1 if bits < 64 else -1)
        if case["out"] == "sum":
            return v.sum().view(1)
        v = torch.nn.functional.pad(v, (0, -n % 1024), value=_width_base(case))
        return v.to({8: torch.uint8, 16: torch.int16, 64: torch.int64}[bits])
    if kind == "batch":
        cols, queries = _batch_inputs(case, seed)
        res = []
        for c, lo, hi, a in queries:
            v = cols[c][1].long()
            mask = (v >= lo) & (v <= hi)
            res.append(torch.stack([cols[a][1].long()[mask].sum(), mask.sum()]))
        return torch.stack(res)
    return None  # encoders return words, not numbers
