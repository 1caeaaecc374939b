"""The work that programs built on orq_b200 have it do, as measurable cases.

A case is one pass through the public Python API: the secret shares of its
inputs are on the GPU beforehand (a program holds shared columns and a
runtime), and the pass runs the oblivious operators on copies of them and
opens what such a program opens. Kinds:

  micro    AND, MULT, EQ, GR and RCA on two vectors (ORQ's micro_primitives)
  convert  sharing, b2a_bit, a2b, prefix sum and opening of one vector
  radix    radix_sort of a key column plus payload applies
  quick    quicksort of a key column plus payload applies
  bitonic  bitonic_sort of one key column
  groupby  group-by SUM and COUNT of a table (EncodedTable.aggregate)
  join     PK-FK inner join, product, group-by SUM and COUNT
  batch    many ragged sorts at once, half bitonic, half radix
"""
import numpy as np
import torch

import orq_b200 as orq
from orq_b200.table import EncodedTable

ASC, DESC = orq.ASC, orq.DESC
NP = {4: np.int32, 8: np.int64}


def listed():
    return [
        # a handful of rows: what a call costs by itself (launches, host path)
        {"name": "micro_1k_i32", "kind": "micro", "n": 1000, "width": 4},
        # ORQ's micro_primitives at its largest published size
        {"name": "micro_16m_i32", "kind": "micro", "n": 1 << 24, "width": 4},
        # share conversions and scans of an ordinary 64-bit column, odd length
        {"name": "convert_3m_i64", "kind": "convert", "n": 3000017, "width": 8},
        # a small table's sort: launch-bound
        {"name": "radix_1k_i32", "kind": "radix", "n": 1000, "width": 4, "bits": 32, "payloads": 1, "desc": False},
        # an ordinary table's sort, odd size, descending
        {"name": "radix_100k_i64", "kind": "radix", "n": 100003, "width": 8, "bits": 40, "payloads": 1, "desc": True},
        # a million rows: the size of the sampled CPU comparison
        {"name": "radix_1m_i64", "kind": "radix", "n": 1 << 20, "width": 8, "bits": 40, "payloads": 2, "desc": False},
        # the headline: 2^22 rows, 40-bit keys, two payloads
        {"name": "radix_4m_i64", "kind": "radix", "n": 1 << 22, "width": 8, "bits": 40, "payloads": 2, "desc": False},
        # the same rows by ORQ's default sort protocol
        {"name": "quick_4m_i64", "kind": "quick", "n": 1 << 22, "width": 8, "bits": 40, "payloads": 2, "desc": False},
        # the network sort of 2^16 32-bit keys
        {"name": "bitonic_64k_i32", "kind": "bitonic", "n": 1 << 16, "width": 4, "desc": False},
        # a group-by request of the serving mix (1024 groups), radix tables
        {"name": "groupby_60k_radix", "kind": "groupby", "n": 60000, "quick": False},
        # the join + group-by pipeline, quicksort tables
        {"name": "join_320k_quick", "kind": "join", "n": 1 << 16, "quick": True},
        # a ragged batch of independent sorts, lengths log-uniform
        {"name": "batch_24", "kind": "batch", "items": 24, "lo": 10, "hi": 18},
    ]


def _size(rng, lo, hi):
    """A length spread over the logarithm of [2^lo, 2^hi]; odd ones as often as not."""
    n = int(2.0 ** rng.uniform(lo, hi))
    return n | 1 if rng.random() < 0.5 else n


def draw(rng):
    kind = rng.choice(["micro", "convert", "radix", "radix", "quick", "bitonic", "groupby", "join", "batch"])
    width = rng.choice([4, 8])
    if kind == "micro":
        return {"kind": kind, "n": _size(rng, 10, 24 if width == 4 else 23), "width": width}
    if kind == "convert":
        return {"kind": kind, "n": _size(rng, 10, 22), "width": width}
    if kind in ("radix", "quick"):
        return {"kind": kind, "n": _size(rng, 10, 21.9), "width": width,
                "bits": rng.randint(8, 32 if width == 4 else 40),
                "payloads": rng.randint(0, 2), "desc": rng.random() < 0.25}
    if kind == "bitonic":
        return {"kind": kind, "n": 1 << rng.randint(10, 20), "width": width, "desc": rng.random() < 0.25}
    if kind == "groupby":
        return {"kind": kind, "n": _size(rng, 12, 17), "quick": rng.random() < 0.5}
    if kind == "join":
        return {"kind": kind, "n": _size(rng, 10, 15), "quick": rng.random() < 0.5}
    return {"kind": kind, "items": rng.randint(8, 24), "lo": 10, "hi": rng.randint(13, 18)}


# ---- inputs ----------------------------------------------------------------
def _uniform(rng, n, width, bits):
    """Keys uniform over `bits` bits (the whole signed range at full width)."""
    v = rng.integers(0, 1 << 63, size=n, dtype=np.uint64) << np.uint64(1)
    v ^= rng.integers(0, 1 << 63, size=n, dtype=np.uint64)
    if bits < 64:
        v &= np.uint64((1 << bits) - 1)
    return v.astype(np.uint32).view(np.int32) if width == 4 else v.view(np.int64)


def _plain(case, seed):
    """The plaintext inputs of a case."""
    rng = np.random.Generator(np.random.PCG64(seed))
    kind = case["kind"]
    if kind == "micro":
        x = _uniform(rng, case["n"], case["width"], 8 * case["width"])
        y = _uniform(rng, case["n"], case["width"], 8 * case["width"])
        y[::7] = x[::7]  # equal pairs, so that EQ and GR see both outcomes
        return x, y
    if kind == "convert":
        return (_uniform(rng, case["n"], case["width"], 8 * case["width"]),)
    if kind in ("radix", "quick"):
        key = _uniform(rng, case["n"], case["width"], case["bits"])
        return (key, *[_uniform(rng, case["n"], case["width"], 31) for _ in range(case["payloads"])])
    if kind == "bitonic":
        return (_uniform(rng, case["n"], case["width"], 8 * case["width"]),)
    if kind == "groupby":
        return rng.integers(0, 1024, case["n"]), rng.integers(0, 1000000, case["n"])
    if kind == "join":
        n = case["n"]
        w = 1.0 / np.arange(1, 10001, dtype=np.float64) ** 1.1
        cdf = np.cumsum(w) / w.sum()
        g = np.minimum(np.searchsorted(cdf, rng.random(n)), 9999).astype(np.int64)
        return (rng.permutation(n).astype(np.int64), g, rng.integers(0, 1000000, n),
                rng.integers(0, n, 4 * n), rng.integers(1, 51, 4 * n))
    sizes = _batch_sizes(case)
    keys = []
    for i, n in enumerate(sizes):
        k = _uniform(rng, n, 4, 32)
        if i % 2 == 0:  # bitonic items are padded to a power of two
            k = np.concatenate([k, np.full(_pow2(n) - n, np.iinfo(np.int32).max, np.int32)])
        keys.append(k)
    return tuple(keys)


def _pow2(n):
    return 1 << max(0, (n - 1).bit_length())


def _batch_sizes(case):
    """Lengths log-uniform over [2^lo, 2^hi), the same for every seed."""
    rng = np.random.Generator(np.random.PCG64(case["items"]))
    return [int(2.0 ** rng.uniform(case["lo"], case["hi"])) for _ in range(case["items"])]


def prepare(case, seed):
    data = _plain(case, seed)
    rt = orq.Runtime(seed=seed % (1 << 31) + 1)
    kind = case["kind"]
    s = {"case": case, "rt": rt}
    if kind == "micro":
        s["b"] = [rt.secret_share_b(data[0], 0), rt.secret_share_b(data[1], 1)]
        s["a"] = [rt.secret_share_a(data[0], 0), rt.secret_share_a(data[1], 1)]
    elif kind == "convert":
        s["x"] = torch.from_numpy(data[0]).cuda()
    elif kind in ("radix", "quick", "bitonic"):
        s["key"] = rt.secret_share_b(data[0], 0)
        s["payloads"] = [rt.secret_share_a(p, 0) for p in data[1:]]
    elif kind == "groupby":
        s["t"] = [_table(rt, case, {"[G]": data[0], "V": data[1]})]
    elif kind == "join":
        s["t"] = [_table(rt, case, {"[K]": data[0], "[G]": data[1], "V": data[2]}),
                  _table(rt, case, {"[K]": data[3], "Q": data[4]})]
    else:
        s["keys"] = [rt.secret_share_b(k, 0) for k in data]
    return s


def _protocol(case):
    return orq.SortingProtocol.QUICKSORT if case["quick"] else orq.SortingProtocol.RADIXSORT


def _table(rt, case, cols):
    return EncodedTable.secret_share(rt, list(cols.values()), list(cols), protocol=_protocol(case))


def _copy(t):
    """The table with columns of its own: operators work in place."""
    cols = {k: type(t[k])(t.rt, t[k].shares.clone()) for k in t.getColumnNames()}
    return EncodedTable(t.rt, cols, t.rows, protocol=t.protocol)


# ---- one pass --------------------------------------------------------------
def run(s):
    case, rt = s["case"], s["rt"]
    kind = case["kind"]
    if kind == "micro":
        (xb, yb), (xa, ya) = s["b"], s["a"]
        return {"and": (xb & yb).shares, "mult": (xa * ya).shares, "eq": (xb == yb).shares,
                "gr": (xb > yb).shares, "rca": (xb + yb).shares}
    if kind == "convert":
        b = rt.secret_share_b(s["x"], 0)
        a = rt.secret_share_a(s["x"], 1)
        bit = b.b2a_bit()
        ab = a.a2b()
        orq.prefix_sum(bit)
        return {"bits": bit.shares, "a2b": ab.shares, "ranks": bit.open(), "opened": ab.open()}
    if kind in ("radix", "quick"):
        key = s["key"].clone()
        order = DESC if case["desc"] else ASC
        perm = orq.radix_sort(key, order, case["bits"]) if kind == "radix" else orq.quicksort(key, order)
        out = {"key": key.shares, "perm": perm.shares, "opened": key.open()}
        for i, p in enumerate(s["payloads"]):
            p = p.clone()
            orq.oblivious_apply_elementwise_perm(p, perm)
            out["payload%d" % i] = p.shares
        return out
    if kind == "bitonic":
        key = s["key"].clone()
        orq.bitonic_sort(key, DESC if case["desc"] else ASC)
        return {"key": key.shares, "opened": key.open()}
    if kind == "batch":
        keys = [k.clone() for k in s["keys"]]
        orq.bitonic_sort_batch(keys[0::2], ASC)
        perms = orq.radix_sort_batch(keys[1::2], ASC, 32)
        return {"keys": [k.shares for k in keys], "perms": [p.shares for p in perms]}
    ag = orq.aggregators
    if kind == "groupby":
        t = _copy(s["t"][0])
        t.addColumns(["CNT"])
        t.aggregate(["[G]"], [("V", "V", ag.sum), ("CNT", "CNT", ag.count)])
    else:
        a, b = (_copy(t) for t in s["t"])
        t = a.inner_join(b, ["[K]"], [("[G]", "[G]", ag.copy), ("V", "V", ag.copy)])
        t.addColumns(["VQ", "CNT"])
        t["VQ"] = t["V"] * t["Q"]
        t.aggregate(["[G]"], [("VQ", "VQ", ag.sum), ("CNT", "CNT", ag.count)])
    return {k: {"shares": t[k].shares, "opened": t[k].open()} for k in t.getColumnNames()}


def exact(case, seed):
    """Opened values in 64 bits; shares are keystream and have no plain value."""
    kind = case["kind"]
    if kind not in ("convert", "radix", "quick", "bitonic"):
        return None
    data = _plain(case, seed)
    if kind == "convert":
        return {"bits": None, "a2b": None, "ranks": torch.from_numpy(np.cumsum(data[0] & 1).astype(data[0].dtype)),
                "opened": torch.from_numpy(data[0])}
    k = np.sort(data[0])
    out = {"key": None, "opened": torch.from_numpy(np.ascontiguousarray(k[::-1]) if case["desc"] else k)}
    if kind != "bitonic":
        out.update({"perm": None, **{"payload%d" % i: None for i in range(case["payloads"])}})
    return out


def work(case):
    """Shares are three arrays a vector: each read once, each result written once."""
    kind = case["kind"]
    if kind == "micro":
        return {"bytes": case["n"] * case["width"] * 3 * (4 + 5), "flops": 0}
    if kind == "convert":
        return {"bytes": case["n"] * case["width"] * (1 + 3 + 3 + 2), "flops": 0}
    if kind in ("radix", "quick"):
        w = case["width"]
        return {"bytes": case["n"] * (6 * w * (1 + case["payloads"]) + 12 + w), "flops": 0}
    if kind == "bitonic":
        return {"bytes": case["n"] * case["width"] * 7, "flops": 0}
    if kind == "groupby":
        return {"bytes": case["n"] * 8 * (3 * 3 + 4 * 4), "flops": 0}
    if kind == "join":
        return {"bytes": case["n"] * 8 * (4 * 3 + 4 * 3 * 3 + 5 * 8 * 4), "flops": 0}
    rows = sum(_pow2(n) if i % 2 == 0 else n for i, n in enumerate(_batch_sizes(case)))
    return {"bytes": rows * (24 + 6), "flops": 0}
