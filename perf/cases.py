"""Performance cases of the exact-decimal path: what a program that uses this
framework has it do, through the Python entry points over the C ABI.

Every case is one of these kinds:

  project    one JIT-compiled expression over resident columns
  query      GROUP BY over raw key bytes with SUM / AVG / COUNT of expressions
  group_sum  SUM / AVG / COUNT per int32 group id, up to 100 000 groups
  filter     a WHERE clause, the selected rows' indices, and an expression over them
  format     compact column -> decimal text in fixed-width slots
  parse      decimal text -> compact column
  series     sin(x) by its Taylor series on truncated decimals

Column values have every digit uniform (the precision sweep's columns) or, for
the money queries, the ranges of lineitem's quantity, price, discount and tax.
All outputs are bytes or whole numbers, and every operation is exact, so every
output has to be the same to the last bit.
"""
from __future__ import annotations

import math

import torch

from ultraprecise_b200 import abi, codec, runtime, workloads
from ultraprecise_b200 import expr as E

GROUP_CAPACITY = 64     # groups a keyed query's outputs have room for
FILTER_SCALE = 9


def listed():
    return [
        # a point query's expression over the few rows that are left: launch latency
        {"name": "project_small", "kind": "project", "op": "revenue", "p": 15, "s": 2, "rows": 1000, "nullable": False},
        # the precision sweep's narrow end: bound by memory
        {"name": "project_mad_p18", "kind": "project", "op": "mad", "p": 18, "s": 4, "rows": 16 << 20,
         "nullable": False},
        # a middle width, a row count that fills no last tile
        {"name": "project_mad_p76", "kind": "project", "op": "mad", "p": 76, "s": 19, "rows": 8_000_003,
         "nullable": False},
        # the sweep's widest product
        {"name": "project_mad_p600", "kind": "project", "op": "mad", "p": 600, "s": 150, "rows": 1 << 20,
         "nullable": False},
        # division at the SQL maximum of most engines
        {"name": "project_div_p38", "kind": "project", "op": "div", "p": 38, "s": 9, "rows": 16 << 20,
         "nullable": False},
        # long division of wide values
        {"name": "project_div_p300", "kind": "project", "op": "div", "p": 300, "s": 75, "rows": 2 << 20,
         "nullable": False},
        # the grouped money query (four groups of two CHAR(1) keys, eight aggregates)
        {"name": "query_money", "kind": "query", "values": "money", "p": 15, "keys0": 2, "keys1": 2,
         "rows": 64 << 20},
        # many groups with skewed sizes
        {"name": "group_sum_100k", "kind": "group_sum", "p": 18, "s": 4, "rows": 8 << 20, "groups": 100_000,
         "zipf": True},
        # WHERE a*b >= c AND a <> 0, then a*b+c of the rows that are kept
        {"name": "filter_p38", "kind": "filter", "p": 38, "s": FILTER_SCALE, "rows": 16 << 20},
        # result output and import of 38-digit values
        {"name": "format_p38", "kind": "format", "p": 38, "s": 9, "rows": 4 << 20},
        {"name": "parse_p38", "kind": "parse", "p": 38, "s": 9, "rows": 4 << 20},
        # the series at its smallest precision
        {"name": "series_p100", "kind": "series", "p": 100, "rows": 1 << 18},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("project", "project", "project", "query", "group_sum", "filter", "format", "parse", "series"))
    if kind == "project":
        op = rng.choice(("mad", "div", "revenue"))
        p = _log_int(rng, 6, 600)
        limbs = _limbs(_value_bits(p))
        cap = min(16 << 20, int(1.2e9 / (7 * 4 * limbs)), int(4.4e9 / (limbs * limbs)))
        return {"kind": kind, "op": op, "p": p, "s": min(p // 4, 150), "rows": _log_int(rng, 1000, cap),
                "nullable": rng.random() < 0.15}
    if kind == "query":
        return {"kind": kind, "values": rng.choice(("money", "money", "full")), "p": rng.randint(12, 18),
                "keys0": rng.randint(1, 7), "keys1": rng.randint(1, 7), "rows": _log_int(rng, 1000, 64 << 20)}
    if kind == "group_sum":
        return {"kind": kind, "p": rng.randint(9, 38), "s": rng.randint(0, 6), "rows": _log_int(rng, 1000, 8 << 20),
                "groups": _log_int(rng, 1, 100_000), "zipf": rng.random() < 0.5}
    if kind == "filter":
        p = rng.randint(9, 38)
        return {"kind": kind, "p": p, "s": min(FILTER_SCALE, p // 4), "rows": _log_int(rng, 1000, 16 << 20)}
    if kind in ("format", "parse"):
        p = _log_int(rng, 6, 120)
        return {"kind": kind, "p": p, "s": rng.randint(0, p // 2),
                "rows": _log_int(rng, 1000, min(4 << 20, (4 << 20) * 38 // p))}
    p = _log_int(rng, 30, 140)
    return {"kind": "series", "p": p, "rows": _log_int(rng, 1000, int((1 << 18) * min(1.0, (100 / p) ** 2)))}


# ------------------------------------------------------------------ inputs
def _value_bits(p):
    return (10 ** p - 1).bit_length()


def _limbs(bits):
    return max(1, (bits + 31) // 32)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _rand_column(rows, p, s, seed, nullable=False, nonzero=False):
    data = runtime.gen_digits(rows, p, seed, signed=True, nonzero=nonzero)
    if nullable:  # one value in twenty is NULL: flag byte 0 before the value
        flag = (torch.rand(rows, 1, device="cuda", generator=_generator(seed)) >= 0.05).to(torch.uint8)
        data = torch.cat([flag, data.view(rows, -1) * flag], 1).reshape(-1).contiguous()
    return runtime.DeviceColumn(data, p, s, nullable)


def _expression(op, p, s, nullable):
    a, b, c = E.col(0), E.col(1), E.col(2)
    if op == "div":
        return a / b, [E.ColType(p, s, nullable)] * 2
    if op == "revenue":
        return a * (E.dec("1.00") - b), [E.ColType(p, s, nullable)] * 2
    return a * b + c, [E.ColType(p, s, nullable)] * 3


def _error_word():
    return torch.zeros(1, dtype=torch.int32, device="cuda")


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed * 1009 + 17)


def _prepare_project(case, seed):
    p, s, rows, nullable = case["p"], case["s"], case["rows"], case["nullable"]
    e, types = _expression(case["op"], p, s, nullable)
    m = runtime.compile_expr(e, types)
    cols = [_rand_column(rows, p, s, seed + k, nullable, nonzero=case["op"] == "div" and k == 1)
            for k in range(len(types))]
    out = torch.zeros(rows * m.value_bytes, dtype=torch.uint8, device="cuda")
    return {"kind": "project", "m": m, "cols": cols, "rows": rows, "out": out, "err": _error_word()}


def _prepare_query(case, seed):
    p, rows = case["p"], case["rows"]
    exprs, aggs, _ = workloads.query_exprs()
    q = runtime.compile_query(exprs, aggs, [E.ColType(p, 2)] * 4)
    if case["values"] == "money":
        data = [runtime.gen_range(rows, p, *workloads.QUERY_RANGES[n], seed + k)
                for k, n in enumerate(("qty", "price", "disc", "tax"))]
    else:
        data = [runtime.gen_digits(rows, p, seed + k) for k in range(4)]
    g = _generator(seed)
    keys = [torch.randint(65, 65 + n, (rows,), dtype=torch.uint8, device="cuda", generator=g)
            for n in (case["keys0"], case["keys1"])]
    outs = [torch.zeros(GROUP_CAPACITY * (8 if k == abi.UP_AGG_COUNT else abi.UP_AGG_DECIMAL_BYTES),
                        dtype=torch.uint8, device="cuda") for k, _ in aggs]
    return {"kind": "query", "q": q, "cols": [runtime.DeviceColumn(t, p, 2) for t in data], "keys": keys,
            "table": torch.zeros(abi.UP_KEY_TABLE_ENTRIES, dtype=torch.int32, device="cuda"), "outs": outs,
            "err": _error_word(), "rows": rows}


def _prepare_group_sum(case, seed):
    p, s, rows, groups = case["p"], case["s"], case["rows"], case["groups"]
    a, b = E.col(0), E.col(1)
    aggs = [(abi.UP_AGG_SUM, 0), (abi.UP_AGG_AVG, 1), (abi.UP_AGG_COUNT, 1)]
    q = runtime.compile_query([a * b, a], aggs, [E.ColType(p, s)] * 2)
    u = torch.rand(rows, dtype=torch.float64, device="cuda", generator=_generator(seed))
    if case["zipf"]:
        cdf = torch.cumsum(torch.arange(1, groups + 1, dtype=torch.float64, device="cuda") ** -1.1, 0)
        gid = torch.searchsorted(cdf / cdf[-1], u, right=True)
    else:
        gid = (u * groups).to(torch.int64)
    gid = gid.clamp_(max=groups - 1).to(torch.int32)
    outs = [torch.zeros(groups * (8 if k == abi.UP_AGG_COUNT else abi.UP_AGG_DECIMAL_BYTES), dtype=torch.uint8,
                        device="cuda") for k, _ in aggs]
    return {"kind": "group_sum", "q": q, "cols": [_rand_column(rows, p, s, seed + k) for k in range(2)], "gid": gid,
            "groups": groups, "outs": outs, "err": _error_word()}


def _prepare_filter(case, seed):
    p, s, rows = case["p"], case["s"], case["rows"]
    a, b, c = E.col(0), E.col(1), E.col(2)
    types = [E.ColType(p, s)] * 3
    where = runtime.compile_expr((a * b).ge(c).and_(a.ne(E.dec("0"))), types)
    value = runtime.compile_expr(a * b + c, types)
    return {"kind": "filter", "where": where, "value": value, "rows": rows, "err": _error_word(),
            "cols": [_rand_column(rows, p, s, seed + k) for k in range(3)],
            "flags": torch.zeros(rows, dtype=torch.uint8, device="cuda"),
            "kept": torch.zeros(rows, dtype=torch.int32, device="cuda"),
            "count": torch.zeros(1, dtype=torch.int64, device="cuda"),
            "out": torch.zeros(rows * value.value_bytes, dtype=torch.uint8, device="cuda")}


def _prepare_format(case, seed):
    p, rows = case["p"], case["rows"]
    width = abi.load().up_format_width(p, 0)
    return {"kind": "format", "p": p, "s": case["s"], "rows": rows, "col": runtime.gen_digits(rows, p, seed),
            "text": torch.zeros(rows * width, dtype=torch.uint8, device="cuda"), "width": width,
            "lens": torch.zeros(rows, dtype=torch.int32, device="cuda")}


def _prepare_parse(case, seed):
    """The fields as a CSV holds them, one after the other: '-', digits, '.'."""
    p, s, rows = case["p"], case["s"], case["rows"]
    text, lens = runtime.format_decimal(runtime.gen_digits(rows, p, seed), rows, p, s)
    keep = torch.arange(text.shape[1], device="cuda")[None, :] < lens[:, None]
    offsets = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    offsets[1:] = torch.cumsum(lens.to(torch.int64), 0)
    return {"kind": "parse", "p": p, "s": s, "text": text[keep].contiguous(), "offsets": offsets}


def _prepare_series(case, seed):
    """x = sin's argument, uniform in (-1, 1) at full scale p-2."""
    p, rows = case["p"], case["rows"]
    e, types = workloads.sin_expr(p)
    m = runtime.compile_expr(e, types)
    narrow, b0, b1 = runtime.gen_digits(rows, p - 2, seed), codec.compact_bytes(p - 2), codec.compact_bytes(p)
    x = torch.zeros(rows, b1, dtype=torch.uint8, device="cuda")
    x[:, :b0] = narrow.view(rows, b0)
    sign = x[:, b0 - 1] & 128
    x[:, b0 - 1] -= sign
    x[:, b1 - 1] += sign
    return {"kind": "project", "m": m, "cols": [runtime.DeviceColumn(x.reshape(-1), p, p - 2)], "rows": rows,
            "out": torch.zeros(rows * m.value_bytes, dtype=torch.uint8, device="cuda"), "err": _error_word()}


# -------------------------------------------------------------------- runs
def run(state):
    return globals()["_run_" + state["kind"]](state)


def _run_project(st):
    return st["m"].launch(st["cols"], st["rows"], out=st["out"], err=st["err"]), st["err"]


def _run_query(st):
    runtime.group_table_from_keys_async(st["keys"], [1, 1], st["table"])
    outs = st["q"].launch_keys_async(st["cols"], st["keys"], [1, 1], st["table"], GROUP_CAPACITY, outs=st["outs"],
                                     err=st["err"], rows=st["rows"])
    return outs, st["table"][abi.UP_KEY_TABLE_COUNT:abi.UP_KEY_TABLE_COUNT + 1], st["err"]


def _run_group_sum(st):
    return st["q"].launch(st["cols"], st["gid"], st["groups"], outs=st["outs"], err=st["err"]), st["err"]


def _run_filter(st):
    flags = st["where"].launch(st["cols"], st["rows"], out=st["flags"], err=st["err"])
    abi.check(abi.load().up_filter_flags(flags.data_ptr(), st["rows"], st["kept"].data_ptr(), st["count"].data_ptr(),
                                         torch.cuda.current_stream().cuda_stream), "up_filter_flags")
    n = int(st["count"].item())
    cols = [runtime.DeviceColumn(c.data, c.precision, c.scale, indices=st["kept"][:n]) for c in st["cols"]]
    return st["kept"], st["count"], st["value"].launch(cols, n, out=st["out"], err=st["err"]), st["err"]


def _run_format(st):
    abi.check(abi.load().up_format_decimal(st["col"].data_ptr(), st["rows"], st["p"], st["s"], 0,
                                           st["text"].data_ptr(), st["width"], st["lens"].data_ptr(),
                                           torch.cuda.current_stream().cuda_stream), "up_format_decimal")
    return st["text"], st["lens"]


def _run_parse(st):
    return runtime.parse_decimal(None, st["p"], st["s"], text=st["text"], offsets=st["offsets"])


# ----------------------------------------------------- what a pass has to do
def work(case):
    """Bytes: each input byte read once, each output byte written once.
    Operations: a limb multiply-add counts two, as a fused multiply-add does."""
    kind, p, rows = case["kind"], case["p"], case["rows"]
    B, L = codec.compact_bytes(p), _limbs(_value_bits(p))
    if kind == "project":
        e, types = _expression(case["op"], p, case["s"], case["nullable"])
        b = E.derive_types(E.build([e], types))
        null = 1 if case["nullable"] else 0
        out_p = E.node_type(b, b.roots[0])[0]
        p10 = _limbs(_value_bits(case["s"] + (4 if case["op"] == "div" else 0)))
        madds = {"mad": L * L + L * p10, "div": L * p10 + (p10 + 1) * L, "revenue": L * (L + 1)}[case["op"]]
        return {"bytes": rows * (len(types) * (B + null) + codec.compact_bytes(out_p) + null), "flops": rows * 2 * madds}
    if kind == "query":
        return {"bytes": rows * (4 * B + 2), "flops": rows * 2 * (L * L + 2 * L * L)}
    if kind == "group_sum":
        return {"bytes": rows * (2 * B + 4) + case["groups"] * (2 * abi.UP_AGG_DECIMAL_BYTES + 8),
                "flops": rows * 2 * L * L}
    if kind == "filter":  # half of the rows are kept: their index, values and result
        out_b = codec.compact_bytes(2 * p + 1)
        return {"bytes": rows * (3 * B + 2) + rows // 2 * (8 + 3 * B + out_b), "flops": rows * 3 * L * L}
    if kind in ("format", "parse"):
        return {"bytes": rows * (B + p + 2 + (4 if kind == "format" else 8)), "flops": rows * L * L}
    steps = 2 * workloads.SIN_TERMS
    return {"bytes": rows * 2 * B, "flops": rows * 2 * steps * 2 * L * L}


def tolerance(case):
    return "exact"


# ------------------------------------------------------- the same, restated
def _decode(col):
    """(sign, magnitude) of every value: little-endian bytes, the sign in the last one's bit 7."""
    raw, width, out = col.data.cpu().numpy().tobytes(), col.value_bytes, []
    for i in range(0, len(raw), width):
        v = bytearray(raw[i:i + width])
        sign = v[-1] >> 7
        v[-1] &= 0x7F
        out.append((sign, int.from_bytes(v, "little")))
    return out


def exact(case, seed):
    """a*b+c and a*(1-b) of small projections in Python's integers."""
    if case["kind"] != "project" or case["op"] == "div" or case["nullable"] or case["rows"] > 20_000:
        return None
    st = prepare(case, seed)
    s, width = case["s"], st["m"].value_bytes
    out = bytearray()
    for row in zip(*(_decode(c) for c in st["cols"])):
        if case["op"] == "mad":
            (sa, a), (sb, b), (sc, c) = row
            x, y, sx, sy = a * b, c * 10 ** s, sa ^ sb, sc
            v = (-x if sx else x) + (-y if sy else y)
            sign, mag = (sx, x + y) if sx == sy else (int(v < 0), abs(v))
        else:
            (sa, a), (sb, b) = row
            sc = max(2, s)
            one, bb = 10 ** sc, b * 10 ** (sc - s)
            v = one - (-bb if sb else bb)
            sign, mag = sa ^ int(v < 0), a * abs(v)
        raw = bytearray(mag.to_bytes(width, "little"))
        raw[-1] |= sign << 7
        out += raw
    return torch.tensor(list(out), dtype=torch.uint8), torch.zeros(1, dtype=torch.int32)
