"""The register kernels' narrow rows: columns at and around the narrow bounds,
mixed with rows that need the general evaluation, against the oracle."""
import random

import pytest

torch = pytest.importorskip("torch")

from oracle import oracle
from ultraprecise_b200 import abi, codec, runtime
from ultraprecise_b200 import expr as E

pytestmark = pytest.mark.gpu


def _raw(t):
    return bytes(t.cpu().numpy().tobytes())


def _column(rows, p, rng, wide):
    """Values around every bound the narrow evaluation checks, of both signs."""
    top = 10 ** p - 1
    edges = [e for b in (20, 30, 31, 42, 47, 61, 62) for e in ((1 << b) - 1, 1 << b, (1 << b) + 1) if e <= top]
    out = []
    for _ in range(rows):
        if rng.random() < wide:
            m = rng.choice(edges + [top, 0]) if rng.random() < 0.5 else rng.randrange(top + 1)
        else:
            m = rng.randrange(min(top, 5_000_000) + 1)
        out.append((rng.getrandbits(1), m))
    return codec.encode(out, p)


def _exprs(kind):
    a, b, c = E.col(0), E.col(1), E.col(2)
    if kind == "money":
        d = a * (E.dec("1.00") - b)
        return [a, d, d * (E.dec("1.00") + c), -b]
    if kind == "sums":  # no product: columns up to 62 bits, three-word sums
        return [a, a - b, (a + b) + E.dec("-3.5")]
    return [a * a, a * b * c, E.lit(-7) * a]


@pytest.mark.parametrize("kind", ["money", "sums", "products"])
@pytest.mark.parametrize("p,groups,rows,wide", [(3, 1, 5, 0.0), (9, 4, 2051, 0.5), (12, 5, 4099, 0.02), (15, 7, 9001, 0.0),
                                                (15, 4, 9001, 1.0), (18, 3, 3000, 0.3), (20, 8, 1027, 0.3),
                                                (38, 6, 2500, 0.05)])
def test_narrow_and_wide_rows(kind, p, groups, rows, wide):
    rng = random.Random(p * 1000 + groups)
    exprs = _exprs(kind)
    aggs = [(abi.UP_AGG_SUM, i) for i in range(len(exprs))] + [(abi.UP_AGG_AVG, 0), (abi.UP_AGG_COUNT, 0)]
    q = runtime.compile_query(exprs, aggs, [E.ColType(p, min(2, p - 1))] * 3)
    raws = [_column(rows, p, rng, wide) for _ in range(3)]
    cols = [runtime.DeviceColumn.from_host(r, p, min(2, p - 1)) for r in raws]
    gid = torch.tensor([rng.randrange(groups) for _ in range(rows)], dtype=torch.int32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    outs = q.launch(cols, gid, groups, err=err)
    exp = oracle.query(q.built, q.aggs, raws, _raw(gid), rows, groups, threads=8)
    assert int(err.item()) == 0
    for k, (o, e) in enumerate(zip(outs, exp)):
        assert _raw(o) == e, f"aggregate {k}"
    # the same groups as one-byte, two-byte and 2 x one-byte keys
    for keys, kb in (([gid.to(torch.uint8)], [1]), ([torch.stack([gid % 3, gid], 1).to(torch.uint8).reshape(-1)], [2]),
                     ([(gid * 0 + 9).to(torch.uint8), gid.to(torch.uint8)], [1, 1])):
        kid, n, _ = runtime.group_ids_from_keys(keys, kb)
        table = torch.zeros(abi.UP_KEY_TABLE_ENTRIES, dtype=torch.int32, device="cuda")
        runtime.group_table_from_keys_async(keys, kb, table)
        got = q.launch_keys_async(cols, keys, kb, table, 64, err=err, rows=rows)
        exp = oracle.query(q.built, q.aggs, raws, _raw(kid), rows, n, threads=8)
        assert int(err.item()) == 0
        for k, (o, e) in enumerate(zip(got, exp)):
            assert _raw(o)[:len(e)] == e, f"keys {kb} aggregate {k}"


def test_register_sums_over_many_tiles():
    """More than 8192 tiles of 1024 rows for one CTA would take 2.4e9 rows; the
    sums of 64M rows of the largest two-word values are checked as int64."""
    rows, p = 1 << 26, 9
    q = runtime.compile_query([E.col(0) * E.col(1)], [(abi.UP_AGG_SUM, 0), (abi.UP_AGG_COUNT, 0)], [E.ColType(p, 0)] * 2)
    a = (torch.arange(rows, device="cuda", dtype=torch.int64) % 7 + 7_000_000).to(torch.int32)
    b = torch.full((rows,), 9_000, dtype=torch.int32, device="cuda")
    gid = (torch.arange(rows, device="cuda", dtype=torch.int32) % 3).to(torch.int32)
    outs = q.launch([runtime.DeviceColumn(t.view(torch.uint8), p, 0) for t in (a, b)], gid, 3)
    want = [int((a.long() * b.long())[gid == g].sum().item()) for g in range(3)]
    got = [d["mag"] for d in codec.decode_agg(_raw(outs[0]), 3)]
    assert got == want


@pytest.mark.parametrize("groups", [3, 7])
def test_columns_met_in_any_order(groups):
    """Expressions that meet their columns out of order or leave some out,
    columns of different precisions and scales, narrow and wide rows."""
    a, b, c, d = (E.col(i) for i in range(4))
    types = [(15, 2), (4, 1), (9, 4), (18, 0)]
    rows = 5003
    for exprs in ([b - a], [c * (E.dec("1.00") - a) + b], [c, c - a], [d * b, b - d], [d - c, b + a]):
        rng = random.Random(groups)
        aggs = [(abi.UP_AGG_SUM, i) for i in range(len(exprs))] + [(abi.UP_AGG_AVG, 0), (abi.UP_AGG_COUNT, 0)]
        q = runtime.compile_query(exprs, aggs, [E.ColType(p, s) for p, s in types])
        raws = [_column(rows, p, rng, 0.1) for p, _ in types]
        cols = [runtime.DeviceColumn.from_host(r, p, s) for r, (p, s) in zip(raws, types)]
        gid = torch.tensor([rng.randrange(groups) for _ in range(rows)], dtype=torch.int32, device="cuda")
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        outs = q.launch(cols, gid, groups, err=err)
        exp = oracle.query(q.built, q.aggs, raws, _raw(gid), rows, groups, threads=8)
        assert int(err.item()) == 0
        for k, (o, e) in enumerate(zip(outs, exp)):
            assert _raw(o) == e, f"aggregate {k}"


@pytest.mark.parametrize("p,word", [(9, torch.int32), (18, torch.int64)])
def test_register_sums_are_folded_several_times(p, word):
    """Two folds and more of the register sums in every CTA (each takes 256
    tiles of 1024 rows between them): sums of two words (products) and of three
    (values of 61 bits), of both signs, against the sums of one period."""
    period, times = 42, 16_000_000
    top = 10 ** p // 40 if word is torch.int32 else (1 << 59) - 1
    vals = [(-1) ** (i % 5) * (top - 7 * i) for i in range(period)]
    sign = 1 << (8 * codec.compact_bytes(p) - 1)
    raw = [v if v >= 0 else (-v | sign) - 2 * sign for v in vals]
    a = torch.tensor(raw, dtype=word, device="cuda").repeat(times)
    keys = [torch.tensor([i % 3 + 65 for i in range(period)], dtype=torch.uint8, device="cuda").repeat(times)]
    x = E.col(0)
    exprs = [x * E.lit(-31)] if word is torch.int32 else [x, -x + E.lit(1)]
    factor = [lambda v: -31 * v] if word is torch.int32 else [lambda v: v, lambda v: 1 - v]
    aggs = [(abi.UP_AGG_SUM, i) for i in range(len(exprs))] + [(abi.UP_AGG_COUNT, 0)]
    q = runtime.compile_query(exprs, aggs, [E.ColType(p, 0)])
    table = torch.zeros(abi.UP_KEY_TABLE_ENTRIES, dtype=torch.int32, device="cuda")
    runtime.group_table_from_keys_async(keys, [1], table)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    outs = q.launch_keys_async([runtime.DeviceColumn(a.view(torch.uint8), p, 0)], keys, [1], table, 4, err=err, rows=period * times)
    assert int(err.item()) == 0
    for k, f in enumerate(factor):
        got = [-d["mag"] if d["sign"] else d["mag"] for d in codec.decode_agg(_raw(outs[k])[:3 * abi.UP_AGG_DECIMAL_BYTES], 3)]
        assert got == [times * sum(f(v) for i, v in enumerate(vals) if i % 3 == g) for g in range(3)], k
    assert outs[-1].view(torch.int64)[:3].tolist() == [14 * times] * 3


@pytest.mark.parametrize("groups,keys", [(3, False), (7, False), (6, True)])
def test_runs_of_wide_and_narrow_tiles(groups, keys):
    """Tiles of wide rows, of narrow ones and of both in turn, several per CTA:
    after tiles of wide rows the kernels evaluate whole tiles the general way."""
    import numpy as np
    rng = np.random.default_rng(groups)
    rows, p = 2_400_000, 18
    tiles = rows // 1024 + 1
    kind = rng.integers(0, 3, tiles // 37 + 1).repeat(37)[:tiles].repeat(1024)[:rows]  # 0 narrow, 1 wide, 2 mixed
    wide = (kind == 1) | ((kind == 2) & (rng.random(rows) < 0.3))
    raws = []
    for _ in range(2):
        v = np.where(wide, rng.integers(0, 10 ** 18, rows), rng.integers(0, 1_000_000, rows)) * rng.choice([-1, 1], rows)
        raws.append(codec.np_compact_from_int64(v, p).tobytes())
    a, b = E.col(0), E.col(1)
    exprs = [a * b, b - a]
    aggs = [(abi.UP_AGG_SUM, 0), (abi.UP_AGG_AVG, 1), (abi.UP_AGG_COUNT, 0)]
    q = runtime.compile_query(exprs, aggs, [E.ColType(p, 2)] * 2)
    cols = [runtime.DeviceColumn.from_host(r, p, 2) for r in raws]
    gid = torch.from_numpy(rng.integers(0, groups, rows).astype(np.int32)).cuda()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    if keys:
        key = [gid.to(torch.uint8)]
        table = torch.zeros(abi.UP_KEY_TABLE_ENTRIES, dtype=torch.int32, device="cuda")
        runtime.group_table_from_keys_async(key, [1], table)
        outs = q.launch_keys_async(cols, key, [1], table, 8, err=err, rows=rows)
    else:
        outs = q.launch(cols, gid, groups, err=err)
    exp = oracle.query(q.built, q.aggs, raws, _raw(gid), rows, groups, threads=8)
    assert int(err.item()) == 0
    for k, (o, e) in enumerate(zip(outs, exp)):
        assert _raw(o)[:len(e)] == e, f"aggregate {k}"
