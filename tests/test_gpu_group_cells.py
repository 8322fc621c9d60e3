"""Grouped aggregation in shared-memory cells and limb sums: group counts at
the edges of the modes, signs, row counts that fold the cells midway."""
import ctypes as C
import random

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle
from ultraprecise_b200 import abi, codec, prewarm, runtime
from ultraprecise_b200 import expr as E

pytestmark = pytest.mark.gpu

AGGS = [(abi.UP_AGG_SUM, 0), (abi.UP_AGG_AVG, 1), (abi.UP_AGG_COUNT, 1)]


def _raw(t):
    return bytes(t.cpu().numpy().tobytes())


# slots: 512 at p=18 (13 cells per group), 256 at p=38; register modes below 9 groups
@pytest.mark.parametrize("p", [5, 18, 38])
@pytest.mark.parametrize("groups,rows", [(1, 1), (8, 3000), (9, 30_011), (16, 4097), (17, 5000), (256, 20_000),
                                         (257, 20_000), (511, 10_000), (513, 10_000), (2049, 40_001)])
def test_group_counts_at_the_mode_edges(p, groups, rows):
    a, b = E.col(0), E.col(1)
    q = runtime.compile_query([a * b, a - b], AGGS, [E.ColType(p, 2)] * 2)
    cols = [runtime.gen_digits(rows, p, 7 + k) for k in range(2)]
    g = torch.Generator(device="cuda").manual_seed(groups)
    # skewed ids, the largest id present
    u = torch.rand(rows, device="cuda", generator=g)
    gid = (u ** 4 * groups).to(torch.int32).clamp_(max=groups - 1)
    gid[rows // 2] = groups - 1
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    outs = q.launch([runtime.DeviceColumn(t, p, 2) for t in cols], gid, groups, err=err)
    assert int(err.item()) == 0
    exp = oracle.query(q.built, q.aggs, [_raw(t) for t in cols], _raw(gid), rows, groups, threads=8)
    for k, (o, e) in enumerate(zip(outs, exp)):
        assert _raw(o) == e, f"aggregate {k}"


@pytest.mark.parametrize("groups", [12, 100_000])
def test_cells_fold_midway(groups):
    """More rows per CTA than the cells stay exact for (32768): values of one
    sign and full pieces, sums checked as int64."""
    rows, p = 24_000_000, 9
    q = runtime.compile_query([E.col(0)], [(abi.UP_AGG_SUM, 0), (abi.UP_AGG_COUNT, 0)], [E.ColType(p, 0)])
    v = torch.full((rows,), 0x3FFFFFF, dtype=torch.int64, device="cuda")  # 67108863: low piece 65535
    v -= torch.arange(rows, device="cuda") % 3
    raw = v.to(torch.int32).view(torch.uint8)
    assert codec.compact_bytes(p) == 4
    g = torch.Generator(device="cuda").manual_seed(3)
    gid = (torch.rand(rows, device="cuda", generator=g) ** 3 * groups).to(torch.int32).clamp_(max=groups - 1)
    outs = q.launch([runtime.DeviceColumn(raw, p, 0)], gid, groups)
    want = torch.zeros(groups, dtype=torch.int64, device="cuda").index_add_(0, gid.long(), v).cpu().numpy()
    img = outs[0].cpu().numpy().reshape(groups, abi.UP_AGG_DECIMAL_BYTES)
    got = img[:, 5:13].copy().view(np.int64).reshape(-1)
    assert np.array_equal(got, want) and not img[:, 13:].any() and not img[:, 1].any()
    cnt = outs[1].cpu().numpy().view(np.int64)
    assert np.array_equal(cnt, torch.bincount(gid.long(), minlength=groups).cpu().numpy())


def test_group_ids_out_of_range_are_flagged():
    rows, groups, p = 5000, 600, 18
    q = runtime.compile_query([E.col(0) * E.col(1), E.col(0)], AGGS, [E.ColType(p, 2)] * 2)
    cols = [runtime.gen_digits(rows, p, 3 + k) for k in range(2)]
    gid = torch.arange(rows, device="cuda", dtype=torch.int32) % groups
    gid[17], gid[18] = groups, -1
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    q.launch([runtime.DeviceColumn(t, p, 2) for t in cols], gid, groups, err=err)
    assert int(err.item()) == 4  # UP_ROWERR_DOMAIN


@pytest.mark.parametrize("threads", [32, 96, 256])
def test_cells_of_other_cta_sizes(threads):
    """Query kernels compiled for other CTA sizes: replicated cells, one cell
    per group, hashed cells."""
    rng = random.Random(threads)
    p, s, rows = 18, 4, 3001
    b = E.derive_types(E.build([E.col(0) * E.col(1), E.col(0)], [E.ColType(p, s)] * 2))
    aggs = [(abi.UP_AGG_SUM, b.roots[0]), (abi.UP_AGG_AVG, b.roots[1]), (abi.UP_AGG_COUNT, b.roots[1])]
    qa = (abi.UpQueryAgg * 3)(*aggs)
    lib, h = abi.load(), C.c_void_p()
    opts = abi.UpCompileOpts(0, threads, 0)
    abi.check(lib.up_query_compile(b.nodes, b.n_nodes, b.col_types, b.n_cols, qa, 3, C.byref(opts), C.byref(h)), "compile")
    raws = [codec.encode([(rng.getrandbits(1), rng.randrange(10 ** p)) for _ in range(rows)], p) for _ in range(2)]
    cols = [runtime.DeviceColumn.from_host(r, p, s) for r in raws]
    for groups in (9, 40, 300, 2000):
        gid = torch.tensor([rng.randrange(groups) for _ in range(rows)], dtype=torch.int32, device="cuda")
        outs = [torch.zeros(groups * w, dtype=torch.uint8, device="cuda") for w in (133, 133, 8)]
        arr = (abi.UpColumn * 2)(*[c.up_column() for c in cols])
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        abi.check(lib.up_query_launch(h, arr, 2, rows, gid.data_ptr(), groups, (C.c_void_p * 3)(*[o.data_ptr() for o in outs]),
                                      err.data_ptr(), torch.cuda.current_stream().cuda_stream), "launch")
        exp = oracle.query(b, aggs, raws, _raw(gid), rows, groups, threads=8)
        assert int(err.item()) == 0
        for k, (o, e) in enumerate(zip(outs, exp)):
            assert _raw(o) == e, (groups, k)
    lib.up_module_release(h)


@pytest.mark.parametrize("p", [9, 18, 38, 140])
@pytest.mark.parametrize("many", [False, True])
def test_group_counts_at_the_cells_edges(p, many):
    """One group less and more than each kernel's cells hold (read from the
    generated source), by group ids and by two-byte keys whose count stays on
    the device, with so few rows that the groups past the first kernel's are
    hashed and with enough for a cell each."""
    import re
    exprs, types = [E.col(0) * E.col(1), E.col(0)], [E.ColType(p, 2)] * 2
    src = prewarm.query_source(exprs, types, AGGS)
    slots = sorted(int(s) for s in re.findall(r"up_query_cells_body<(\d+), \d+, \d+, \d+>\(a, sm\)", src))
    pieces = int(re.search(r"constexpr int R = \d+, WP = (\d+), NLS", src).group(1))
    assert len(slots) == 2
    q = runtime.compile_query(exprs, AGGS, types)
    rng = np.random.default_rng(p)
    for groups in (slots[0], slots[0] + 1, slots[1], slots[1] + 1):
        rows = 2 ** 25 // max(pieces, 16) + 77 if many else groups + 3001
        cols = [runtime.DeviceColumn(runtime.gen_digits(rows, p, 7 + k), p, 2) for k in range(2)]
        ids = np.concatenate([np.arange(groups), (groups * rng.random(rows - groups) ** 3).astype(np.int64)]).astype(np.int32)
        gid = torch.from_numpy(rng.permutation(ids)).cuda()
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        outs = q.launch(cols, gid, groups, err=err)
        exp = oracle.query(q.built, q.aggs, [_raw(c.data) for c in cols], _raw(gid), rows, groups, threads=8)
        keys = [torch.stack([gid // 256, gid % 256], 1).to(torch.uint8).reshape(-1).contiguous()]
        table = torch.zeros(abi.UP_KEY_TABLE_ENTRIES, dtype=torch.int32, device="cuda")
        runtime.group_table_from_keys_async(keys, [2], table)
        got = q.launch_keys_async(cols, keys, [2], table, groups + 5, err=err, rows=rows)
        assert int(err.item()) == 0
        for k, e in enumerate(exp):
            assert _raw(outs[k]) == e and _raw(got[k])[:len(e)] == e, (groups, k)


@pytest.mark.parametrize("p", [5, 15, 38])
@pytest.mark.parametrize("rows", [1, 255, 2047, 30_001])
def test_columns_off_16_byte_boundaries(p, rows):
    """Columns, group ids and keys that bulk copies cannot take: each kernel's
    tiles copied in bytes, several per thread and the rest one by one."""
    a, b = E.col(0), E.col(1)
    q = runtime.compile_query([a * b, a - b], AGGS, [E.ColType(p, 2)] * 2)
    raws = [runtime.gen_digits(rows, p, 7 + k) for k in range(2)]
    rng = np.random.default_rng(rows)

    def off(t, shift):
        t = t.contiguous().view(torch.uint8)
        buf = torch.zeros(t.numel() + 16, dtype=torch.uint8, device="cuda")
        buf[shift:shift + t.numel()] = t
        return buf[shift:shift + t.numel()]

    cols = [runtime.DeviceColumn(off(t, 1 + 2 * k), p, 2) for k, t in enumerate(raws)]
    for groups in (3, 40, 3000):
        ids = rng.integers(0, groups, rows).astype(np.int32)
        gid = off(torch.from_numpy(ids).cuda(), 4).view(torch.int32)
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        outs = q.launch(cols, gid, groups, err=err)
        exp = oracle.query(q.built, q.aggs, [_raw(t) for t in raws], ids.tobytes(), rows, groups, threads=8)
        assert int(err.item()) == 0
        for k, e in enumerate(exp):
            assert _raw(outs[k]) == e, (groups, k)
        if groups == 40:
            keys = [off(torch.from_numpy((ids % 5).astype(np.uint8)).cuda(), 3)]
            table = torch.zeros(abi.UP_KEY_TABLE_ENTRIES, dtype=torch.int32, device="cuda")
            runtime.group_table_from_keys_async(keys, [1], table)
            kid, n, _ = runtime.group_ids_from_keys(keys, [1])
            got = q.launch_keys_async(cols, keys, [1], table, 8, err=err, rows=rows)
            exp = oracle.query(q.built, q.aggs, [_raw(t) for t in raws], _raw(kid), rows, n, threads=8)
            assert int(err.item()) == 0
            for k, e in enumerate(exp):
                assert _raw(got[k])[:len(e)] == e, k
