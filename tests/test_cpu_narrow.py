"""CPU: the generated narrow evaluation of grouped queries (up_qnarrow),
compiled for the host as the kernels call it, against Python integers: the
order in which an expression meets its columns, columns of different widths,
shared nodes."""
import ctypes as C
import os
import random
import re
import shutil
import subprocess

import pytest

from ultraprecise_b200 import abi, codec, prewarm
from ultraprecise_b200 import expr as E

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")

N_COLS = 5


def _built(roots, types):
    b = E.build(roots, types)
    return E.derive_types(b)


def _sum_aggs(n):
    return [(abi.UP_AGG_SUM, i) for i in range(n)]


def _host(tmp_path, sources):
    """One library with a function narrow_<k>(x, y) per query: x[column] in,
    y[root] out, returns what up_qnarrow does.  Signed overflow wraps, as the
    GPU's arithmetic does."""
    parts = ["typedef long long i64; typedef unsigned long long u64; typedef unsigned u32;\n#define UP_DI static inline\n"]
    for k, src in enumerate(sources):
        fn = re.search(r"UP_DI bool up_qnarrow\(.*?\n}\n", src, re.S).group(0)
        call = re.search(r"const bool ok = (up_qnarrow\(.*?\)) && bad == 0u;", src).group(1)
        names = re.findall(r"\b([xy]\d+)\b", call)
        decl = "".join(f" i64 {n}{' = x[' + n[1:] + ']' if n[0] == 'x' else ' = 0'};" for n in names)
        out = "".join(f" y[{n[1:]}] = {n};" for n in names if n[0] == "y")
        parts.append(f"namespace q{k} {{\n{fn}}}\nextern \"C\" bool narrow_{k}(const i64* x, i64* y) {{\n   {decl}\n"
                     f"    const bool ok = q{k}::{call};\n   {out}\n    return ok;\n}}\n")
    cpp, so = str(tmp_path / "narrow.cpp"), str(tmp_path / "narrow.so")
    with open(cpp, "w") as f:
        f.write("".join(parts))
    subprocess.run(["g++", "-std=c++17", "-O1", "-fwrapv", "-shared", "-fPIC", "-o", so, cpp], check=True)
    return C.CDLL(so)


def _scale(b, k):
    nd = b.nodes[k]
    return b.col_types[nd.column].scale if nd.kind == abi.UP_NODE_COLUMN else nd.scale


def _exact(b, row):
    """Every node's value at its own scale."""
    v = []
    for k in range(b.n_nodes):
        nd = b.nodes[k]
        if nd.kind == abi.UP_NODE_COLUMN:
            x = row[nd.column]
        elif nd.kind == abi.UP_NODE_CONST:
            x = sum(nd.const_limbs[i] << (32 * i) for i in range(nd.const_nlimbs)) * (-1 if nd.const_sign else 1)
        elif nd.kind == abi.UP_NODE_INT:
            x = nd.int_value
        elif nd.kind == abi.UP_NODE_MUL:
            x = v[nd.left] * v[nd.right]
        else:
            s = max(_scale(b, nd.left), _scale(b, nd.right))
            x, y = (v[i] * 10 ** (s - _scale(b, i)) for i in (nd.left, nd.right))
            x = x + y if nd.kind == abi.UP_NODE_ADD else x - y
        v.append(-x if nd.reverse else x)
    return v


def _check(lib, k, b, row):
    """True when the narrow evaluation takes the row; its values are then exact."""
    x, y = (C.c_longlong * N_COLS)(*row), (C.c_longlong * len(b.roots))()
    fn = getattr(lib, f"narrow_{k}")
    fn.restype = C.c_bool
    if not fn(x, y):
        return False
    v = _exact(b, row)
    for i, r in enumerate(b.roots):
        assert y[i] == v[r], (k, i, row, y[i], v[r])
    return True


def _col_bits(src):
    return int(re.search(r"quad_value<\d+, (\d+)>", src).group(1))


def test_columns_in_any_order(tmp_path):
    """Expressions that meet their columns out of order, one that leaves
    columns out, columns of different precisions and scales."""
    a, b, c, d, e = (E.col(i) for i in range(N_COLS))
    types = [E.ColType(15, 2), E.ColType(4, 1), E.ColType(9, 4), E.ColType(18, 0), E.ColType(7, 3)]
    queries = [[b - a], [c * (E.dec("1.00") - a) + b], [c - a, a], [e * d, d - b], [d - c, c - b, b - a], [E.lit(7) * c - a * e]]
    srcs = [prewarm.query_source(q, types, _sum_aggs(len(q))) for q in queries]
    lib = _host(tmp_path, srcs)
    rng = random.Random(1)
    for k, q in enumerate(queries):
        built = _built(q, types)
        taken = 0
        for _ in range(300):
            row = [rng.randint(-1000, 1000) for _ in types]
            taken += _check(lib, k, built, row)
        assert taken == 300


def _edge(rng, bits):
    """A value of at most `bits` bits, often next to a power of two."""
    k = rng.randint(0, bits)
    m = (1 << k) + rng.choice((-3, -1, 0, 0, 1, 3)) if rng.random() < 0.8 else rng.getrandbits(bits)
    return rng.choice((-1, 1)) * min(abs(m), (1 << bits) - 1)


def test_bounds_leave_both_ends_out(tmp_path):
    """Two operands checked to 30 bits whose sum is -2^31, negated: a row whose
    value an int does not hold is not taken."""
    x0, x1, x2, x3, x4 = (E.col(i) for i in range(N_COLS))
    types = [E.ColType(18, 0)] * N_COLS
    b, c, a = x0 + x1, x2 + x3, (x0 + x2) + x4
    roots = [a * b, a * c, -(b + c)]
    lib = _host(tmp_path, [prewarm.query_source(roots, types, _sum_aggs(3))])
    built = _built(roots, types)
    h = 1 << 29
    for x4v in (0, 1, 3, (1 << 30) - 1):
        for s in (-1, 1):
            for delta in (-1, 0, 1):
                _check(lib, 0, built, [s * h, s * h, s * h, s * h + delta, x4v])
    assert _check(lib, 0, built, [h, 1, -h, 5, 7])


def _random_query(rng):
    """Up to four sums over a pool of shared, sometimes negated nodes."""
    types = [E.ColType(p, rng.randint(0, min(4, p))) for p in (rng.choice((4, 9, 12, 15, 18)) for _ in range(N_COLS))]
    pool = [E.col(i) for i in range(N_COLS)] + [E.dec("1.00"), E.lit(-7)]
    for _ in range(rng.randint(2, 7)):
        x, y = rng.choice(pool), rng.choice(pool)
        n = rng.choice((x + y, x - y, x * y))
        pool.append(-n if rng.random() < 0.3 else n)
    return pool[-rng.randint(1, 4):], types


def test_random_nodes_at_their_bounds(tmp_path):
    rng = random.Random(5)
    queries, srcs = [], []
    while len(queries) < 120:
        roots, types = _random_query(rng)
        src = prewarm.query_source(roots, types, _sum_aggs(len(roots)))
        if "up_qnarrow" in src and "quad_value" in src:
            queries.append((_built(roots, types), types, _col_bits(src)))
            srcs.append(src)
    lib = _host(tmp_path, srcs)
    taken = 0
    for k, (built, types, bits) in enumerate(queries):
        for _ in range(400):
            row = [_edge(rng, min(bits, 8 * codec.compact_bytes(t.precision) - 1)) for t in types]
            taken += _check(lib, k, built, row)
    assert taken > 5000
