"""CPU: the shared memory that cooperative kernels ask for, over widths, group
sizes and expressions, from the generated sources: never more than a CTA may
have."""
import random
import re

from ultraprecise_b200 import prewarm
from ultraprecise_b200 import expr as E

CTA_LIMIT = 232448      # bytes of shared memory a CTA may have (227 KB)


def _plan(e, types, tpv):
    """(shared memory of up_expr_tile, tensor products in the source)"""
    src = prewarm.expr_source(e, types, tpv)
    m = re.search(r"valid, \(u32\*\)\(sm \+ (\d+)\) \+ \(threadIdx\.x >> 5\) \* (\d+)\);", src)
    return int(m.group(1)) + 8 * 4 * int(m.group(2)), len(re.findall(r"tpi_mul(?:_const)?<[^>]*>\([^;]*, ws\)", src))


def test_shared_memory_fits_a_cta():
    a, b, c, d = (E.col(i) for i in range(4))
    rng = random.Random(3)
    exprs = [a * b + c + d, a * b * c, a * b + c * d, (a + b) * (c - d), a * b, a * b * c * d, a * b + c]
    tensor = 0
    cases = [([202, 96, 202, 210], a * b + c + d, 2)]
    cases += [([rng.randint(5, 600) for _ in range(4)], rng.choice(exprs), rng.choice((2, 4, 8, 16, 32))) for _ in range(1500)]
    for ps, e, tpv in cases:
        types = [E.ColType(p, rng.randint(0, p // 2)) for p in ps]
        smem, products = _plan(e, types, tpv)
        assert smem <= CTA_LIMIT, (ps, tpv, smem)
        tensor += products > 0
    assert tensor > 100

