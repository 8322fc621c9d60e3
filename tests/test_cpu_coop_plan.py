"""CPU: the shared memory that cooperative kernels ask for, over widths, group
sizes and expressions, from the generated sources: what a CTA may have, and
two CTAs per SM wherever a kernel's products on the tensor cores do not come in
twos."""
import random
import re

from ultraprecise_b200 import prewarm
from ultraprecise_b200 import expr as E

CTA_LIMIT = 232448      # bytes of shared memory a CTA may have (227 KB)
TWO_PER_SM = 113 * 1024


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
        if products == 1:
            assert smem <= TWO_PER_SM, (ps, tpv, smem)
        tensor += products > 0
    assert tensor > 100


def test_narrow_products_stay_on_the_window():
    """Operands and group sizes where the window product measured faster."""
    a, b, c = (E.col(i) for i in range(3))
    for p, e, tpvs in ((60, a * b * c, (2, 4, 8, 16)), (110, a * b * c, (2, 4, 8, 16)), (110, a * b + c * b, (2, 4, 8, 16)),
                       (220, a * b + c * b, (2, 4)), (200, a * b + c, (4, 8)), (300, (a + b) * (a - b), (4,))):
        for t in tpvs:
            assert _plan(e, [E.ColType(p, p // 4)] * 3, t)[1] == 0, (p, t)
    for p, e, tpvs in ((150, a * b * c, (16,)), (300, a * b + c, (8, 16)), (450, a * b + c, (32,)), (600, a * b + c, (16, 32))):
        for t in tpvs:
            assert _plan(e, [E.ColType(p, p // 4)] * 3, t)[1] > 0, (p, t)
