"""Products on the tensor cores (cooperative values) against one thread per
value: limb counts at the edges of the fragments' steps and tiles, all group
sizes, operands of unequal width, values of all nines and zeros."""
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle
from ultraprecise_b200 import codec, runtime
from ultraprecise_b200 import expr as E

pytestmark = pytest.mark.gpu


def _column(p, rows, seed):
    """Uniform digits with zeros, ones, all nines and long runs of ones bits among them."""
    B = codec.compact_bytes(p)
    t = runtime.gen_digits(rows, p, seed).view(rows, B)
    for r, v in ((0, 0), (1, 1), (2, 10 ** p - 1), (3, (1 << (3 * p)) - 1), (4, 10 ** p - 1), (5, (1 << (3 * p)) - (1 << 32))):
        if r < rows and v >= 0:
            raw = bytearray(v.to_bytes(B, "little"))
            raw[-1] |= (r & 1) << 7
            t[r] = torch.tensor(list(raw), dtype=torch.uint8)
    return t.reshape(-1).contiguous()


# a at precision p, b at q: 6 limbs (the shortest on the tensor cores), 8 and 9
# (a step of 32 bytes with 7 of shift), 16, 17, 32, 63 and 64 limbs
@pytest.mark.parametrize("p,q", [(57, 57), (58, 55), (77, 77), (85, 86), (153, 154), (163, 60), (300, 300), (300, 57),
                                 (308, 303), (600, 600), (606, 160)])
@pytest.mark.parametrize("rows", [1, 37, 1500])
def test_products_match_one_thread(p, q, rows):
    a, b = E.col(0), E.col(1)
    types = [E.ColType(p, 3), E.ColType(q, 30)]
    cols = [runtime.DeviceColumn(_column(p, rows, 3), p, 3), runtime.DeviceColumn(_column(q, rows, 4).view(rows, -1).flip(0)
                                                                               .reshape(-1).contiguous(), q, 30)]
    for name, e in (("mul", a * b), ("align", a * b - b * E.dec("-7") + a)):
        one = runtime.compile_expr(e, types, threads_per_value=1)
        err1 = torch.zeros(1, dtype=torch.int32, device="cuda")
        want = one.launch(cols, rows, err=err1)
        for tpv in (2, 4, 8, 16, 32):
            m = runtime.compile_expr(e, types, threads_per_value=tpv)
            err = torch.zeros(1, dtype=torch.int32, device="cuda")
            out = torch.full((rows * m.value_bytes + 64,), 0xEE, dtype=torch.uint8, device="cuda")
            m.launch(cols, rows, out=out[:rows * m.value_bytes], err=err)
            assert torch.equal(out[:rows * m.value_bytes], want), (name, tpv)
            assert bool((out[rows * m.value_bytes:] == 0xEE).all()) and int(err.item()) == int(err1.item())


# the shorter operand at the limbs from which products go to the tensor cores
# (6 at 32 threads per value, 16 at 16, 24 at 8, 28 in pairs at 4) and below
@pytest.mark.parametrize("p,q,tpvs", [(163, 57, (16, 32)), (163, 48, (16, 32)), (150, 154, (8, 16, 32)), (200, 143, (8, 16)),
                                      (300, 231, (8,)), (310, 216, (8, 16)), (260, 270, (4, 8)), (260, 255, (4,)), (600, 600, (16,))])
def test_products_match_the_oracle(p, q, tpvs):
    rows = 333
    a, b = E.col(0), E.col(1)
    types = [E.ColType(p, 3), E.ColType(q, 30)]
    raws = [_column(p, rows, 5), _column(q, rows, 6).view(rows, -1).flip(0).reshape(-1).contiguous()]
    cols = [runtime.DeviceColumn(t, ty.precision, ty.scale) for t, ty in zip(raws, types)]
    host = [bytes(t.cpu().numpy().tobytes()) for t in raws]
    for e in (a * b, a * b + b * a, a * b * E.dec("-7.5") + a):
        for tpv in tpvs:
            m = runtime.compile_expr(e, types, threads_per_value=tpv)
            err = torch.zeros(1, dtype=torch.int32, device="cuda")
            out = m.launch(cols, rows, err=err)
            exp, exp_err = oracle.eval_expr(m.built, m.root, host, rows, m.value_bytes)
            assert bytes(out.cpu().numpy().tobytes()) == exp and int(err.item()) == exp_err, tpv
