"""The generic expression kernel's word loads and staged results: every value
width class, column and output addresses off word boundaries, row indices,
NULLs, against the contiguous kernel's results of the same rows."""
import pytest

torch = pytest.importorskip("torch")

from ultraprecise_b200 import codec, runtime
from ultraprecise_b200 import expr as E

pytestmark = pytest.mark.gpu


def _shifted(t, shift):
    """The same bytes at `shift` bytes past a 256-byte boundary, the buffer ending with them."""
    buf = torch.zeros(shift + t.numel(), dtype=torch.uint8, device="cuda")
    buf[shift:] = t
    return buf[shift:]


@pytest.mark.parametrize("p", [1, 3, 5, 7, 9, 12, 15, 18, 20, 28, 38, 57, 76, 150, 300])
@pytest.mark.parametrize("shift,out_shift,rows", [(0, 0, 1000), (4, 1, 257), (8, 7, 256), (1, 0, 300), (2, 16, 31), (3, 5, 1)])
def test_indexed_rows_equal_contiguous_rows(p, shift, out_shift, rows):
    s = min(2, p - 1)
    a, b, c = E.col(0), E.col(1), E.col(2)
    m = runtime.compile_expr(a * b + c, [E.ColType(p, s)] * 3, threads_per_value=1)
    raw = [runtime.gen_digits(rows, p, 5 + k) for k in range(3)]
    whole = m.launch([runtime.DeviceColumn(t, p, s) for t in raw], rows).view(rows, -1)
    g = torch.Generator(device="cuda").manual_seed(rows)
    idx = torch.randint(0, rows, (2 * rows + 1,), device="cuda", generator=g).to(torch.int32)
    idx[0], idx[-1] = rows - 1, rows - 1  # the buffer's last bytes
    cols = [runtime.DeviceColumn(_shifted(t, shift), p, s, indices=idx) for t in raw]
    n = idx.numel()
    buf = torch.full((out_shift + n * m.value_bytes + 32,), 0xEE, dtype=torch.uint8, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    m.launch(cols, n, out=buf[out_shift:out_shift + n * m.value_bytes], err=err)
    got = buf[out_shift:out_shift + n * m.value_bytes].view(n, -1)
    assert int(err.item()) == 0 and torch.equal(got, whole[idx.long()])
    assert bool((buf[:out_shift] == 0xEE).all()) and bool((buf[out_shift + n * m.value_bytes:] == 0xEE).all())


@pytest.mark.parametrize("p", [3, 9, 12, 15, 16, 18, 38, 77])
@pytest.mark.parametrize("rows", [1, 255, 1025])
def test_nullable_rows(p, rows):
    s = min(2, p - 1)
    a, b = E.col(0), E.col(1)
    e = a * (E.dec("1.00") - b)
    raw = [runtime.gen_digits(rows, p, 9 + k) for k in range(2)]
    whole = runtime.compile_expr(e, [E.ColType(p, s)] * 2, threads_per_value=1).launch(
        [runtime.DeviceColumn(t, p, s) for t in raw], rows).view(rows, -1)
    g = torch.Generator(device="cuda").manual_seed(p)
    flags = [(torch.rand(rows, 1, device="cuda", generator=g) < 0.8).to(torch.uint8) for _ in range(2)]
    B = codec.compact_bytes(p)
    cols = [runtime.DeviceColumn(torch.cat([f, t.view(rows, B)], 1).reshape(-1).contiguous(), p, s, True)
            for f, t in zip(flags, raw)]
    m = runtime.compile_expr(e, [E.ColType(p, s, True)] * 2)
    got = m.launch(cols, rows).view(rows, -1)
    ok = (flags[0] & flags[1]).bool().reshape(-1)
    assert torch.equal(got[:, 0].bool(), ok)
    assert torch.equal(got[ok, 1:], whole[ok]) and not bool(got[~ok].any())
