"""The staged text kernels at their edges: limb instances, slot widths and
alignments, fields that leave the fast path, against the Python restatement."""
import random

import pytest

torch = pytest.importorskip("torch")

from oracle import pyref
from ultraprecise_b200 import abi, codec, runtime

pytestmark = pytest.mark.gpu

EDGE = [b"", b"-", b"0", b"-0.00", b"12.", b".5", b"1.2.3", b"+5", b"abc", b"1e5", b" 1", b"9" * 40,
        b"-" + b"9" * 1500, b"1" * 1501, b"00000123.4500000"]


def _fields(p, s, n, rng):
    out = list(EDGE)
    while len(out) < n:
        ip = str(rng.randint(0, 10 ** rng.randint(0, max(0, p - s)) - 1)) if rng.random() < 0.9 else ""
        fd = rng.randint(0, s + 3)
        fp = "".join(rng.choice("0123456789") for _ in range(fd))
        txt = ("-" if rng.random() < 0.5 else "") + ip + ("." + fp if fd or rng.random() < 0.2 else "")
        out.append(txt.encode())
    rng.shuffle(out)
    return out

def _format_case(p, s, rows, width, shift, rng):
    """Slots of `width` characters at `shift` bytes into a buffer of '#'."""
    B = codec.compact_bytes(p)
    top = 2 ** (8 * B - 1) - 1
    vals = [(rng.getrandbits(1), rng.choice([0, 1, 9, 10, 10 ** s if s < p else 1, 10 ** (p - 1), 10 ** p - 1, top])
             if rng.random() < 0.3 else rng.randrange(10 ** rng.randint(1, p))) for _ in range(rows)]
    raw = codec.encode(vals, p)
    buf = torch.full((rows * width + 64,), ord("#"), dtype=torch.uint8, device="cuda")
    lens = torch.zeros(rows, dtype=torch.int32, device="cuda")
    col = torch.frombuffer(bytearray(raw), dtype=torch.uint8).cuda()
    abi.check(abi.load().up_format_decimal(col.data_ptr(), rows, p, s, 0, buf.data_ptr() + shift, width,
                                           lens.data_ptr(), torch.cuda.current_stream().cuda_stream), "format")
    return raw, B, bytes(buf.cpu().numpy().tobytes()), lens.cpu().tolist()


# limbs at the edges of the staged instances, the widest one and one past it;
# slots that are too small, odd and unaligned; partial tiles
@pytest.mark.parametrize("p,s", [(1, 0), (9, 9), (10, 3), (18, 4), (19, 19), (28, 0), (38, 9), (57, 20), (77, 38), (115, 1),
                                 (154, 154), (230, 75), (300, 150), (320, 80)])
@pytest.mark.parametrize("rows,cut,shift", [(1, 0, 0), (127, 0, 1), (128, -1, 2), (389, 3, 0)])
def test_format_slots(p, s, rows, cut, shift):
    rng = random.Random(p * 31 + rows)
    width = max(1, abi.load().up_format_width(p, 0) - (cut if cut >= 0 else 0))
    raw, B, buf, lens = _format_case(p, s, rows, width, shift, rng)
    assert buf[:shift] == b"#" * shift and buf[shift + rows * width:] == b"#" * (64 - shift)
    for r in range(rows):
        want = pyref.format_decimal(raw[r * B:(r + 1) * B], s, False).encode()
        slot = buf[shift + r * width:shift + (r + 1) * width]
        assert lens[r] == (len(want) if len(want) <= width else -1)
        assert slot == want[:width].ljust(width, b"#")  # nothing past the string is touched


@pytest.mark.parametrize("p,s", [(1, 0), (9, 4), (10, 10), (18, 4), (19, 0), (28, 7), (38, 9), (77, 38), (154, 60), (300, 150),
                                 (320, 80)])
def test_parse_fields_at_the_staged_edges(p, s):
    """Text longer than a CTA's staging, fields longer than the limbs hold,
    leading zeros, cut and padded fractions, an unaligned text buffer."""
    rng = random.Random(p)
    fields = _fields(p, s, 1000, rng)
    for n in (p - 1, p, p + 1, p + 4, 2 * p + 20, 1100):
        if n > 0:
            fields += [b"0" * n, b"9" * n, b"-" + b"1" * n, b"0" * n + b"7.25", b"3." + b"4" * n, b"8" * n + b".x"]
    fields += [b"123", b"1.", b".", b"-.", b"--1", b"1-", b"12:4", b"/", b"1234/678", b"00:0"] * 3
    rng.shuffle(fields)
    joined = b"~" + b"".join(fields)
    offsets = [1]
    for f in fields:
        offsets.append(offsets[-1] + len(f))
    text = torch.frombuffer(bytearray(joined), dtype=torch.uint8).cuda()
    got, err = runtime.parse_decimal(None, p, s, text=text, offsets=torch.tensor(offsets, device="cuda"))
    B = codec.compact_bytes(p)
    want = [pyref.parse_decimal(f, B, s) for f in fields]
    got = bytes(got.cpu().numpy().tobytes())
    for r, f in enumerate(fields):
        assert got[r * B:(r + 1) * B] == want[r][0], f
    exp_err = 0
    for _, e in want:
        exp_err |= e
    assert err == exp_err


def test_parse_offsets_that_do_not_ascend():
    """A field that ends before it starts reads nothing and stores 0; its
    neighbours, and fields that overlap, are what they are alone."""
    rng = random.Random(9)
    text = "".join(rng.choice("0123456789") for _ in range(6000)).encode()
    offsets = [rng.randrange(40)]
    for r in range(700):
        offsets.append(min(5900, offsets[-1] + rng.randrange(0, 12)) if rng.random() < 0.8 else rng.randrange(0, 5900))
    offsets[128], offsets[256] = 3000, 3900  # two CTAs' ranges that ascend and fit, whatever is inside
    p, s = 38, 0
    B = codec.compact_bytes(p)
    dev = torch.frombuffer(bytearray(text), dtype=torch.uint8).cuda()
    got, err = runtime.parse_decimal(None, p, s, text=dev, offsets=torch.tensor(offsets, device="cuda"))
    got = bytes(got.cpu().numpy().tobytes())
    exp_err = 0
    for r, (a, b) in enumerate(zip(offsets, offsets[1:])):
        want, e = pyref.parse_decimal(text[a:max(a, b)], B, s)
        assert got[r * B:(r + 1) * B] == want, (r, a, b)
        exp_err |= e
    assert err == exp_err
