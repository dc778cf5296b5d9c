"""Device field arithmetic where a carry or borrow runs through many words:
sums and differences that wrap at 2^256 next to a run of ones or zeros, and
products and squares of values near powers of two and multiples of the modulus,
against Python integers.  Every comparison is exact."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = 2**255 - 19
Q = 2**255 - 85737960593035654572250192257530476641
FIELDS = {0: P, 1: Q}


def edge_values(m: int) -> list:
    c = 2**256 % m
    vals = {0, 1, 2, c, c - 1, c + 1, m - 1, m, m + 1, 2 * m - 1, 2 * m, 2**256 - 1, 2**256 - c, 2**256 - c - 1}
    for k in range(0, 257, 32):
        for d in (-2, -1, 0, 1, c):
            vals.add((2**k + d) % 2**256)
            vals.add((2**256 - 2**k + d) % 2**256)
    vals.add(int("aaaaaaaa" * 8, 16))
    vals.add(sum(2**(64 * i) * 0xffffffff for i in range(4)))
    return sorted(vals)


def pack(vals) -> np.ndarray:
    return np.frombuffer(b"".join(v.to_bytes(32, "little") for v in vals), dtype=np.uint8)


def unpack(a: np.ndarray) -> list:
    return [int.from_bytes(r.tobytes(), "little") for r in a.reshape(-1, 32)]


@pytest.mark.parametrize("field", [0, 1])
def test_binary_ops_over_all_edge_pairs(ctx, field):
    m = FIELDS[field]
    v = edge_values(m)
    a = [x for x in v for _ in v]
    b = [y for _ in v for y in v]
    for op, fn in ((0, lambda x, y: x * y), (2, lambda x, y: x + y), (3, lambda x, y: x - y)):
        got = unpack(ctx.field_op(field, op, pack(a), pack(b)))
        bad = [(hex(x), hex(y)) for x, y, g in zip(a, b, got) if g != fn(x, y) % m]
        assert not bad, (op, len(bad), bad[:3])


@pytest.mark.parametrize("field", [0, 1])
def test_unary_ops_over_edges(ctx, field):
    m = FIELDS[field]
    rng = np.random.default_rng(7 + field)
    v = edge_values(m) + [int.from_bytes(rng.bytes(32), "little") for _ in range(2000)]
    for op, fn in ((1, lambda x: x * x), (5, lambda x: pow(x, -1, m) if x % m else 0), (6, lambda x: -x)):
        got = unpack(ctx.field_op(field, op, pack(v)))
        assert got == [fn(x) % m for x in v], op
