"""The limb schedules of the device product and of the reduction of a 512-bit
value (Fp::mul_inl, Fp::mul_wide, Fp::sqr_wide, Fp::redc, Fp::make_positive
in zkp-dynaverse_b200/csrc/field.cuh), restated with PTX carry semantics and
checked against plain integers for both BN254 fields.  Every chain asserts
that the carry it drops is zero, which is what the bounds of the schedule say.
Both moduli, the smallest and largest residues and random ones."""
import random

import pytest

M32 = (1 << 32) - 1
Q = 21888242871839275222246405745257275088696311157297823662689037894645226208583
R = 21888242871839275222246405745257275088548364400416034343698204186575808495617


def _limbs(x, n=8):
    return [(x >> (32 * i)) & M32 for i in range(n)]


def _value(words):
    return sum(w << (32 * i) for i, w in enumerate(words))


def _mac(d, xs, b, carry=0):
    """Pairs of d += xs[k] b with a carry in; (words, carry out)."""
    out = list(d)
    for k, x in enumerate(xs):
        s = (out[2 * k] | out[2 * k + 1] << 32) + x * b + carry
        out[2 * k], out[2 * k + 1], carry = s & M32, (s >> 32) & M32, s >> 64
    return out, carry


def _mac_top(d, top, xs, b):
    d, c = _mac(d, xs, b)
    assert top + c <= M32
    return d, top + c


def _mac_closed(d, xs, b, carry=0):
    d, c = _mac(d, xs, b, carry)
    assert c == 0
    return d


def _shift_mac(o, e, xs, b):
    s = o[0] + e[1]
    o = [s & M32] + o[1:]
    return _mac_closed(e[2:] + [0, 0], xs, b, s >> 32), o


class Field:
    def __init__(self, p):
        self.p, self.P = p, _limbs(p)
        self.inv = -pow(p, -1, 1 << 32) % (1 << 32)
        assert (p * self.inv + 1) % (1 << 32) == 0
        self.N = _limbs((p * self.inv + 1) >> 32)

    def reduce_step(self, e, o):
        m = e[0] * self.inv & M32
        o = _mac_closed(o, self.P[1::2], m)
        e, o[7] = _mac_top(e, o[7], self.P[0::2], m)
        assert e[0] == 0
        return e, o

    def shift_reduce(self, e, o):
        t0 = e[0]
        t, o = _shift_mac(o, e, self.N[1::2], t0)
        o, t[7] = _mac_top(o, t[7], self.N[0::2], t0)
        return o, t

    def finish(self, e, o, high=0):
        r = _value(e[1:]) + _value(o) + high
        assert r < 2 * self.p
        return r - self.p if r >= self.p else r

    def mul(self, a, b):
        e, o = _mac_closed([0] * 8, a[0::2], b[0]), _mac_closed([0] * 8, a[1::2], b[0])
        for i in range(6):
            e, o = self.shift_reduce(e, o)
            o = _mac_closed(o, a[1::2], b[i + 1])
            e, o[7] = _mac_top(e, o[7], a[0::2], b[i + 1])
        e, o = self.reduce_step(e, o)
        t, o = _shift_mac(o, e, a[1::2], b[7])
        o, t[7] = _mac_top(o, t[7], a[0::2], b[7])
        return self.finish(*self.reduce_step(o, t))

    def redc(self, w):
        t0 = w[0]
        e = _mac_closed([w[1]] + [0] * 7, self.N[0::2], t0)
        o = _mac_closed(w[2:8] + [0, 0], self.N[1::2], t0)
        for _ in range(5):
            e, o = self.shift_reduce(e, o)
        e, o = self.reduce_step(e, o)
        m = (o[0] + e[1]) * self.inv & M32
        t, o = _shift_mac(o, e, self.P[1::2], m)
        o, t[7] = _mac_top(o, t[7], self.P[0::2], m)
        assert o[0] == 0
        return self.finish(o, t, _value(w[8:]))


def _chain(d, at, xs, m):
    """A chain at word `at` of d; its carry goes to the word above."""
    out, c = _mac(d[at:at + 2 * len(xs)], xs, m)
    d[at:at + 2 * len(xs)] = out
    top = min(at + 2 * len(xs), 16)
    assert d[top] + c <= M32
    d[top] += c


def _combine(e, o):
    assert e[16] == 0 and o[15] == o[16] == 0
    return _limbs(_value(e[:16]) + (_value(o[:15]) << 32), 16)


def mul_wide(a, b):
    e, o = [0] * 17, [0] * 17
    for i in range(8):
        if i & 1:
            _chain(o, i - 1, a[0::2], b[i])
            _chain(e, i + 1, a[1::2], b[i])
        else:
            _chain(e, i, a[0::2], b[i])
            _chain(o, i, a[1::2], b[i])
    return _combine(e, o)


def sqr_wide(a):
    e, o = [0] * 17, [0] * 17
    d = [0] + [(a[j] << 1 | a[j - 1] >> 31) & M32 for j in range(1, 8)]
    for i in range(8):
        _chain(e, 2 * i, [a[i]] + d[i + 2::2], a[i])
        y = ([a[i + 1] << 1 & M32] if i < 7 else []) + d[i + 3::2]
        _chain(o, 2 * i, y, a[i])
    return _combine(e, o)


def make_positive(t, p):
    if _value(t) >> 511:
        return _limbs(_value(t) + (p << 255) & (1 << 512) - 1, 16)
    return t


@pytest.mark.parametrize("p", [Q, R])
def test_product_schedules(p):
    f, rng, r_inv = Field(p), random.Random(7), pow(1 << 256, -1, p)
    edge = [0, 1, 2, p - 1, p - 2, M32, p - (p & M32), (1 << 253) - 1]
    cases = [(x, y) for x in edge for y in edge] + [(rng.randrange(p), rng.randrange(p)) for _ in range(1500)]
    for x, y in cases:
        a, b = _limbs(x), _limbs(y)
        assert f.mul(a, b) == x * y * r_inv % p
        assert _value(mul_wide(a, b)) == x * y and _value(sqr_wide(a)) == x * x
        assert f.redc(sqr_wide(a)) == x * x * r_inv % p


@pytest.mark.parametrize("p", [Q, R])
def test_reduction_of_differences(p):
    f, rng, r_inv = Field(p), random.Random(8), pow(1 << 256, -1, p)
    edge = [0, 1, -1, p * p, -p * p, 2 * (p - 1) ** 2, -2 * (p - 1) ** 2, p << 254, 1 << 256, -(1 << 256)]
    for t in edge + [rng.randrange(-2 * (p - 1) ** 2, 2 * (p - 1) ** 2) for _ in range(1500)]:
        w = make_positive(_limbs(t % (1 << 512), 16), p)
        assert f.redc(w) == t * r_inv % p


@pytest.mark.parametrize("p", [Q, R])
def test_product_of_unreduced_operand(p):
    """Fp::mul_lazy: a < p times b < 4p stays below 2p before the last
    subtraction (asserted in finish) without losing a carry."""
    f, rng, r_inv = Field(p), random.Random(9), pow(1 << 256, -1, p)
    edge_b = [0, 1, p, 2 * p - 1, 2 * p, 3 * p, 4 * p - 1, 4 * p - 2]
    cases = [(x, y) for x in (0, 1, p - 1, p - 2) for y in edge_b]
    cases += [(rng.randrange(p), rng.randrange(4 * p)) for _ in range(1500)] + [(p - 1, rng.randrange(3 * p, 4 * p)) for _ in range(300)]
    for x, y in cases:
        assert f.mul(_limbs(x), _limbs(y)) == x * y * r_inv % p


@pytest.mark.parametrize("p", [Q, R])
def test_product_with_unreduced_rows(p):
    """Fp::mul_lazy the other way round, a < 2p times b < p, as Fq2::sqr and the
    scaling after a transform have it: below 2p, no carry lost."""
    f, rng, r_inv = Field(p), random.Random(10), pow(1 << 256, -1, p)
    edge_a = [0, 1, p - 1, p, p + 1, 2 * p - 2, 2 * p - 1]
    cases = [(x, y) for x in edge_a for y in (0, 1, p - 1, p - 2, p - (p & M32), (1 << 253) - 1)]
    cases += [(rng.randrange(2 * p), rng.randrange(p)) for _ in range(1500)]
    cases += [(rng.randrange(2 * p - 99, 2 * p), rng.randrange(p - (1 << 200), p)) for _ in range(300)]
    for x, y in cases:
        assert f.mul(_limbs(x), _limbs(y)) == x * y * r_inv % p


class RawField(Field):
    def finish(self, e, o, high=0):
        r = _value(e[1:]) + _value(o) + high
        assert r < 1 << 256
        return r


@pytest.mark.parametrize("p", [Q, R])
def test_reduction_of_large_sums(p):
    """Fp::redc_raw: a high half of up to 4.27 p keeps the sum below 2^256, and
    below the high half plus p and p / 2^32."""
    f, rng, r_inv = RawField(p), random.Random(11), pow(1 << 256, -1, p)
    top = 427 * p // 100
    lows = [0, 1, M32, (1 << 256) - 1, (1 << 256) - (1 << 32), p << 2]
    cases = [(h, low) for h in (0, 1, p, 2 * p, 4 * p, top - 1, top) for low in lows]
    cases += [(rng.randrange(top + 1), rng.randrange(1 << 256)) for _ in range(1500)]
    for h, low in cases:
        t = h << 256 | low
        got = f.redc(_limbs(t, 16))
        assert got % p == t * r_inv % p and got <= h + p + (p >> 32)


def test_quotient_estimate_from_the_top_bits():
    """reduce_top of the pairing: for v < 10 q with top = v >> 252, 21 top / 64
    is the quotient by q or one less, at both ends of every top's values."""
    for top in range((10 * Q - 1 >> 252) + 1):
        for v in (top << 252, min((top + 1 << 252) - 1, 10 * Q - 1)):
            assert v // Q - 1 <= top * 21 >> 6 <= v // Q
