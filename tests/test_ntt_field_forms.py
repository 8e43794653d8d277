"""Field operations written as PTX carry sequences, replayed instruction by
instruction with PTX's CC.CF semantics (add.cc / addc carry, sub.cc / subc
borrow, mad.lo.cc / madc.hi.cc, shf.l.wrap) and checked exactly against the
field (or the integer product) on random and edge-case operands:

  ntt_field.cuh  nt_sub, nt_add (a subtraction of the negation), nt_canon,
                 nt_mul and the products by powers of two
  gl64.cuh       mul_add_words, sqr_words, mont_reduce, pr_fold, mul_wide and
                 pr_reduce128

The GPU parity tests pin the compiled kernels' outputs; this pins the algebra
of each sequence."""

import random

import pytest

P = 0xFFFFFFFF00000001
M32 = 0xFFFFFFFF


class Flags:
    """The condition-code carry flag of a PTX instruction sequence (32-bit words)."""

    def __init__(self):
        self.cf = 0

    def add_cc(self, a, b):
        r = a + b
        self.cf = r >> 32
        return r & M32

    def addc_cc(self, a, b):
        r = a + b + self.cf
        self.cf = r >> 32
        return r & M32

    def addc(self, a, b):
        return (a + b + self.cf) & M32

    def sub_cc(self, a, b):
        r = a - b
        self.cf = int(r < 0)
        return r & M32

    def subc_cc(self, a, b):
        r = a - (b + self.cf)
        self.cf = int(r < 0)
        return r & M32

    def subc(self, a, b):
        return (a - (b + self.cf)) & M32

    def mad_lo_cc(self, a, b, c):
        r = ((a * b) & M32) + c
        self.cf = r >> 32
        return r & M32

    def madc_hi_cc(self, a, b, c):
        r = ((a * b) >> 32) + c + self.cf
        self.cf = r >> 32
        return r & M32


def halves(x):
    return x & M32, x >> 32


def mad_wide(a, b, c):
    return (a * b + c) % 2**64


def nt_sub(a, b):
    f = Flags()
    a0, a1 = halves(a)
    b0, b1 = halves(b)
    lo = f.sub_cc(a0, b0)
    hi = f.subc_cc(a1, b1)
    bw = f.subc(0, 0)
    lo = f.sub_cc(lo, bw)
    hi = f.subc(hi, 0)
    return (hi << 32) | lo


def nt_add(a, b):
    """nt_add: a - (p - b) through nt_sub (p - b is p itself when b = 0)."""
    return nt_sub(a, P - b)


def nt_canon(x):
    f = Flags()
    x0, x1 = halves(x)
    f.add_cc(x0, M32)
    f.addc_cc(x1, 0)
    k = f.addc(0, 0)
    return mad_wide(k, M32, x)


def mul_add_words(a, b, c=0):
    """a b + c as 128 bits: the middle products summed first, the halves of c starting the first two."""
    f = Flags()
    (a0, a1), (b0, b1), (c0, c1) = halves(a), halves(b), halves(c)
    low, mid, high = a0 * b0 + c0, a0 * b1 + c1, a1 * b1
    assert max(low, mid, high) < 2**64  # mad.wide does not wrap
    w0, l1 = halves(low)
    m0, m1 = halves(mid)
    h0, h1 = halves(high)
    m0 = f.mad_lo_cc(a1, b0, m0)
    m1 = f.madc_hi_cc(a1, b0, m1)
    k = f.addc(h1, 0)
    w1 = f.add_cc(l1, m0)
    w2 = f.addc_cc(h0, m1)
    w3 = f.addc(k, 0)
    return w0, w1, w2, w3


def sqr_words(a):
    """a^2 from a0^2, a1^2 and the cross term a0 a1, doubled by shifts (shf.l.wrap) and added once."""
    f = Flags()
    a0, a1 = halves(a)
    w0, l1 = halves(a0 * a0)
    m0, m1 = halves(a0 * a1)
    h0, h1 = halves(a1 * a1)
    c = m1 >> 31
    m1 = ((m1 << 1) | (m0 >> 31)) & M32  # shf.l.wrap.b32 m1, m0, m1, 1
    m0 = (m0 << 1) & M32
    w1 = f.add_cc(l1, m0)
    w2 = f.addc_cc(h0, m1)
    w3 = f.addc(h1, c)
    return w0, w1, w2, w3


def mont_reduce(w0, w1, w2, w3):
    f = Flags()
    s = f.add_cc(w1, w0)
    t = f.addc(s, 0)
    b0 = f.sub_cc(w0, t)
    b1 = f.subc(s, 0)
    r0 = f.sub_cc(w2, b0)
    r1 = f.subc_cc(w3, b1)
    k = f.subc(0, 0)
    r0 = f.sub_cc(r0, k)
    r1 = f.subc(r1, 0)
    return (r1 << 32) | r0


def nt_mul(a, bm):
    """a b for a table value bm = b 2^64 mod p."""
    return mont_reduce(*mul_add_words(a, bm))


def pr_fold(x0, x1, t):
    f = Flags()
    n0, n1 = (t + 1) & M32, ~t & M32
    r0 = f.sub_cc(x0, n0)
    r1 = f.subc_cc(x1, n1)
    k = f.subc(0, 0)
    r0 = f.sub_cc(r0, k)
    r1 = f.subc(r1, 0)
    return (r1 << 32) | r0


def mul2_24(x):
    return pr_fold((x << 24) & M32, (x >> 8) & M32, x >> 40)


def mul2_48_neg(x):
    return mont_reduce((x << 16) & M32, (x >> 16) & M32, x >> 48, 0)


def mul2_72(x):
    xl, xh = x & 0xFFFFFF, x >> 24
    return nt_sub(((xl << 40) - (xl << 8)) % 2**64, xh)


def mul_wide(a, b):
    f = Flags()
    (a0, a1), (b0, b1) = halves(a), halves(b)
    r0, r1 = halves(a0 * b0)
    r2, r3 = halves(a1 * b1)
    for x, y in ((a0, b1), (a1, b0)):
        r1 = f.mad_lo_cc(x, y, r1)
        r2 = f.madc_hi_cc(x, y, r2)
        r3 = f.addc(r3, 0)
    return r0, r1, r2, r3


def pr_reduce128(l0, l1, h0, h1):
    f = Flags()
    r0 = f.sub_cc(l0, h1)
    r1 = f.subc_cc(l1, 0)
    b = f.subc(0, 0)
    r0 = f.sub_cc(r0, b)
    r1 = f.subc(r1, 0)
    r1 = f.add_cc(r1, h0)
    k = f.addc(0, 0)
    r0 = f.sub_cc(r0, h0)
    r1 = f.subc_cc(r1, 0)
    k = -f.subc(k, 0) & M32  # neg.s32: all ones when the fold left 2^64
    assert k in (0, M32)
    r0 = f.add_cc(r0, k)
    r1 = f.addc(r1, 0)
    return (r1 << 32) | r0


def words(v):
    return tuple(v >> (32 * i) & M32 for i in range(4))


def mont(b):
    return b * 2**64 % P


EDGES = [0, 1, 2, P - 1, P - 2, 0xFFFFFFFF, 0x100000000, 0xFFFFFFFF00000000, P // 2, 2**63, 0xFFFFFFFE00000001]


def check(a, b):
    """Canonical a, b."""
    assert nt_sub(a, b) == (a - b) % P
    assert nt_add(a, b) == (a + b) % P
    assert nt_mul(a, mont(b)) == a * b % P
    assert mul2_24(a) == a * 2**24 % P
    assert mul2_48_neg(a) == -a * 2**48 % P
    assert mul2_72(a) == a * 2**72 % P


def check_any(a, b, c):
    """Any 64-bit a, b, c."""
    assert nt_canon(a) == a % P
    assert mul_add_words(a, b) == mul_wide(a, b) == words(a * b)
    assert mul_add_words(a, b, c) == words(a * b + c)
    assert sqr_words(a) == words(a * a)
    v = a << 64 | b
    assert pr_reduce128(*words(v)) % P == v % P
    assert mont_reduce(*words(v)) * 2**64 % P == v % P


WIDE = EDGES + [2**64 - 1, P, P + 1, 2**64 - 2**32, 0x80000000, 0xFFFFFFFF80000000]


def test_edge_operands():
    for a in EDGES:
        for b in EDGES:
            check(a % P, b % P)
    for a in WIDE:
        for b in WIDE:
            for c in (0, 1, M32, M32 << 32, 2**64 - 1):
                check_any(a, b, c)


@pytest.mark.parametrize("seed", [1, 2])
def test_random_operands(seed):
    rng = random.Random(seed)
    for _ in range(10000):
        check(rng.randrange(P), rng.randrange(P))
        a, b, c = (rng.choice([rng.getrandbits(64), P + rng.randrange(2**32 - 1), rng.choice(WIDE)]) for _ in range(3))
        check_any(a, b, c)


def test_extreme_128_bit_inputs():
    for v in [(2**64 - 1) ** 2, 2**128 - 1, 0, 2**96, 2**96 - 1, P * (2**64 - 1)]:
        assert pr_reduce128(*words(v)) % P == v % P
        assert mont_reduce(*words(v)) * 2**64 % P == v % P
