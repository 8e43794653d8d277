"""The hash kernels' and the NTT's arithmetic (gl64.cuh, hash.cuh, ntt_field.cuh) replayed on the CPU with
PTX's carry semantics: the Montgomery reduction, x^7 from four Montgomery
products, the folds that end the linear layers, Poseidon2's diagonal lane, and
the two-rounds-at-once form of Poseidon's partial rounds with the bounds that
its exact FP64 sums rely on.  The GPU parity tests pin the compiled kernels."""

import random
import re
from pathlib import Path

import pytest

P = 0xFFFFFFFF00000001
M32 = 0xFFFFFFFF
R = 2**64
RINV = pow(R, -1, P)
EDGES = [0, 1, 2, M32 - 1, M32, M32 + 1, 2**33, 2**63, P - 1, P, P + 1, 2**64 - 2**33, 2**64 - 2, 2**64 - 1]


def sub(a, b, borrow=0):
    r = a - b - borrow
    return r & M32, int(r < 0)


def add_p_on_borrow(r0, r1, k):
    """sub.cc r0, r0, -k; subc r1, r1, 0: on a borrow, minus 2^32 - 1 (never below zero)."""
    r = (r1 << 32 | r0) - (M32 if k else 0)
    assert r >= 0
    return r


def mont_reduce(v):
    w = [v >> (32 * i) & M32 for i in range(4)]
    s = w[1] + w[0]
    s, e = s & M32, s >> 32
    t = s + e
    assert t <= M32
    b0, bw = sub(w[0], t)
    b1, bw = sub(s, 0, bw)
    assert not bw
    r0, bw = sub(w[2], b0)
    r1, k = sub(w[3], b1, bw)
    return add_p_on_borrow(r0, r1, k)


def pr_fold(x0, x1, t):
    assert t < M32
    r0, bw = sub(x0, t + 1)
    r1, k = sub(x1, ~t & M32, bw)
    return add_p_on_borrow(r0, r1, k)


def pr_reduce_split_add(al, ah, c=0):
    x = al + c
    k = (ah >> 32) + (x >> 64)
    x1 = (x >> 32 & M32) + (ah & M32)
    return pr_fold(x & M32, x1 & M32, k + (x1 >> 32))


def pow7(x):
    x2 = mont_reduce(x * x)
    return mont_reduce(mont_reduce(x * x2) * mont_reduce(x2 * x2))


def sum_mont(z):
    z0, z1, z2 = z & M32, z >> 32 & M32, z >> 64
    b = z0 + z1
    b0, b1 = b & M32, z2 + (b >> 32)
    a0, bw = sub(0, b0)
    a1, k = sub(z0, b1, bw)
    return add_p_on_borrow(a0, a1, k)


def values(n, seed):
    rnd = random.Random(seed)
    return EDGES + [rnd.getrandbits(64) for _ in range(n)]


def test_montgomery_reduction():
    v = values(200, 1)
    for a in v:
        for b in v:
            r = mont_reduce(a * b)
            assert r < R and r % P == a * b * RINV % P
            if a < P and b < P:
                assert r < P  # canonical for canonical operands
            assert mont_reduce(a << 64 | b) % P == (a << 64 | b) * RINV % P


def test_pow7_needs_no_conversion():
    assert pow(R, 3, P) == 1
    for x in values(2000, 2):
        assert pow7(x) % P == pow(x, 7, P)


def test_folds_of_the_linear_layers():
    rnd = random.Random(3)
    hi = [0, 1, M32, M32 + 1, 2**40, 2**50 - 1, 2**63 - 1] + [rnd.getrandbits(50) for _ in range(100)]
    for al in values(100, 4):
        for ah in hi:
            assert pr_reduce_split_add(al, ah) % P == (al + (ah << 32)) % P
            for c in (0, 1, P - 1, 2**64 - 1):
                assert pr_reduce_split_add(al, ah, c) % P == (al + (ah << 32) + c) % P


def test_poseidon2_diagonal_lane():
    for z in values(300, 5) + [12 * (2**64 - 1), 2**64, 2**67]:
        s = sum_mont(z)
        assert s % P == z * R % P
        for x, d in ((2**64 - 1, P - 1), (0, 5), (P, 1), (z & (2**64 - 1), 0xC3B6C08E23BA9300)):
            v = x * (d * R % P) + s
            assert v < 2**128
            assert mont_reduce(v) % P == (x * d + z) % P


def test_ntt_power_of_two_products():
    """ntt_field.cuh: x 2^24 as a fold, -x 2^48 as a Montgomery reduction of x 2^16; canonical results."""
    for x in values(3000, 6):
        x %= P
        v = x << 24
        assert pr_fold(v & M32, v >> 32 & M32, v >> 64) == x * 2**24 % P
        assert mont_reduce(x << 16) == -x * 2**48 % P


def poseidon_constants():
    txt = (Path(__file__).resolve().parents[1] / "zeknox_b200/csrc/zk_constants.h").read_text()

    def table(name):
        body = re.search(r"#define " + name + r"_LIST((?:.*\\\n)*.*)", txt).group(1)
        return [int(x, 0) for x in re.findall(r"0x[0-9a-fA-F]+|\b\d+\b", re.sub(r"(?<=[0-9a-fA-F])[uUlL]+", "", body))]

    return table("ZK_POSEIDON_RC"), table("ZK_POSEIDON_MDS_CIRC"), table("ZK_POSEIDON_MDS_DIAG")


def kpair(k, offset, bias):
    d = (k - bias * (1 + 2**32)) % P
    return bias - offset + (d & M32), bias - offset + (d >> 32)


@pytest.mark.parametrize("seed", range(3))
def test_two_partial_rounds_at_once(seed):
    """The pair's integer sums, as the kernels form them, against two plain rounds; every sum below 2^53."""
    rc, circ, diag = poseidon_constants()
    assert len(rc) == 360 and len(circ) == 12
    at = lambda j: circ[j % 12]  # noqa: E731
    at2 = lambda j: sum(at(i) * at(j - i) for i in range(12))  # noqa: E731
    q1 = [sum(at(k) - at(k + 6) for k in range(6))]
    off1 = q1[0] * 2**31
    off2 = [(1 if r < 6 else -1) * 2**31 * sum(at2(k - r % 6) - at2(k + 6 - r % 6) for k in range(6)) for r in range(12)]
    mds = lambda x: [(sum(at(k - r) * x[k] for k in range(12)) + (diag[0] * x[0] if r == 0 else 0)) % P for r in range(12)]  # noqa: E731
    rnd = random.Random(seed)
    for q in range(11):
        x = [rnd.choice([rnd.getrandbits(64), 2**64 - 1, 0, M32, P - 1]) for _ in range(12)]
        c, c2 = rc[12 * (5 + 2 * q):][:12], rc[12 * (6 + 2 * q):][:12]
        want = [pow(x[0], 7, P)] + x[1:]
        want = [(a + b) % P for a, b in zip(mds(want), c)]
        want[0] = pow(want[0], 7, P)
        want = [(a + b) % P for a, b in zip(mds(want), c2)]

        s = [pow7(x[0])] + x[1:]
        half = lambda v, h: v >> 32 if h else v & M32  # noqa: E731
        u = [[half(s[i], h) + half(s[i + 6], h) for i in range(6)] for h in (0, 1)]
        w = [[half(s[i], h) - half(s[i + 6], h) + 2**32 for i in range(6)] for h in (0, 1)]
        mid = kpair(c[0], off1, 2**40)
        y0 = []
        for h in (0, 1):
            pa = sum((at(k) + at(k + 6)) * u[h][k] for k in range(6))
            qa = sum((at(k) - at(k + 6)) * w[h][k] for k in range(6))
            assert (pa + qa) % 2 == 0
            y0.append((pa + qa) // 2 + diag[0] * half(s[0], h) + mid[h])
            assert 0 <= y0[h] < 2**42
        y = pow7(pr_reduce_split_add(*y0))
        out = []
        for r in range(12):
            k = (c2[r] + sum(at(j - r) * c[j] for j in range(12))) % P
            acc = []
            for h in (0, 1):
                kk = kpair(k, off2[r], 2**48)[h]
                rr, sg = r % 6, 1 if r < 6 else -1
                pa = sum((at2(i - rr) + at2(i + 6 - rr)) * u[h][i] for i in range(6))
                qa = sum((at2(i - rr) - at2(i + 6 - rr)) * w[h][i] for i in range(6))
                g = diag[0] * half(s[0], h) + half(y, h) - y0[h]
                v = (pa + sg * qa) // 2 + kk + at(-r) * g + (diag[0] * half(y, h) if r == 0 else 0)
                assert max(pa, abs(qa), abs(g) * 41) < 2**53 and 0 <= v < 2**50
                acc.append(v)
            out.append(pr_reduce_split_add(*acc) % P)
        assert out == want


@pytest.mark.parametrize("seed", range(3))
def test_three_partial_rounds_at_once(seed):
    """The triple's integer sums, as the one-thread kernel forms them, against three plain rounds; every sum below 2^53."""
    rc, circ, diag = poseidon_constants()
    conv = lambda a: [sum(a[i] * circ[(j - i) % 12] for i in range(12)) for j in range(12)]  # noqa: E731
    row = {1: circ, 2: conv(circ), 3: conv(conv(circ))}
    at = lambda n, j: row[n][j % 12]  # noqa: E731
    kappa, d = 2755704, diag[0]
    pm = lambda n, r, k: at(n, k - r) + at(n, k + 6 - r) - (kappa if n == 3 else 0)  # noqa: E731
    qm = lambda n, r, k: at(n, k - r) - at(n, k + 6 - r)  # noqa: E731
    offset = lambda n, r: (1 if r < 6 else -1) * 2**31 * sum(qm(n, r % 6, k) for k in range(6))  # noqa: E731
    mds = lambda x: [(sum(circ[(k - r) % 12] * x[k] for k in range(12)) + (d * x[0] if r == 0 else 0)) % P for r in range(12)]  # noqa: E731
    half = lambda v, h: v >> 32 if h else v & M32  # noqa: E731
    rnd = random.Random(seed)

    def exact(*v):
        assert all(abs(x) < 2**53 for x in v)
        return v[0]

    def rows(n, u, w, t=0):
        """4 C^n x + t by the 3x3 split; every partial sum bounded."""
        up, um = [u[i] + u[i + 3] for i in range(3)], [u[i] - u[i + 3] for i in range(3)]
        out = [0] * 12
        for r in range(3):
            ps = [(pm(n, r, k) + pm(n, r, k + 3)) * up[k] for k in range(3)]
            pd = [(pm(n, r, k) - pm(n, r, k + 3)) * um[k] for k in range(3)]
            exact(*[abs(t) + sum(map(abs, ps))], *[sum(map(abs, pd))])
            sp, sm = t + sum(ps), sum(pd)
            for rr, pa in ((r, sp + sm), (r + 3, sp - sm)):
                q = [2 * qm(n, rr, k) * w[k] for k in range(6)]
                qa = sum(q)
                exact(pa, sum(map(abs, q)), pa + qa, pa - qa)
                assert (pa + qa) % 4 == (pa - qa) % 4 == 0
                out[rr], out[rr + 6] = (pa + qa) // 4, (pa - qa) // 4
        return out

    for q in range(7):
        fill = rnd.choice([0, 2**64 - 1, None])  # all lanes at an end of their range, or mixed
        x = [rnd.choice([rnd.getrandbits(64), 2**64 - 1, 0, M32, M32 << 32, P - 1]) if fill is None else fill for _ in range(12)]
        if q % 2:
            x = [2**64 - 1 if i in (0, 3, 6, 9) else 0 for i in range(12)]  # the signs of C^3 - kappa / 2
        want = list(x)
        for j in range(3):
            want[0] = pow(want[0], 7, P)
            want = [(a + b) % P for a, b in zip(mds(want), rc[12 * (5 + 3 * q + j):])]
        c = rc[12 * (5 + 3 * q):][:12]
        ctimes = lambda v: [sum(circ[(k - r) % 12] * v[k] for k in range(12)) % P for r in range(12)]  # noqa: E731
        c2 = [(a + b) % P for a, b in zip(ctimes(c), rc[12 * (6 + 3 * q):])]
        c3 = [(a + b) % P for a, b in zip(ctimes(c2), rc[12 * (7 + 3 * q):])]

        s = [pow7(x[0])] + x[1:]
        u = [[half(s[i], h) + half(s[i + 6], h) for i in range(6)] for h in (0, 1)]
        w = [[half(s[i], h) - half(s[i + 6], h) + 2**32 for i in range(6)] for h in (0, 1)]
        ky, kz = kpair(c[0], offset(1, 0), 2**40), kpair(c2[0], offset(2, 0), 2**45)
        y = [exact(rows(1, u[h], w[h])[0] + d * half(s[0], h) + ky[h]) for h in (0, 1)]
        assert min(y) >= 0
        yr = pr_reduce_split_add(*y)
        yp = pow7(yr)
        total = pr_reduce_split_add(sum(u[0]), sum(u[1]))
        t = pr_reduce_split_add(*[exact(kappa // 2 * half(total, h)) for h in (0, 1)])
        g0 = [d * half(s[0], h) + half(yp, h) - half(yr, h) for h in (0, 1)]
        z = [exact(rows(2, u[h], w[h])[0] + kz[h] + d * half(yp, h) + circ[0] * g0[h]) for h in (0, 1)]
        assert min(z) >= 0
        zr = pr_reduce_split_add(*z)
        zq = pow7(zr)
        out = [[], []]
        for h in (0, 1):
            g1 = d * half(yp, h) + half(zq, h) - half(zr, h)
            for r, v in enumerate(rows(3, u[h], w[h], 4 * half(t, h))):
                v = exact(v + kpair(c3[r], offset(3, r), 2**49)[h])
                v = exact(v + at(2, -r) * g0[h], at(2, -r) * g0[h])
                v = exact(v + at(1, -r) * g1 + (d * half(zq, h) if r == 0 else 0))
                assert v >= 0
                out[h].append(v)
        assert [pr_reduce_split_add(a, b) % P for a, b in zip(*out)] == want


BN_R = 0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001
MASK = 2**29 - 1


def limbs(x):
    return [x >> (29 * i) & MASK for i in range(9)]


def bn_value(v):
    return sum(a << (29 * i) for i, a in enumerate(v))


def bn_mul_sum(terms, addend=(0,) * 9):
    """(sum of x y) / 2^261 + addend mod r as the kernel's 64-bit columns form it."""
    ninv = -pow(BN_R, -1, 2**29) % 2**29
    c = [0] * 9 + list(addend)
    for x, y in terms:
        for i in range(9):
            for j in range(9):
                c[i + j] += x[i] * y[j]
    for i in range(9):
        m = c[i] * ninv & MASK
        for j, r in enumerate(limbs(BN_R)):
            c[i + j] += m * r
        assert max(c) < 2**64
        c[i + 1] += c[i] >> 29
    out = []
    for i in range(9):
        out.append(c[9 + i] & MASK)
        if i < 8:
            c[10 + i] += c[9 + i] >> 29
        else:
            assert c[17] <= MASK  # the value is below 2^261
    assert max(c) < 2**64
    return out


def test_bn254_columns_hold_a_matrix_row():
    """Five products of full limbs and a reduction fit the columns; results are the field's."""
    rnd = random.Random(7)
    top = limbs(BN_R - 1)
    full = [MASK] * 8 + [(67 * BN_R) >> 232]  # the largest state value of the partial rounds, every other limb full
    for x, y in [(full, [MASK] * 8 + [top[8]]), (limbs(rnd.randrange(67 * BN_R)), limbs(rnd.randrange(BN_R)))]:
        got = bn_value(bn_mul_sum([(x, y)] * 5, x))
        want = 5 * bn_value(x) * bn_value(y) * pow(2**261, -1, BN_R) + bn_value(x)
        assert got % BN_R == want % BN_R and got < 2**261


def test_bn254_partial_round_growth():
    """Sixty rounds of the lanes' update from the largest first-half outputs stay below 2^260."""
    rnd = random.Random(8)
    st = limbs(2 * BN_R - 1)
    for _ in range(60):
        st = bn_mul_sum([(limbs(2 * BN_R - 1), limbs(BN_R - 1 - rnd.getrandbits(20)))], st)
    assert bn_value(st) < 2**260
    # a full round's S-box of that value: squares below 2^259, the fifth power below 2^256
    x2 = bn_mul_sum([(st, st)])
    x4 = bn_mul_sum([(x2, x2)])
    x5 = bn_mul_sum([(x4, st)], limbs(BN_R - 1))
    assert bn_value(x2) < 2**259 and bn_value(x5) < 2**256
    assert bn_mul_sum([], limbs(0)) == [0] * 9
    # out of Montgomery form the value is at most r
    assert bn_value(bn_mul_sum([(limbs(2**261 - 1), limbs(1))])) <= BN_R
