"""The integer field arithmetic (product, square, a b - c d) at coordinate words where its carry
chains are longest or empty: point formulas over arbitrary coordinates, on the curve or not, give
the oracle's XYZZ coordinates word for word."""
import numpy as np
import pytest

from oracle import bn254
from zk_gpu._lib import check, lib, u32p

pytestmark = pytest.mark.gpu
Q = bn254.Q
MONT = (1 << 256) % Q
UNMONT = pow(MONT, -1, Q)

# Montgomery words: all-ones words, single words, the modulus' neighbours, the half, powers of two
WORDS = [1, 2, Q - 1, Q - 2, (Q - 1) // 2, (Q + 1) // 2, (1 << 253) - 1, (1 << 224) - 1, 1 << 253,
         Q - (1 << 32), Q - (1 << 224), sum(0xFFFFFFFF << (64 * i) for i in range(4)) % Q,
         sum(0xFFFFFFFF << (64 * i + 32) for i in range(3)), 0xFFFFFFFF, 0xFFFFFFFF << 32, (1 << 128) - 1, 0]


def elements(seed, count):
    rnd = np.random.default_rng(seed)
    def pick():
        if rnd.random() < 0.8:
            return WORDS[int(rnd.integers(0, len(WORDS)))]
        return int.from_bytes(rnd.bytes(32), "little") % Q

    return [pick() for _ in range(count)]


@pytest.mark.parametrize("group", ["G1", "G2"])
def test_point_formulas_word_for_word(gpu, group):
    F = bn254.FIELD[group]
    per = 1 if group == "G1" else 2  # words of Fq per coordinate
    count = 400
    vals = elements(17 + per, 4 * per * count)
    words = np.array([w for v in vals for w in bn254.words32(v)], dtype=np.uint32)
    xw = 32 * per
    out = np.zeros(count * 3 * xw, dtype=np.uint32)
    check(lib().zkg_test_point_ops(gpu.handle, per, words.ctypes.data_as(u32p), count, out.ctypes.data_as(u32p)))

    def coordinate(k):  # the field element behind Montgomery words k
        if per == 1:
            return vals[k] * UNMONT % Q
        return bn254.Fq2(vals[2 * k] * UNMONT % Q, vals[2 * k + 1] * UNMONT % Q)

    def plain(c):
        return [c * MONT % Q] if per == 1 else [c.a * MONT % Q, c.b * MONT % Q]

    for i in range(count):
        x = [coordinate(4 * i + k) for k in range(4)]
        zero = lambda c: c == 0 if per == 1 else c.a == 0 and c.b == 0
        p = None if zero(x[0]) and zero(x[1]) else (x[0], x[1])
        q = None if zero(x[2]) and zero(x[3]) else (x[2], x[3])
        s = bn254.xyzz_add_affine(F, bn254.xyzz_from_affine(F, p), q)
        d = bn254.xyzz_double(F, bn254.xyzz_from_affine(F, p))
        for k, want in enumerate((s, d, bn254.xyzz_add(F, s, d))):
            got = out[(3 * i + k) * xw: (3 * i + k + 1) * xw]
            ints = [bn254.from_words32(got[8 * j: 8 * j + 8]) for j in range(4 * per)]
            if zero(want[2]):  # infinity: ZZ = 0 (the other coordinates carry no meaning)
                assert all(v == 0 for v in ints[2 * per: 3 * per]), (group, i, k)
                continue
            assert ints == [v for c in want for v in plain(c)], (group, i, k)
