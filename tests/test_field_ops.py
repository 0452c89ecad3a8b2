"""The field operations of the G2 kernels (products with one reduction per component), the inversion by division
steps and the products by constants with a precomputed quotient, word for word at operands where their
carry chains, signs and exits are at an extreme, and at random ones."""
import numpy as np
import pytest

from oracle import bn254
from test_field_words import WORDS
from zk_gpu import ZkGpuError
from zk_gpu._lib import check, lib, u32p

pytestmark = pytest.mark.gpu
Q, R = bn254.Q, bn254.R
TWO256 = 1 << 256
UNMONT = pow(TWO256, -1, Q)


def run(gpu, op, items, words_out):
    """items: lists of integers (8 words each); the results likewise."""
    flat = np.array([w for item in items for v in item for w in bn254.words32(v)], dtype=np.uint32)
    out = np.zeros(len(items) * words_out, dtype=np.uint32)
    check(lib().zkg_test_field_ops(gpu.handle, op, flat.ctypes.data_as(u32p), len(items), out.ctypes.data_as(u32p)))
    values = [bn254.from_words32(out[i: i + 8]) for i in range(0, out.size, 8)]
    per = words_out // 8
    return [values[i: i + per] for i in range(0, len(values), per)]


def random_element(rnd, modulus):
    return int.from_bytes(rnd.bytes(32), "little") % modulus


def test_fq2_products(gpu):
    rnd = np.random.default_rng(11)

    def pick():
        return WORDS[int(rnd.integers(0, len(WORDS)))] if rnd.random() < 0.8 else random_element(rnd, Q)

    items = [[pick() for _ in range(8)] for _ in range(4000)]
    items += [[v] * 8 for v in WORDS] + [[Q - 1, Q - 1, Q - 1, Q - 1, a, b, c, d]
                                         for a in (0, Q - 1) for b in (0, Q - 1) for c in (0, Q - 1) for d in (0, Q - 1)]

    def mul(a, b):
        return (a[0] * b[0] - a[1] * b[1]) * UNMONT, (a[0] * b[1] + a[1] * b[0]) * UNMONT

    for item, got in zip(items, run(gpu, 0, items, 48)):
        x, y, z, w = (item[2 * k: 2 * k + 2] for k in range(4))
        xy, xx, zw = mul(x, y), mul(x, x), mul(z, w)
        want = [*xy, *xx, xy[0] - zw[0], xy[1] - zw[1]]
        assert got == [v % Q for v in want], item


EDGES = sorted({v % Q for k in range(254) for v in (1 << k, (1 << k) - 1, (1 << k) + 1, Q - (1 << k), Q - (1 << k) + 1)}
               | {Q - 1, Q - 2, (Q - 1) // 2, (Q + 1) // 2, TWO256 % Q, pow(TWO256, 2, Q), *WORDS})


def inverse(v):
    return pow(v, -1, Q) * TWO256 * TWO256 % Q if v else 0


def test_inverse(gpu):
    rnd = np.random.default_rng(12)
    items = [[v] for v in EDGES] + [[random_element(rnd, Q)] for _ in range(20000)]
    for (v,), (got,) in zip(items, run(gpu, 1, items, 8)):
        assert got == inverse(v), hex(v)


def test_inverse_fq2(gpu):
    rnd = np.random.default_rng(13)
    edges = EDGES[::7] + [0, 1, Q - 1]
    items = [[a, b] for a in edges for b in (0, 1, Q - 1, edges[int(rnd.integers(0, len(edges)))])]
    items += [[b, a] for a, b in items] + [[random_element(rnd, Q), random_element(rnd, Q)] for _ in range(4000)]
    for (a, b), got in zip(items, run(gpu, 2, items, 16)):
        norm = pow(a * a + b * b, -1, Q) if a or b else 0  # of Montgomery words: 1/x R = (a - b u) / norm R^2
        assert got == [a * norm * TWO256 * TWO256 % Q, -b * norm * TWO256 * TWO256 % Q], (hex(a), hex(b))


def test_products_by_constants(gpu):
    rnd = np.random.default_rng(14)
    ones = sum(0xFFFFFFFF << (64 * i) for i in range(4))
    xs = [0, 1, R - 1, 2 * R - 1, 4 * R - 1, TWO256 - 1, ones, ones << 32, (1 << 192) - 1]
    ms = [0, 1, 2, R - 1, R - 2, R // 2, TWO256 % R, pow(TWO256, 2, R)] + [R - k for k in range(3, 40)]
    items = [[x, m] for x in xs for m in ms]
    items += [[int.from_bytes(rnd.bytes(32), "little"), random_element(rnd, R)] for _ in range(4000)]
    unmont = pow(TWO256, -1, R)
    for (x, m), (p, w, quotient) in zip(items, run(gpu, 3, items, 24)):
        assert w == m * unmont % R and quotient == w * TWO256 // R, hex(m)
        if x < TWO256 - (1 << 227):
            assert p % R == x * w % R and p * TWO256 < R * (TWO256 + x + (1 << 227)), (hex(x), hex(m))


def test_unknown_operation(gpu):
    with pytest.raises(ZkGpuError, match="field operation must be 0..3"):
        run(gpu, 4, [[1]], 8)
