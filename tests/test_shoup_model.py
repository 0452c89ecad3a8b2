"""Integer model of the products by constants with a precomputed quotient (csrc/field_shoup.cuh: high_product,
mul), run on the CPU to pin the bound that the transform's unreduced elements rely on.

The model keeps what the device code keeps: the products of words i of x and j of the quotient with
i + j >= 6. The residue is congruent to x w modulo r and below r (1 + x / 2^256 + 2^-29), which is below
1.757r for x < 4r."""
import random

from oracle.bn254 import R

TWO256 = 1 << 256
M32 = (1 << 32) - 1


def quotient(x, w_prime):
    xs, ws = ([(v >> (32 * i)) & M32 for i in range(8)] for v in (x, w_prime))
    return sum(xs[i] * ws[j] << (32 * (i + j)) for i in range(8) for j in range(8) if i + j >= 6) >> 256


def product(x, w):
    return x * w - quotient(x, w * TWO256 // R) * R


def constants(rnd):
    """Random ones, and those for which w 2^256 / r loses the most or the least to its floor."""
    inv = pow(TWO256, -1, R)
    special = [(R - k) * inv % R for k in range(1, 40)] + [k * inv % R for k in range(1, 40)]
    return [0, 1, 2, R - 1, R - 2, R // 2] + special + [rnd.randrange(R) for _ in range(300)]


def operands(rnd, top):
    ones = sum(M32 << (64 * i) for i in range(4))
    near = [top - 1 - k for k in range(20)] + [ones % top, (ones << 32) % top, (1 << 192) - 1, 0, 1]
    return near + [rnd.randrange(top) for _ in range(100)]


def test_residue_and_bound():
    rnd = random.Random(7)
    worst = 0
    for w in constants(rnd):
        for top in (4 * R, TWO256):
            for x in operands(rnd, top):
                p = product(x, w)
                assert 0 <= p and p % R == x * w % R
                assert p * TWO256 < R * (TWO256 + x + (1 << 227))
                if x < 4 * R:
                    worst = max(worst, p)
    assert 1.70 * R < worst < 1.757 * R  # the bound is near what occurs


def test_products_left_out_are_below_a_unit():
    """All words of both factors at their largest: what the 21 products would have added to the quotient."""
    left_out = sum(M32 * M32 << (32 * (i + j)) for i in range(8) for j in range(8) if i + j < 6)
    assert left_out < 1 << 227  # 2^-29 of 2^256
