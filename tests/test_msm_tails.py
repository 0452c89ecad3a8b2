"""The bucket reduction and window combination (marginals, bit sums, folds and the lane-group
additions under them): every window size, with buckets that are equal, opposite, empty or alone, so
that additions meet equal points, opposite points and infinity at every level."""
import numpy as np
import pytest

from common import fr_words, gpu_msm, msm_ref, random_fr, random_points
from oracle import bn254
from zk_gpu import Group

pytestmark = pytest.mark.gpu
R = bn254.R


def negated(bases, aw):
    """The points' negatives (plain affine words): y -> q - y in every component."""
    out = bases.reshape(-1, aw).copy()
    for row in out:
        for k in range(aw // 2, aw, 8):
            y = bn254.from_words32(row[k: k + 8])
            row[k: k + 8] = bn254.words32((bn254.Q - y) % bn254.Q)
    return out.reshape(-1)


def cases(group, c):
    aw = 16 if group == "G1" else 32
    half = 1 << (c - 1)
    n = min(half, 1500 if group == "G1" else 300)
    one = random_points(group, 31, 1)
    same = np.tile(one, n)
    yield "every bucket the same point", same, fr_words(range(1, n + 1))
    flip = same.reshape(n, aw).copy()
    flip[1::2] = negated(one, aw)
    yield "buckets alternately opposite", flip.reshape(-1), fr_words(range(1, n + 1))
    flip[n // 2:] = negated(same[: aw * (n - n // 2)], aw).reshape(-1, aw)
    yield "halves opposite", flip.reshape(-1), fr_words(range(1, n + 1))
    yield "one bucket, the last", one, fr_words([half])
    yield "one bucket, the first", one, fr_words([1])
    yield "first and last windows", np.tile(one, 3), fr_words([1, R - 1, 1 << 253])
    yield "random", random_points(group, 32, n), random_fr(33, n)


@pytest.mark.parametrize("group,c", [("G1", c) for c in range(9, 21)] + [("G2", c) for c in (9, 10, 12, 13, 14, 15, 16, 18)])
def test_bucket_reduction(gpu, group, c):
    for what, bases, scalars in cases(group, c):
        want = msm_ref(group, bases, scalars)
        for glv in ((None, False) if group == "G1" else (None,)):
            got = gpu_msm(gpu, bases, scalars, (c, None), Group.G1 if group == "G1" else Group.G2, glv=glv)
            assert np.array_equal(got, want), (group, c, what, glv)


@pytest.mark.parametrize("group", ["G1", "G2"])
def test_long_runs_of_heads(gpu, group):
    """One bucket, or a few, over many accumulation threads: runs of partial sums that end at, before
    and after a merge tile's edge, fill several tiles, and continue through several levels."""
    grp = Group.G1 if group == "G1" else Group.G2
    aw = grp.affine_words()
    tile = 256 if group == "G1" else 128
    sizes = [2, 3, tile - 1, tile, tile + 1, 2 * tile + 1, 5 * tile + 7] + ([tile * tile + tile + 2] if group == "G1" else [])
    pool = random_points(group, 41, max(sizes))
    for n in sizes:
        bases = pool[: aw * n]
        for scalars in (np.tile(fr_words([1]), n), np.tile(fr_words([3, 3, 3, 1, 5]), n)[: 8 * n],
                        np.concatenate([np.tile(fr_words([2]), n // 2), np.tile(fr_words([7]), n - n // 2)])):
            want = msm_ref(group, bases, scalars)
            for items in (1, 2, 3):
                got = gpu_msm(gpu, bases, scalars, (9, items), grp)
                assert np.array_equal(got, want), (group, n, items)
