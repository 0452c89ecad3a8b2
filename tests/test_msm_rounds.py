"""The affine rounds of the accumulation, at sizes where plans use them: pairs of equal and opposite
points, infinity on either side, buckets of every fill of their last group, hot buckets, empty input,
against the oracle; batches, passes and the plan's switches."""
import numpy as np
import pytest

from common import R, fr_words, gpu_msm, msm_ref, random_fr, random_points
from oracle import bn254
from zk_gpu import Group, Msm, xyzz_to_affine, xyzz_to_affine_g2
from zk_gpu.msm import affine_words
from zk_gpu.synthetic import scalar_distribution

pytestmark = pytest.mark.gpu
SIZE = {"G1": (1 << 19) + 37, "G2": (1 << 18) - 9999}  # above the least entries of the rule (2^23 and 2^22)
GROUP = {"G1": Group.G1, "G2": Group.G2}


def pool(group, count, n):
    """n points drawn from `count` distinct ones, half of them negated."""
    aw = GROUP[group].affine_words()
    some = random_points(group, 51, count).reshape(count, aw)
    neg = some.copy()
    for row in neg:
        for k in range(aw // 2, aw, 8):
            y = bn254.from_words32(row[k: k + 8])
            row[k: k + 8] = bn254.words32((bn254.Q - y) % bn254.Q)
    both = np.concatenate([some, neg])
    pick = np.random.default_rng(52).integers(0, len(both), size=n)
    return both[pick].reshape(-1)


def inputs(group, what, n):
    aw = GROUP[group].affine_words()
    if what == "random":
        return random_points(group, 53, n), random_fr(54, n)
    if what == "few points and their negatives":
        return pool(group, 3, n), random_fr(55, n)
    if what == "one point":
        return np.tile(random_points(group, 56, 1), n), random_fr(57, n)
    if what == "half infinity":
        b = pool(group, 200, n).reshape(n, aw)
        b[np.random.default_rng(58).random(n) < 0.5] = 0
        return b.reshape(-1), random_fr(59, n)
    if what == "all infinity":
        return np.zeros(n * aw, dtype=np.uint32), random_fr(60, n)
    if what == "zero scalars":
        return pool(group, 50, n), np.zeros(8 * n, dtype=np.uint32)
    if what == "hot buckets":
        s = np.resize(fr_words([1, 1, 1, 2, R - 1, 1 << 40, 7]), 8 * n)
        return pool(group, 500, n), s
    return pool(group, 500, n), scalar_distribution(n, what, 61)  # "sparse", "r-1"


@pytest.mark.parametrize("group", ["G1", "G2"])
@pytest.mark.parametrize("what", ["random", "few points and their negatives", "one point", "half infinity", "all infinity",
                                  "zero scalars", "hot buckets", "sparse", "r-1"])
def test_rounds_match_oracle(gpu, group, what):
    n = SIZE[group]
    bases, scalars = inputs(group, what, n)
    want = msm_ref(group, bases, scalars)
    assert np.array_equal(gpu_msm(gpu, bases, scalars, group=GROUP[group]), want), (group, what)


@pytest.mark.parametrize("group", ["G1", "G2"])
def test_rounds_with_the_plan_switches(gpu, group):
    """One plan through forms with and without rounds, passes of sizes on both sides of the rule,
    GLV on and off and the fixed-base mode, back and forth."""
    grp, n = GROUP[group], SIZE[group]
    bases, scalars = inputs(group, "few points and their negatives", n)
    want = msm_ref(group, bases, scalars)
    base_buf, scalar_buf = Msm.upload_bases(gpu, bases), gpu.buffer(scalars)
    conv = xyzz_to_affine if group == "G1" else xyzz_to_affine_g2

    def check(msm, b, what):
        for _ in range(2):
            got = affine_words(conv(gpu.read(msm.run(gpu, b, scalar_buf), grp.xyzz_words())), grp)
            assert np.array_equal(got, want), (group, what)

    c = Msm.default_window(n)
    msm = Msm.for_group(gpu, grp, n, c)
    default = msm.params()["variant"]
    for variant in (default, 1, default):
        msm.set_variant(variant)
        check(msm, base_buf, variant)
    for chunk in (n // 2, 1000 if group == "G1" else 30000, n - 1, 0):
        msm.set_chunk(chunk)
        check(msm, base_buf, ("chunk", chunk))
    if group == "G1":
        for glv in (False, True):
            msm.set_glv(glv)
            check(msm, base_buf, ("glv", glv))
    table = Msm.fixed_base_table(gpu, grp, base_buf, n, c)
    msm.set_fixed_base(True)
    check(msm, table, "fixed base")


def test_rounds_report_the_entries(gpu):
    """The entry count of a run is the nonzero digits', not the padded places'."""
    import ctypes

    from zk_gpu._lib import check, lib
    n = SIZE["G1"]
    bases, _ = inputs("G1", "few points and their negatives", n)
    scalars = np.zeros((n, 8), dtype=np.uint32)
    scalars[:1000, 0] = 5  # one nonzero digit each
    msm = Msm(gpu, n, Msm.default_window(n))
    msm.run(gpu, Msm.upload_bases(gpu, bases), gpu.buffer(scalars.reshape(-1)))
    entries = ctypes.c_uint64()
    check(lib().zkg_msm_last_entries(msm._h, ctypes.byref(entries)))
    assert entries.value == 1000


def test_server_slots_with_and_without_rounds(gpu):
    """A proof's captured graph with the rounds' side stream in it, and the slot a small budget gets."""
    from test_serving import affine_points, make_request
    from zk_gpu.serving import Server
    log_m = 18
    n = 1 << log_m
    g1, g2 = pool("G1", 100, n), pool("G2", 100, n)
    keys = Msm.upload_bases(gpu, g1), Msm.upload_bases(gpu, g2)
    outs, used = [], []
    for budget in (0, 1 << 30):
        server = Server(gpu, lanes=2, hbm_budget_bytes=budget, coset_g=7)
        server.add_key(n, *keys)
        for _ in range(2):
            req = make_request(log_m, 71)
            server.wait(server.submit(req))
        used.append(server.stats()["bytes_used"])
        outs.append((affine_points(req.points()), req.h()))
        server.close()
    assert used[0] > used[1]
    assert np.array_equal(outs[0][1], outs[1][1])
    for a, b in zip(outs[0][0], outs[1][0]):
        assert np.array_equal(a, b)
    assert np.array_equal(outs[0][0][3], msm_ref("G2", g2, req.g2.array))
    assert np.array_equal(outs[0][0][0], msm_ref("G1", g1, req.g1[0].array))
