"""Words at or above the modulus (a caller's mistake): a transform or an accumulation in any form reads and
writes nothing outside its buffers and tables, so the call returns, and the plan and the device serve the
next call as before. Transforms of words below 2r are right modulo r in the forms that hold sums below 2r."""
import numpy as np
import pytest

from common import gpu_msm, msm_ref, random_fr, random_points
from oracle import bn254, cpu
from zk_gpu import Group, Msm, Ntt

pytestmark = pytest.mark.gpu
R = bn254.R


def above(seed, count):
    """Words of every size up to 2^256 - 1."""
    rnd = np.random.default_rng(seed)
    w = rnd.integers(0, 1 << 32, size=(count, 8), dtype=np.uint64).astype(np.uint32)
    w[::5] = 0xFFFFFFFF
    w[1::5] = 0
    w[2::5] = bn254.words32(4 * R)
    return w.reshape(-1)


@pytest.mark.parametrize("form", range(5))
@pytest.mark.parametrize("log_n", [10, 13])
def test_transforms(gpu, log_n, form):
    n = 1 << log_n
    ntt = Ntt(gpu, log_n)
    ntt.set_variant(form)
    good = random_fr(3, n)
    for inverse in (False, True):
        run = ntt.inverse if inverse else ntt.forward
        buf = gpu.buffer(above(4 + inverse, n))
        run(gpu, buf)
        gpu.wait()  # a fault would surface here
        buf = gpu.buffer(good)
        run(gpu, buf)
        assert np.array_equal(gpu.read(buf, good.size), cpu.ntt(good, inverse)), (log_n, form, inverse)


@pytest.mark.parametrize("form", [2, 3])
@pytest.mark.parametrize("log_n", [10, 15])
def test_transforms_of_words_below_2r(gpu, log_n, form):
    n = 1 << log_n
    x = random_fr(5, n).reshape(n, 8)
    y = x.copy()
    y[::2] = [bn254.words32(bn254.from_words32(v) + R) for v in x[::2]]
    ntt = Ntt(gpu, log_n)
    ntt.set_variant(form)
    for inverse in (False, True):
        buf = gpu.buffer(y.reshape(-1))
        (ntt.inverse if inverse else ntt.forward)(gpu, buf)
        assert np.array_equal(gpu.read(buf, 8 * n), cpu.ntt(x.reshape(-1), inverse)), (log_n, form, inverse)


@pytest.mark.parametrize("group,forms", [("G1", range(7)), ("G2", range(5))])
def test_accumulations(gpu, group, forms):
    n = 3000
    grp = Group.G1 if group == "G1" else Group.G2
    bases, scalars = random_points(group, 6, n), random_fr(7, n)
    want = msm_ref(group, bases, scalars)
    bad = gpu.buffer(above(8, n * grp.affine_words() // 8))
    good, sb = Msm.upload_bases(gpu, bases), gpu.buffer(scalars)
    for form in forms:
        msm = Msm.for_group(gpu, grp, n, Msm.default_window(n))
        msm.set_variant(form)
        msm.run(gpu, bad, sb)
        gpu.wait()
        msm.close()
        assert np.array_equal(gpu_msm(gpu, bases, scalars, group=grp, variant=form), want), (group, form)
