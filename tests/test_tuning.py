"""The candidates that the MSM tuner times."""
import pytest

from zk_gpu import Group, Msm
from zk_gpu.autotune import search_msm
from zk_gpu.synthetic import generator_multiples, uniform_scalars

pytestmark = pytest.mark.gpu


def test_candidates_of_a_size_with_affine_rounds(gpu):
    """The plan's own points per thread are among them, and the fixed ones leave the device a few waves of
    threads: in the form with rounds a thread's points are sums of 2^rounds entries."""
    n, c = 1 << 19, 14
    bases = generator_multiples(gpu, Group.G1, uniform_scalars(n, 5), mont256=True)
    scalars = gpu.buffer(uniform_scalars(n, 6))
    msm = Msm(gpu, n, c)
    assert Msm.default_window(n) == c and msm.rounds()[0] == 2
    entries = 2 * n * msm.windows()[0]
    msm.close()

    def points(variant):
        return {r["item_points"] for r in search_msm(gpu, Group.G1, n, bases, scalars, reps=1)
                if (r["c"], r["glv"], r["variant"]) == (c, 1, variant)}

    waves = 148 * 256
    for variant, sums in ((4, entries // 4), (1, entries)):
        assert points(variant) <= {0} | {k for k in (16, 32, 64, 128, 256) if k == 16 or sums // k >= waves}, variant
    assert {0, 16, 32, 64} <= points(4)
