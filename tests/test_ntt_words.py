"""The word form of the transform (form 2): every tile size and stage parity its plans use, on the
values that reach the ends of its unreduced ranges, against the oracle."""
import numpy as np
import pytest

from common import fr_words, gpu_ntt, random_fr
from oracle import bn254, cpu
from zk_gpu import Ntt

pytestmark = pytest.mark.gpu
R = bn254.R


def inputs(log_n):
    n = 1 << log_n
    x = random_fr(9000 + log_n, n)
    ends = fr_words([R - 1, 0, 1, R - 2, (R - 1) // 2, (1 << 253) - 1, (1 << 32) - 1, R - (1 << 32)])
    mixed = x.copy().reshape(n, 8)
    mixed[::3] = np.resize(ends.reshape(-1, 8), mixed[::3].shape)
    return {"random": x, "largest": np.tile(fr_words([R - 1]), n), "alternating": np.tile(fr_words([R - 1, 0]), n // 2),
            "ends": mixed.reshape(-1)}


@pytest.mark.parametrize("log_n", range(10, 20))
def test_word_form_matches_oracle(gpu, log_n):
    for split in (None, 6, 7, 9, 10):
        ntt = Ntt(gpu, log_n)
        ntt.set_variant(2)
        if split is not None:
            if log_n == 10:
                continue  # one tile: a single split
            ntt.set_max_stages(split)
        for name, x in inputs(log_n).items():
            want = cpu.ntt(x)
            assert np.array_equal(gpu_ntt(gpu, ntt, x), want), (log_n, split, name, "forward")
            assert np.array_equal(gpu_ntt(gpu, ntt, want, inverse=True), x), (log_n, split, name, "inverse")
