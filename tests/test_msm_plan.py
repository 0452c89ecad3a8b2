"""What a plan holds and reports between runs."""
import ctypes

import numpy as np
import pytest

from common import random_fr, random_points
from zk_gpu import Group, Msm
from zk_gpu._lib import check, lib

pytestmark = pytest.mark.gpu


def last_entries(msm) -> int:
    entries = ctypes.c_uint64()
    check(lib().zkg_msm_last_entries(msm._h, ctypes.byref(entries)))
    return entries.value


def test_the_last_runs_entry_count_outlives_a_switch(gpu):
    """zkg_msm_last_entries is the last run's, whatever mode the plan has been switched to since."""
    n, c = 3000, 11
    msm = Msm.for_group(gpu, Group.G2, n, c)
    bases = Msm.upload_bases(gpu, random_points("G2", 1, n))
    scalars = np.zeros((n, 8), dtype=np.uint32)
    scalars[:700, 0] = 5  # one nonzero digit each
    few, many = gpu.buffer(scalars.reshape(-1)), gpu.buffer(random_fr(2, n))
    msm.run(gpu, bases, few)
    assert last_entries(msm) == 700
    msm.set_fixed_base(True)
    assert last_entries(msm) == 700
    table = Msm.fixed_base_table(gpu, Group.G2, bases, n, c)
    msm.run(gpu, table, many)
    entries = last_entries(msm)
    assert entries > 20 * n
    msm.set_fixed_base(False)
    assert last_entries(msm) == entries
    msm.run(gpu, bases, many)
    assert last_entries(msm) == entries
