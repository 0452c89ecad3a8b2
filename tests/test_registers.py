"""What the compiler reports of kernels whose block's bound sets their registers (ptxas -v, kept by the
build beside the objects)."""
import os
import re

import pytest

from conftest import ROOT

REPORT = os.path.join(ROOT, "zk-gpu_b200", "_build", "msm.ptxas.txt")


def kernels(name):
    """{mangled name: (frame, spill stores, spill loads)} of the kernels whose name contains `name`."""
    text = open(REPORT).read()
    found = re.findall(r"Function properties for (\S+)\s+(\d+) bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads",
                       text)
    return {k: tuple(map(int, v)) for k, *v in found if name in k}


@pytest.mark.skipif(not os.path.exists(REPORT), reason="the library was not built here")
def test_window_combination_of_the_default_windows_reloads_nothing():
    """Default windows are 11 to 16 bits, so at most 24 of them: 12 warps (in G2 a form of its own, Lj12)."""
    got = kernels("msm_combine_lanes")
    g1 = [v for k, v in got.items() if "Fq2T" not in k]
    g2 = [v for k, v in got.items() if "Fq2T" in k and "Lj12" in k]
    assert g1 and g2, got
    assert all(loads == 0 for _, _, loads in g1 + g2), got
