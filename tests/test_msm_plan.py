"""What a plan holds and reports between runs."""
import ctypes
import threading

import numpy as np
import pytest

from common import random_fr, random_points
from zk_gpu import Gpu, Group, Msm, xyzz_to_affine
from zk_gpu._lib import check, lib
from zk_gpu.synthetic import generator_multiples, uniform_scalars

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


# ------------------------------------------------------------------ the affine rounds' scratch


def large(gpu, log_n=22):
    """A G1 plan with affine rounds, resident inputs and the run that reads its affine result."""
    n = 1 << log_n
    bases = generator_multiples(gpu, Group.G1, uniform_scalars(n, 3), mont256=True)
    scalars = gpu.buffer(uniform_scalars(n, 4))
    msm = Msm(gpu, n, Msm.default_window(n))
    return msm, bases, scalars, lambda: xyzz_to_affine(gpu.read(msm.run(gpu, bases, scalars), 32))


def free_bytes() -> int:
    import torch
    return torch.cuda.mem_get_info(0)[0]


GIB = 1 << 30


def test_a_buffer_that_fits_without_the_rounds_fits(gpu):
    """With the device full up to 1 GiB, a buffer of 2 GiB finds room in the plan's rounds' scratch (about
    3 GiB), and the plan goes on with the same result."""
    msm, bases, scalars, run = large(gpu)
    want = run()
    ballast = gpu.empty_buffer((free_bytes() - GIB) // 4)
    wanted = gpu.empty_buffer(2 * GIB // 4)
    assert run() == want
    wanted.free()
    ballast.free()
    assert run() == want


def test_an_allocation_that_cannot_fit_takes_nothing(gpu):
    from zk_gpu import ZkGpuError
    msm, _, _, run = large(gpu, 20)
    want, before = run(), msm.rounds()
    assert before[0] > 0 and before[1] > 0
    with pytest.raises(ZkGpuError):
        gpu.empty_buffer(1 << 38)
    assert msm.rounds() == before and run() == want


def test_a_captured_plan_keeps_its_scratch(gpu):
    """A batch's graph holds the scratch's addresses: nothing is given back while the plan may be in one."""
    from zk_gpu import Batch, ZkGpuError
    msm, bases, scalars, run = large(gpu)
    want, before = run(), msm.rounds()
    result = gpu.empty_buffer(32)
    batch = Batch(gpu)
    batch.add_msm(msm, bases, scalars, result)
    batch.capture()
    ballast = gpu.empty_buffer((free_bytes() - GIB) // 4)
    with pytest.raises(ZkGpuError, match="out of memory"):
        gpu.empty_buffer(2 * GIB // 4)
    assert msm.rounds() == before
    batch.launch()
    assert xyzz_to_affine(gpu.read(result, 32)) == want
    ballast.free()
    batch.close()


def test_rounds_switched_off_and_on(gpu):
    msm, _, _, run = large(gpu, 20)
    want, (rounds, scratch) = run(), msm.rounds()
    held = free_bytes()
    msm.set_rounds(False)
    assert msm.rounds() == (0, 0) and free_bytes() - held > 0.9 * scratch
    assert run() == want
    msm.set_rounds(True)
    assert msm.rounds() == (rounds, scratch)
    assert run() == want
    msm.set_variant(1)  # not the plan's own form: no rounds, the scratch stays
    assert msm.rounds() == (0, scratch) and run() == want


def test_a_change_that_does_not_fit_leaves_an_error(gpu):
    """A slice whose scratch the device has no room for is refused, and so are runs (the plan has lost the
    scratch of before, not only part of it) until a slice that fits."""
    from zk_gpu import ZkGpuError
    n = 1 << 22
    bases = generator_multiples(gpu, Group.G1, uniform_scalars(n, 3), mont256=True)
    scalars = gpu.buffer(uniform_scalars(n, 4))
    msm = Msm(gpu, n, Msm.default_window(n))
    msm.set_chunk(1 << 16)
    run = lambda: xyzz_to_affine(gpu.read(msm.run(gpu, bases, scalars), 32))  # noqa: E731
    want = run()
    ballast = gpu.empty_buffer((free_bytes() - (GIB >> 2)) // 4)
    with pytest.raises(ZkGpuError, match="out of memory"):
        msm.set_chunk(n)
    with pytest.raises(ZkGpuError, match="no scratch"):
        run()
    with pytest.raises(ZkGpuError, match="no scratch"):
        msm.profile(gpu, bases, scalars)
    msm.set_chunk(1 << 16)
    assert run() == want
    ballast.free()
    msm.set_chunk(0)
    assert run() == want


def test_scratch_given_back_while_another_thread_runs_the_plan(gpu):
    """One thread runs the plan over and over, another one's allocation takes the rounds' scratch."""
    msm, bases, scalars, run = large(gpu)
    want = run()
    results, stop = [], threading.Event()

    def runs():
        while not stop.is_set():
            results.append(run())

    ballast = gpu.empty_buffer((free_bytes() - GIB) // 4)
    thread = threading.Thread(target=runs)
    thread.start()
    try:
        wanted = Gpu().empty_buffer(2 * GIB // 4)  # another context, another stream
    finally:
        stop.set()
        thread.join()
    assert msm.rounds() == (0, 0)
    assert results and all(r == want for r in results) and run() == want
    wanted.free()
    ballast.free()
