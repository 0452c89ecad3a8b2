"""What a transform plan takes on the device."""
import numpy as np
import pytest

from zk_gpu import Ntt, ZkGpuError
from zk_gpu.synthetic import uniform_scalars

pytestmark = pytest.mark.gpu


def test_a_plan_fits_where_the_smaller_tables_fit(gpu):
    """2^24 elements: 2.5 GiB with the default form's tables, 1.8 with form 3's. With 2.2 GiB left the plan is
    made, and transforms as one with all its memory does."""
    import torch
    log_n = 24
    x = uniform_scalars(1 << log_n, 5)
    data, free = gpu.buffer(x), lambda: torch.cuda.mem_get_info(0)[0]
    ntt = Ntt(gpu, log_n)
    assert ntt.params()["variant"] == 2
    ntt.forward(gpu, data)
    want = gpu.read(data, x.size)
    ntt.set_variant(3)  # its kernels are on the device before the memory is taken
    ntt.inverse(gpu, data)
    ntt.close()
    ballast = gpu.empty_buffer((free() - 2252 * (1 << 20)) // 4)
    small = Ntt(gpu, log_n)
    assert small.params()["variant"] == 3
    small.forward(gpu, data)
    assert np.array_equal(gpu.read(data, x.size), want)
    with pytest.raises(ZkGpuError, match="out of memory"):
        small.set_variant(2)  # refused, and the plan stays as it was
    assert small.params()["variant"] == 3
    small.inverse(gpu, data)
    assert np.array_equal(gpu.read(data, x.size), x)
    ballast.free()


def test_a_form_whose_tables_came_halfway_is_refused_again(gpu):
    """Forms 0 and 1 keep tables for each direction. Where the device has room for one of the two, the form is
    refused as often as it is asked for, and taken with all its tables once there is room."""
    import torch
    log_n = 22
    x = uniform_scalars(1 << log_n, 6)
    data, free = gpu.buffer(x), lambda: torch.cuda.mem_get_info(0)[0]
    ntt = Ntt(gpu, log_n)
    ntt.forward(gpu, data)
    want = gpu.read(data, x.size)
    ntt.inverse(gpu, data)
    for form, table in ((0, 64 << 20), (1, 80 << 20)):
        other = Ntt(gpu, 10)  # its kernels are on the device before the memory is taken
        other.set_variant(form)
        small = gpu.buffer(x[: 8 << 10])
        other.forward(gpu, small)
        other.inverse(gpu, small)
        gpu.wait()
        ballast = gpu.empty_buffer((free() - table * 3 // 2) // 4)
        for _ in range(2):
            with pytest.raises(ZkGpuError, match="out of memory"):
                ntt.set_variant(form)
            assert ntt.params()["variant"] != form
        ballast.free()
        ntt.set_variant(form)
        ntt.forward(gpu, data)
        assert np.array_equal(gpu.read(data, x.size), want)
        ntt.inverse(gpu, data)
        assert np.array_equal(gpu.read(data, x.size), x)
