"""The server's HBM budget holds as many slots as without affine rounds: slots have the rounds' scratch only
while nothing else needs the bytes."""
import re
import threading

import numpy as np
import pytest

from test_serving import affine_points, make_request, same_points
from zk_gpu import Group, ZkGpuError
from zk_gpu.serving import Server
from zk_gpu.synthetic import generator_multiples, uniform_scalars

pytestmark = pytest.mark.gpu
LARGE, SMALL = 18, 17  # of the two, slots of 2^18 have rounds (G2)


class Sizes:
    """Bytes of slots: as the server counts them once made, and as it estimates them before."""

    def __init__(self, gpu, key):
        self.key = key
        # 64 lanes: no slot of a budget below 128 of them has rounds
        server = self.server(gpu, 64, 16 << 30)
        server.reserve(LARGE, 1)
        self.large = server.stats()["bytes_used"]
        server.reserve(SMALL, 1)
        self.small = server.stats()["bytes_used"] - self.large
        server.close()
        server = self.server(gpu, 64, 1)
        self.large_estimate, self.small_estimate = (self.estimate(server, k) for k in (LARGE, SMALL))
        server.close()
        server = self.server(gpu, 1, 16 << 30)
        server.reserve(LARGE, 1)
        self.large_with_rounds = server.stats()["bytes_used"]
        server.close()
        self.slots = 9  # of the large size without rounds
        self.budget = (self.slots - 1) * max(self.large, self.large_estimate) + self.large_estimate + (64 << 20)

    @staticmethod
    def estimate(server, log_m):
        with pytest.raises(ZkGpuError) as e:
            server.reserve(log_m, 1)
        return int(re.search(r"(\d+) needed", str(e.value)).group(1))

    def small_beside(self, large_slots):
        """How many small slots fit beside large ones without rounds: more than beside large ones with them."""
        count = (self.budget - large_slots * self.large) // max(self.small, self.small_estimate)
        assert count * self.small > self.budget - large_slots * self.large_with_rounds
        return count

    def server(self, gpu, lanes, budget):
        server = Server(gpu, lanes=lanes, hbm_budget_bytes=budget, coset_g=7)
        server.add_key(1 << LARGE, *self.key)
        return server


@pytest.fixture(scope="module")
def sizes(gpu):
    k = uniform_scalars(1 << LARGE, 5)
    s = Sizes(gpu, [generator_multiples(gpu, g, k, mont256=True) for g in (Group.G1, Group.G2)])
    assert s.large_with_rounds > 1.5 * s.large
    return s


@pytest.fixture(scope="module")
def expected(gpu, sizes):
    """Outputs of make_request(log_m, seed) on a server with all the memory."""
    server, known = sizes.server(gpu, 2, 0), {}

    def get(log_m, seed):
        if (log_m, seed) not in known:
            req = make_request(log_m, seed)
            server.wait(server.submit(req))
            known[log_m, seed] = affine_points(req.points()), req.h()
        return known[log_m, seed]

    yield get
    server.close()


def check_requests(server, expected, wanted):
    reqs = [make_request(log_m, seed) for log_m, seed in wanted]
    ids = [server.submit(r) for r in reqs]
    finish(server, expected, wanted, reqs, ids)


def finish(server, expected, wanted, reqs, ids):
    for i in ids:
        server.wait(i)
    for (log_m, seed), r in zip(wanted, reqs):
        points, h = expected(log_m, seed)
        assert same_points(affine_points(r.points()), points) and np.array_equal(r.h(), h), (log_m, seed)


def test_as_many_slots_of_one_size(gpu, sizes, expected):
    server = sizes.server(gpu, 1, sizes.budget)
    server.reserve(LARGE, sizes.slots)
    stats = server.stats()
    assert stats["slots"] == sizes.slots and stats["bytes_used"] <= stats["budget"]
    check_requests(server, expected, [(LARGE, 3)])
    server.close()


def test_slots_give_their_scratch_to_another_size(gpu, sizes, expected):
    server = sizes.server(gpu, 1, sizes.budget)
    server.reserve(LARGE, 2)
    assert server.stats()["bytes_used"] > 1.5 * 2 * sizes.large  # with rounds
    check_requests(server, expected, [(LARGE, 3)])
    count = sizes.small_beside(2)
    server.reserve(SMALL, count)
    stats = server.stats()
    assert stats["slots"] == 2 + count and stats["slots_evicted"] == 0 and stats["bytes_used"] <= stats["budget"]
    check_requests(server, expected, [(LARGE, 3), (SMALL, 4), (LARGE, 5)])
    with pytest.raises(ZkGpuError, match="does not fit the HBM budget"):
        server.reserve(LARGE, 4)
    check_requests(server, expected, [(SMALL, 6), (LARGE, 3)])
    assert server.stats()["slots_evicted"] == 0
    server.close()


def test_a_request_of_another_size_evicts_nothing(gpu, sizes, expected):
    server = sizes.server(gpu, 1, sizes.budget)
    count, left = 0, sizes.budget
    while left >= sizes.large_estimate:  # one by one: the first ones with rounds, the later ones without
        count += 1
        server.reserve(LARGE, count)
        left = sizes.budget - server.stats()["bytes_used"]
    assert server.stats()["bytes_used"] > count * sizes.large + (sizes.large_with_rounds - sizes.large)
    while left >= sizes.small_estimate:
        small = server.stats()["slots"] - count + 1
        server.reserve(SMALL, small)
        left = sizes.budget - server.stats()["bytes_used"]
    check_requests(server, expected, [(LARGE, 3), (16, 4), (LARGE, 5), (16, 6), (LARGE, 3)])
    stats = server.stats()
    assert stats["slots_evicted"] == 0 and stats["bytes_used"] <= stats["budget"]
    server.close()


def test_slots_at_work_give_their_scratch_when_done(gpu, sizes, expected):
    server = sizes.server(gpu, 1, sizes.budget)
    server.reserve(LARGE, 2)
    wanted = [(LARGE, 3 + 2 * (k & 1)) for k in range(4)]
    reqs = [make_request(log_m, seed) for log_m, seed in wanted]
    ids = [server.submit(r) for r in reqs]
    count = sizes.small_beside(2)
    server.reserve(SMALL, count)
    finish(server, expected, wanted, reqs, ids)
    stats = server.stats()
    assert stats["slots"] == 2 + count and stats["slots_evicted"] == 0 and stats["bytes_used"] <= stats["budget"]
    check_requests(server, expected, [(LARGE, 5), (SMALL, 4)])
    server.close()


def reserve_beside(server, log_m, count):
    """Starts reserve(log_m, count) in a thread and returns it with the bytes taken for the first slot, while
    that slot is still being made."""
    before = server.stats()["bytes_used"]
    thread = threading.Thread(target=server.reserve, args=(log_m, count))
    thread.start()
    while True:
        taken = server.stats()["bytes_used"] - before
        if taken or not thread.is_alive():
            return thread, taken


def test_a_slot_being_reserved_gives_its_scratch_to_one_asked_for_beside_it(gpu, sizes, expected):
    server = sizes.server(gpu, 1, 16 << 30)
    thread, estimate = reserve_beside(server, LARGE, 1)  # with rounds
    thread.join()
    server.close()
    server = sizes.server(gpu, 1, 2 * estimate)
    small = 0
    while 2 * estimate - server.stats()["bytes_used"] >= estimate + sizes.small_estimate:
        small += 1
        server.reserve(SMALL, small)
    thread, taken = reserve_beside(server, LARGE, 1)
    server.reserve(SMALL, small + 1)  # fits once the large slot is there and has given up its rounds
    thread.join()
    stats = server.stats()
    assert taken == estimate and stats["slots"] == small + 2 and stats["bytes_used"] <= stats["budget"]
    check_requests(server, expected, [(LARGE, 3), (SMALL, 4)])
    server.close()
