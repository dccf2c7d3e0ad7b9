"""Copies between pageable host memory and the device (csrc/host_copy.cu) at the sizes where they change form - one piece, one
segment, a full ring, and one element on either side - bit for bit, and from several threads at once."""
import threading

import numpy as np
import pytest

from mimir_framework_b200 import abi

pytestmark = pytest.mark.gpu

PIECE, SEGMENT, RING = 256 << 10, 2 << 20, 8


@pytest.fixture(scope="module")
def rt():
    from mimir_framework_b200 import runtime

    runtime.init(0)
    return runtime


@pytest.mark.parametrize("bytes_", [64 << 10, PIECE, 2 * PIECE, SEGMENT, 4 * SEGMENT, RING * SEGMENT, 2 * RING * SEGMENT + PIECE])
@pytest.mark.parametrize("extra", [-1, 0, 1])
def test_round_trip_is_exact(rt, bytes_, extra):
    x = np.random.default_rng(bytes_ + extra).standard_normal(bytes_ // 4 + extra, dtype=np.float32)
    assert np.array_equal(rt.eltwise(abi.ELT_RELU, x), np.maximum(x, 0))


def test_threads_do_not_mix(rt):
    bad = []

    def work(seed):
        rt.init(0)
        for i in range(6):
            x = np.random.default_rng(seed * 100 + i).standard_normal(300_000 * (1 + seed % 3), dtype=np.float32)
            if not np.array_equal(rt.eltwise(abi.ELT_RELU, x), np.maximum(x, 0)):
                bad.append((seed, i))

    ts = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


def test_idle_call_buffers_are_not_counted(rt):
    before = rt.guard_stats()["current"]
    rt.eltwise(abi.ELT_RELU, np.ones(1 << 20, np.float32))
    assert rt.guard_stats()["current"] == before
