"""Copies between pageable host memory and the device (csrc/host_copy.cu) at the sizes where they change form - one piece, one
segment, a full ring, and one element on either side - bit for bit, and from several threads at once."""
import threading
import time

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


@pytest.mark.parametrize("bytes_", [128 << 10, 512 << 10, (512 << 10) + (64 << 10), 3 * (512 << 10), 3 << 20, (3 << 20) + (64 << 10), (3 * 512 << 10) + (16 << 20), 19 << 20])
@pytest.mark.parametrize("extra", [-1, 0, 1])
def test_round_trip_at_the_edges_of_uneven_segments(rt, bytes_, extra):
    x = np.random.default_rng(bytes_ + extra).standard_normal(bytes_ // 4 + extra, dtype=np.float32)
    assert np.array_equal(rt.eltwise(abi.ELT_RELU, x), np.maximum(x, 0))


@pytest.mark.parametrize("batch,n,inputs", [(1, 1, 1), (3, 5, 2), (1, 1023, 1), (1, 1025, 1), (2, 4097, 2), (4, 1025, 7), (2, 33, 9),
                                            (1, 16385, 3), (1, 65535, 1), (1, 65536, 1), (1, 65537, 1), (8, 8192, 2), (3, 21846, 2)])
def test_small_tensors_through_the_staging_block(rt, batch, n, inputs):
    """Results around a CTA's 4 KB, the 64 KB of a launch's CTAs together and the block's 256 KB, of inputs of each sample's own and broadcast ones,
    which change from call to call."""
    descs, names = [], ["x"] + [f"i{k}" for k in range(1, inputs)]
    for k in range(1, inputs):
        descs.append(abi.make_desc(f"a{k}", "Add", inputs=["x" if k == 1 else f"s{k - 1}", names[k]], output="x" if k + 1 == inputs else f"s{k}"))
    if not descs:
        descs.append(abi.make_desc("r", "ReLU", inputs=["x"], output="x"))
    mod = rt.GraphModel(descs)
    mod.plan({m: (n, k % 2 == 1) for k, m in enumerate(names)}, batch)
    for seed in range(4):
        r = np.random.default_rng(seed)
        a = {m: r.standard_normal((1 if k % 2 else batch, n), dtype=np.float32) for k, m in enumerate(names)}
        want = np.maximum(a["x"], 0) if inputs == 1 else a["x"]
        for m in names[1:]:
            want = want + a[m]
        got = mod.forward({m: (a[m].ravel(), k % 2 == 1) for k, m in enumerate(names)}, batch, n)
        assert np.array_equal(got.reshape(batch, n), want.reshape(batch, n))
    mod.close()


@pytest.mark.parametrize("scale", [0.0, 1e-42, 1e-30, 2.0**-13, 1.0, 3.0, 1e30])
@pytest.mark.parametrize("rows,k,n", [(17, 64, 40), (600, 100, 1000)])
def test_weight_scale_found_on_the_device(rt, scale, rows, k, n):
    """One call on host arrays has the bits of a planned model, whose weight scale is found on the host."""
    r = np.random.default_rng(k)
    x, w = r.standard_normal((rows, k), dtype=np.float32), (r.standard_normal((n, k)) * scale).astype(np.float32)
    b = r.standard_normal(n, dtype=np.float32)
    mod = rt.GraphModel([abi.make_desc("l", "Linear", inputs=["x"], output="x", in_features=k, out_features=n, seq_len=rows, use_bias=1, params_count=n * k + n)])
    mod.upload_weights(0, np.concatenate([w.ravel(), b]))
    mod.plan({"x": (rows * k, False)}, 1)
    want = mod.forward({"x": (x.ravel(), False)}, 1, rows * n).ravel()
    mod.close()
    assert np.array_equal(rt.linear_forward(x.ravel(), w.ravel(), b, rows, k, n), want, equal_nan=True)  # (1e30 leaves the planes' range either way)


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


@pytest.mark.parametrize("large", ["input", "output"])
def test_a_call_reports_its_own_wait_that_gave_up(rt, large):
    """Two threads on one device.  A wait runs out during the large call; the other thread's small calls see the device's error word
    as well and clear it while the large call still copies.  The large call has to report it all the same."""
    lib = rt.lib()
    rt.check(lib.mimir_b200_check_device(None))
    x = np.ones(16 << 20, np.float32)
    a, w = np.ones((4096, 4), np.float32), np.ones((4096, 4), np.float32)
    call = {"input": lambda: rt.eltwise(abi.ELT_RELU, x), "output": lambda: rt.linear_forward(a, w, None, 4096, 4, 4096)}[large]
    small = np.ones(64, np.float32)
    call()
    done = threading.Event()

    def others():
        rt.init(0)
        done.wait(0.02)  # the large call has begun
        while not done.is_set():
            try:
                rt.eltwise(abi.ELT_RELU, small)
            except rt.MimirB200Error as e:
                assert e.status == abi.E_TIMEOUT

    t = threading.Thread(target=others)
    rt.check(lib.mimir_b200_selftest_wait_timeout(90_000_000, None))  # ahead of the calls in the stream; gives up after 90 ms
    t.start()
    try:
        with pytest.raises(rt.MimirB200Error) as e:
            call()
    finally:
        done.set()
        t.join()
    assert e.value.status == abi.E_TIMEOUT
    rt.check(lib.mimir_b200_check_device(None))
    call()


@pytest.mark.parametrize("waits_with", ["its copy in", "its copy out", "copies in flight", "its copy out, and a second call without the ring"])
def test_a_copy_does_not_wait_for_another_call_s_kernels(rt, waits_with):
    """A per-op call stands behind a 90 ms kernel on the default stream.  A model on its own streams copies in, runs and copies out
    meanwhile, whatever the waiting call holds of the page-locked ring: all of it, for a copy in larger than the ring or for a copy
    out, or the slots of a copy in that it has left behind (its result is small and page-locked: inside a small copy to pageable memory
    the driver itself makes other threads' copies wait)."""
    import torch

    from mimir_framework_b200.abi import make_desc

    lib = rt.lib()
    rt.check(lib.mimir_b200_check_device(None))
    n = 1 << 20
    x = np.random.default_rng(0).standard_normal(n).astype(np.float32)
    m = rt.GraphModel([make_desc("r", "ReLU", inputs=["x"], output="x")])
    m.plan({"x": (n, False)}, 1)
    big = np.ones((48 if waits_with == "its copy in" else 4) << 18, np.float32)
    mean = torch.empty(1).pin_memory()
    pool = lambda: rt.check(lib.mimir_b200_global_avgpool(big.ctypes.data, mean.data_ptr(), 1, 1, 1024, 1024))
    waiting = pool if waits_with == "copies in flight" else lambda: rt.eltwise(abi.ELT_RELU, big)
    for _ in range(3):
        m.forward({"x": (x, False)}, 1, n)
        waiting()
    done = threading.Event()

    def blocked():
        rt.init(0)
        try:
            waiting()
        except rt.MimirB200Error as e:
            assert e.status == abi.E_TIMEOUT  # (the 90 ms are a wait that gives up)
        done.set()

    ts = [threading.Thread(target=blocked) for _ in range(2 if "second" in waits_with else 1)]
    rt.check(lib.mimir_b200_selftest_wait_timeout(90_000_000, None))
    for t in ts:
        t.start()
    time.sleep(0.02)
    got = m.forward({"x": (x, False)}, 1, n)
    overtook = not done.is_set()
    for t in ts:
        t.join()
    lib.mimir_b200_check_device(None)
    m.close()
    assert np.array_equal(got.ravel(), np.maximum(x, 0))
    assert overtook


@pytest.mark.parametrize("n", [100, 16 << 10, 1 << 20, (9 << 20) + 3])
@pytest.mark.parametrize("inject", [0, 1, 2, 3])
def test_copies_without_page_locked_memory_or_threads(rt, inject, n):
    """No room for the ring, or no more threads: the copy is done all the same, and nothing is thrown through the C interface.  With the
    ring both copies of a call take it, although the copy out finds slots in flight on the copy-in stream."""
    import ctypes

    src, dst, staged = np.random.default_rng(n).standard_normal(n).astype(np.float32), np.zeros(n, np.float32), ctypes.c_int(-1)
    rt.check(rt.lib().mimir_b200_selftest_host_copy(inject, src.ctypes.data, dst.ctypes.data, n, ctypes.addressof(staged)))
    assert np.array_equal(src, dst)
    assert staged.value == (0 if inject & 1 or n < 16 << 10 else 2)
