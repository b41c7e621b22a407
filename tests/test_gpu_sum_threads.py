"""Threads that launch, each over its own device manager, while another takes
the memory of their engines' sums and gives it back."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import irisb200
import workload as W

pytestmark = pytest.mark.gpu


def test_launches_beside_a_thread_that_takes_sums():
    K, n_q, n_db, n_threads = 6400, 40, 8192, 3
    start, stop = threading.Barrier(n_threads + 1), threading.Event()
    failed, ran = [], []

    def work(k):
        try:
            rng = np.random.default_rng(k)
            dm = irisb200.DeviceManager(0)
            e = irisb200.ShareDB(0, dm, n_db, n_q * 32, K, W.SEEDS[0])
            base = rng.integers(0, 1 << 16, (n_q, K), dtype=np.uint16)
            slots = [(j, 0, 31, j) for j in range(n_q)]

            def load():
                e.alloc_db(n_db)
                e.fill_random(k, n_db)
                e.query_upload_slots(base, slots)

            def dots():
                for _ in range(20):
                    e.dot(0, n_db, 1)
                gemm = e.last_gemm()[0]
                return gemm, e.fetch_results(n_db)
            load()
            gemm, want = dots()
            assert gemm == "quad"
            start.wait(60)
            while not stop.is_set():
                gemm, got = dots()
                assert np.array_equal(got, want)
                ran.append(gemm)
                if not e.has_sums():
                    load()  # takes them again, where there is room
                else:
                    e.query_upload_slots(base, slots)
            e.close()
            dm.close()
        except BaseException as x:  # noqa: BLE001
            failed.append(x)
            start.abort()
    threads = [threading.Thread(target=work, args=(k,)) for k in range(n_threads)]
    for t in threads:
        t.start()
    dm = irisb200.DeviceManager(0)
    try:
        start.wait(120)
        for _ in range(6):
            taken = [irisb200.DeviceBuffer(dm, dm.mem_info()[0] - (8 << 30))]
            while True:  # down to the sums of the threads' engines, and past them
                try:
                    taken.append(irisb200.DeviceBuffer(dm, 1 << 30))
                except irisb200.IrisError:
                    break
            for b in taken:
                b.free()
    finally:
        stop.set()
        for t in threads:
            t.join(120)
        dm.close()
    assert not failed and not any(t.is_alive() for t in threads)
    assert "quad" in ran


def test_sums_give_way_one_engine_at_a_time():
    """An allocation takes no more sums than it needs, and none where all of
    them would not do."""
    dm = irisb200.DeviceManager(0)
    engines = [irisb200.ShareDB(0, dm, 64, 640, 6400, W.SEEDS[0]) for _ in range(3)]
    for e in engines:
        e.alloc_db(40000)  # 640 MB of sums each
    total = dm.mem_info()[1]
    with pytest.raises(irisb200.IrisError):
        irisb200.DeviceBuffer(dm, total)
    assert all(e.has_sums() for e in engines)
    taken = []
    while all(e.has_sums() for e in engines):
        taken.append(irisb200.DeviceBuffer(dm, max(1 << 28, dm.mem_info()[0] - (6 << 30))))
    assert sorted(e.has_sums() for e in engines) == [False, True, True]
    with pytest.raises(irisb200.IrisError):
        irisb200.DeviceBuffer(dm, total // 2)
    assert sorted(e.has_sums() for e in engines) == [False, True, True]
    while sum(e.has_sums() for e in engines) == 2:
        taken.append(irisb200.DeviceBuffer(dm, 1 << 28))
    assert sorted(e.has_sums() for e in engines) == [False, False, True]
    for b in taken:
        b.free()
    for e in engines:
        e.close()
    dm.close()


def test_free_memory_is_what_any_allocator_can_have():
    """mem_info is the device's free memory; the sums count apart, and are given
    back on demand."""
    import torch
    dm = irisb200.DeviceManager(0)
    e = irisb200.ShareDB(0, dm, 64, 640, 6400, W.SEEDS[0])
    e.alloc_db(40000)
    sums = 2 * -(-40000 // 128) * 128 * 8000
    assert e.has_sums() and dm.mem_info() == torch.cuda.mem_get_info(0)
    before, held = dm.mem_info()[0], dm.derived_bytes()
    assert sums <= held < sums * 1.1
    assert dm.derived_bytes(give_back=True) == 0 and not e.has_sums()
    assert dm.mem_info()[0] >= before + sums
    e.close()
    dm.close()
