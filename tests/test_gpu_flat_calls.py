"""Calls over flat share vectors beside other work: on a stream of the caller's
they start after party 0's stream, they are refused under a capture, and an
empty vector is no error."""
from __future__ import annotations

import numpy as np
import pytest

import irisb200
import workload as W

pytestmark = pytest.mark.gpu


# elements on both sides of the few-word kernel's limit (888 x 1,024)
@pytest.mark.parametrize("entries", [1024, 8192])
def test_flat_call_on_another_stream_follows_the_dots(dm, entries):
    K, rows = 12800, 768
    rng = np.random.default_rng(entries)
    e = irisb200.ShareDB(0, dm, entries, rows, K, W.SEEDS[0])
    e.alloc_db(entries)
    e.fill_random(4, entries)
    c = irisb200.Circuits(dm, W.SEEDS)
    n = rows * entries
    opened = irisb200.DeviceBuffer(dm, n // 8)
    ptr, stride = e.result_view()
    assert stride == rows

    def compare():
        c.compare_threshold_masked_many([ptr] * 3, [ptr] * 3, n, 16384, opened=opened, stream=dm.stream(2))
        dm.synchronize()
        return opened.download(np.uint8, n // 8)
    got = []
    for k in range(3):
        e.query_upload(rng.integers(0, 1 << 16, (rows, K), dtype=np.uint16))
        dm.synchronize()
        for _ in range(150):
            e.dot(0, 32, 1)  # a few blocks each: the rest of the GPU is free meanwhile
        e.dot(0, entries, 1)
        got.append(compare())
        assert np.array_equal(got[-1], compare())  # with the dots done
        lifted = irisb200.DeviceBuffer(dm, 64)
        c.lift_mpc([ptr] * 3, 0, [lifted.ptr] * 3)
        lifted.free()
    assert not np.array_equal(got[0], got[1]) and not np.array_equal(got[1], got[2])
    opened.free()
    c.close()
    e.close()


def test_flat_calls_are_refused_under_capture(dm):
    c = irisb200.Circuits(dm, W.SEEDS)
    buf = irisb200.DeviceBuffer(dm, 1 << 16)
    p = [buf.ptr] * 3
    for call in (lambda: c.compare_threshold_masked_many(p, p, 4096, 16384),
                 lambda: c.compare_threshold_masked_many_with_or_tree(p, p, 4096, 16384),
                 lambda: c.extract_msb_of_code(p, 4096), lambda: c.or_reduce(p, 4096),
                 lambda: c.lift_mpc(p, 64, p)):
        refused = []

        def body():
            with pytest.raises(irisb200.IrisError):
                call()
            refused.append(True)
        irisb200.Graph.capture(dm, body).close()
        assert refused
    dm.synchronize()
    c.compare_threshold_masked_many_with_or_tree(p, p, 4096, 16384)
    buf.free()
    c.close()
