"""lst_batch_get_output through its pinned staging (up to 1 MiB) and past it, against
lst_batch_get_output_static, which has no such staging; and by more threads at a
time than the event setup has staging buffers."""
import ctypes
import threading

import numpy as np
import pytest

from tracklooper_b200 import gen, lst

pytestmark = pytest.mark.gpu

FILL = (0xABABABAB, 0xABABABAB, -0x55, -0x55)


def call(fn, s, count, tc_capacity, hits_capacity):
    arrays = [np.full(n, v, dt) for n, v, dt in zip((hits_capacity, tc_capacity, tc_capacity, tc_capacity), FILL,
                                                    (np.uint32, np.uint32, np.int32, np.int16))]
    tco, hco = np.zeros(count + 1, np.uint64), np.zeros(count + 1, np.uint64)
    a, b, c, d = (x.ctypes.data for x in arrays)
    out = lst.Output(a, hits_capacity, b, c, d, tc_capacity, tco.ctypes.data, hco.ctypes.data)
    fn.argtypes, fn.restype = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.POINTER(lst.Output)], ctypes.c_int
    rc = fn(s.handle, 0, count, ctypes.byref(out))
    return rc, arrays, tco, hco


def output_bytes(tco, hco):
    return 4 * int(hco[-1]) + 10 * int(tco[-1])


# (events, slots of the set, whether the output fits the staging)
CASES = [([(1, 80, 0.0)], 1, True), ([(2, 81, 200.0)], 1, True), ([(2, 920, 400.0)], 1, True),
         ([(2, 920, 400.0)], 2, True), ([(2, 82, 200.0)] * 5, 5, True), ([(2, 83, 200.0)] * 8, 8, False)]


@pytest.fixture(scope="module")
def es():
    e = lst.ES(device=0)
    yield e
    e.close()


@pytest.mark.parametrize("events,slots,fits", CASES)
def test_either_way_gives_the_output(es, events, slots, fits):
    inputs = [gen.generate_event(*e) for e in events]
    n = len(inputs)
    s = lst.EventSet(es, slots, max(i.n_hits for i in inputs) + 1024)
    try:
        s.upload_packed(0, *lst.pack_events(inputs))
        s.run(0, n)
        lib = lst.library()
        rc, want, tco, hco = call(lib.lst_batch_get_output_static, s, n, 31000 * n, 31000 * 14 * n)
        assert rc == 0 and tco[-1] > 0
        assert (output_bytes(tco, hco) < (1 << 20) - 1024) == fits
        for _ in range(2):
            rc, got, t, h = call(lib.lst_batch_get_output, s, n, 31000 * n, 31000 * 14 * n)
            assert rc == 0 and np.array_equal(t, tco) and np.array_equal(h, hco)
            for a, b in zip(got, want):
                assert np.array_equal(a, b)
    finally:
        s.close()


@pytest.mark.parametrize("events,slots,fits", CASES)
@pytest.mark.parametrize("tc_short,hits_short", [(1, 0), (0, 1), (1 << 20, 1 << 20)])
def test_too_small_arrays_stay_as_they_were(es, events, slots, fits, tc_short, hits_short):
    """Refused, with the offsets filled and nothing else written."""
    inputs = [gen.generate_event(*e) for e in events]
    n = len(inputs)
    s = lst.EventSet(es, slots, max(i.n_hits for i in inputs) + 1024)
    try:
        s.upload_packed(0, *lst.pack_events(inputs))
        s.run(0, n)
        fn = lst.library().lst_batch_get_output
        rc, _, tco, hco = call(fn, s, n, 31000 * n, 31000 * 14 * n)
        assert rc == 0
        rc, got, t, h = call(fn, s, n, max(int(tco[-1]) - tc_short, 0), max(int(hco[-1]) - hits_short, 0))
        assert rc == -1 and b"capacity too small" in lst.library().lst_last_error()
        assert np.array_equal(t, tco) and np.array_equal(h, hco)
        for a, v in zip(got, FILL):
            assert (a == a.dtype.type(v)).all()
    finally:
        s.close()


def test_more_threads_than_buffers(es):
    """Each thread with a set of its own, one event after the other."""
    n, rounds = 12, 8
    inputs = [gen.generate_event(*((3, 90 + i, 20.0) if i % 3 else (2, 90 + i, 200.0))) for i in range(n)]
    sets = [lst.EventSet(es, 1, max(i.n_hits for i in inputs) + 1024) for _ in range(n)]
    fn = lst.library().lst_batch_get_output
    try:
        want, got, gate = [], [[] for _ in range(n)], threading.Barrier(n)
        for inp in inputs:
            sets[0].upload_packed(0, *lst.pack_events([inp]))
            sets[0].run(0, 1)
            want.append(call(fn, sets[0], 1, 31000, 31000 * 14))

        def work(i):
            for k in range(rounds):
                sets[i].upload_packed(0, *lst.pack_events([inputs[(i + k) % n]]))
                gate.wait(60)
                sets[i].run(0, 1)
                got[i].append(call(fn, sets[i], 1, 31000, 31000 * 14))

        threads = [threading.Thread(target=work, args=(i,)) for i in range(n)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for i in range(n):
            assert len(got[i]) == rounds
            for k, (rc, arrays, tco, hco) in enumerate(got[i]):
                w = want[(i + k) % n]
                assert rc == 0 and np.array_equal(tco, w[2]) and np.array_equal(hco, w[3])
                for a, b in zip(arrays, w[1]):
                    assert np.array_equal(a, b)
    finally:
        for s in sets:
            s.close()
