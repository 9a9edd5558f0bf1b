"""Values that belong to a GPU: every device is asked for its own, and an answer that failed is not kept."""
import ctypes

from hcomm_b200 import _lib


def ask(*calls):
    n = len(calls)
    devices = (ctypes.c_int * n)(*[d for d, _ in calls])
    answers = (ctypes.c_int * n)(*[a for _, a in calls])
    values = (ctypes.c_int * n)()
    asked = _lib.load().HcommToolPerDevice(n, devices, answers, values)
    return asked, list(values)


def test_each_device_has_its_own_value():
    assert ask((0, 296), (1, 264), (0, 1), (1, 1), (63, 7), (63, 8)) == (3, [296, 264, 296, 264, 7, 7])


def test_a_failed_query_is_repeated():
    assert ask((0, 0), (0, -1), (0, 296), (0, 5)) == (3, [0, -1, 296, 296])


def test_devices_beyond_the_table_are_asked_every_time():
    assert ask((64, 5), (64, 6), (-1, 7)) == (3, [5, 6, 7])
