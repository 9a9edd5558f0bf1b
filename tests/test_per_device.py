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


def test_what_a_gemm_finds_is_kept_only_if_every_query_was_answered():
    def kept(*answers):
        caps = (ctypes.c_int * 4)(*[-7] * 4)
        return bool(_lib.load().HcommToolGemmClusterCaps((ctypes.c_int * 4)(*answers), caps)), list(caps)
    assert kept(74, 33, 22, 15) == (True, [74, 33, 22, 15])
    assert kept(74, 33, 0, 15) == (True, [74, 33, 0, 15])           # a device that holds no cluster of three pairs
    for i in range(4):
        answers = [74, 33, 22, 15]
        answers[i] = -1
        assert kept(*answers) == (False, [max(0, n) for n in answers])
