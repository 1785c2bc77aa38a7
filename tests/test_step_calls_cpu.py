"""What the Python calls of every step keep between calls (no GPU)."""
import ctypes

import pytest


def _backend():
    from knp_gb300 import GB300Backend

    b = GB300Backend.__new__(GB300Backend)  # no device
    b._uids = {}
    return b


def test_uids_are_kept_by_value():
    b = _backend()
    u = bytes(range(16))
    assert bytes(b._uid(u).bytes) == u
    assert b._uid(bytes(range(16))) is b._uid(u)
    for bad in (b"short", bytes(17)):
        with pytest.raises(ValueError):
            b._uid(bad)


def test_a_uid_in_a_buffer_is_read_at_every_call():
    b = _backend()
    buf = (ctypes.c_uint8 * 16)(*range(16))
    assert bytes(b._uid(buf).bytes) == bytes(range(16))
    buf[0] = 200
    assert bytes(b._uid(buf).bytes)[0] == 200


def test_gemm_errors_are_checked_without_a_gpu():
    from knp_gb300 import bptt

    bptt.check_gemm_errors("cpu")  # nothing ran there
