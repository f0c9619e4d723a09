"""The bytes objects that Context.derive and derive_noalloc hand to the library to fill."""
import ctypes

import pytest

from meikey_b200 import engine


@pytest.mark.parametrize("n", [2**63, 2**64, 32 * 2**59, 32 * 2**60 + 32, -1, -32, -2**63, -2**70, 2.0, "ab", None])
def test_sizes_are_refused_as_by_create_string_buffer(n):
    """2^59 keys are 2^64 bytes, which must not become a buffer of none for the library to write past."""
    with pytest.raises((OverflowError, ValueError, TypeError)) as want:
        ctypes.create_string_buffer(n)
    with pytest.raises(want.type):
        engine._new_bytes(n)


@pytest.mark.parametrize("n", [0, 1, 32, 65536])
def test_sizes_are_exact(n):
    assert len(engine._new_bytes(n)) == n


def test_other_users_of_the_python_api_are_left_alone(monkeypatch):
    """ctypes.pythonapi's functions belong to the whole process: another module may declare
    PyBytes_FromStringAndSize as it likes, and finds what it declared."""
    shared = ctypes.pythonapi.PyBytes_FromStringAndSize
    monkeypatch.setattr(shared, "restype", ctypes.c_void_p)
    monkeypatch.setattr(shared, "argtypes", [ctypes.c_void_p, ctypes.c_size_t])
    got = engine._new_bytes(32)
    assert type(got) is bytes and len(got) == 32
