"""The bytes object that a recovery fills in place (no copy of the result)."""
import ctypes

import pytest


@pytest.mark.parametrize("n", [2, 492, 4096, 1 << 20])
def test_filled_bytes_are_ordinary_bytes(pkg, n):
    out = pkg._unset_bytes(n)
    other = pkg._unset_bytes(n)
    assert type(out) is bytes and len(out) == n and out is not other
    want = bytes(i * 7 & 255 for i in range(n))
    # as a C call with a char* argument fills it
    ctypes.memmove(ctypes.cast(ctypes.c_char_p(out), ctypes.c_void_p), want, n)
    ctypes.memset(ctypes.cast(ctypes.c_char_p(other), ctypes.c_void_p), 0, n)
    assert out == want and hash(out) == hash(want) and {want: 1}[out] == 1
    assert out[:n - 1] == want[:-1] and other == bytes(n)
