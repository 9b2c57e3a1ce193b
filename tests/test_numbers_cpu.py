"""The numbers that tag items' flags and entries of the table of explored states
(td_core.cuh): no launch takes one that an earlier launch, or its complement, may
have left behind, without the tags being cleared first; and requests keep their
64-bit number where an item holds the low half."""
import ctypes as C

import pytest

MAX = 0x7FFFFFFF


@pytest.mark.parametrize("last", [0, 1, 1000, MAX - 33, MAX - 32, MAX - 31, MAX - 2, MAX - 1, MAX])
@pytest.mark.parametrize("epochs", [1, 2, 32])
def test_epochs(emu, last, epochs):
    emu.td_emu_next_epoch.restype = C.c_uint32
    again = C.c_int(-1)
    e = emu.td_emu_next_epoch(C.c_uint32(last), C.c_uint32(epochs), C.byref(again))
    taken = range(e - epochs + 1, e + 1)
    assert taken[0] >= 1 and taken[-1] <= MAX  # none is zero, and none the complement of another
    if again.value:
        assert taken[0] == 1 and last + epochs > MAX
    else:
        assert taken[0] == last + 1


@pytest.mark.parametrize("number", [0, 1, 2 ** 32 - 1, 2 ** 32, 2 ** 32 + 5, 2 ** 40 + 2 ** 32 - 1])
@pytest.mark.parametrize("later", [1, 2, 65536, 2 ** 32 - 1])
def test_request_numbers(emu, number, later):
    emu.td_emu_request_number.restype = C.c_uint64
    assert emu.td_emu_request_number(C.c_uint64(number + later), C.c_uint32(number & 0xFFFFFFFF)) == number
