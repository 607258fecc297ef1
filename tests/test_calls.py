"""Calls of the C ABI through the extension module: every argument arrives, whatever the order of integers and floats and however many there
are, results keep their sign and width, and what it cannot pass on goes to the ctypes function."""
import ctypes

import pytest

KINDS = {"p": ctypes.c_void_p, "i": ctypes.c_int, "l": ctypes.c_int64, "f": ctypes.c_float}


@pytest.fixture(scope="module")
def calls(pkg):
    if pkg._native.calls is None:
        pytest.skip("not built: no headers of this interpreter")
    return pkg._native.calls


def bound(calls, kinds, fn, restype=ctypes.c_int):
    callback = ctypes.CFUNCTYPE(restype, *[KINDS[k] for k in kinds])(fn)
    return calls.bind(ctypes.cast(callback, ctypes.c_void_p).value, kinds, "i" if restype is ctypes.c_int else "z", callback), callback


@pytest.mark.parametrize("kinds", ["", "p", "f", "ipl", "fifi", "pppppiiii", "ppllfpipfliiiiipppp", "plfifffl" + "il" * 10, "i" * 28, "f" + "l" * 27])
def test_every_argument_arrives(calls, kinds):
    seen = []
    call, keep = bound(calls, kinds, lambda *a: seen.append(a) or -len(a))
    args = [1.5 + k if t == "f" else (1 << 40) + k if t in "pl" else -k - 1 for k, t in enumerate(kinds)]
    assert call(*args) == -len(kinds) and seen == [tuple(args)]


def test_widths_null_bytes_and_results(calls):
    seen = []
    call, keep = bound(calls, "pili", lambda *a: seen.append(a) or 7)
    assert call(None, (1 << 32) + 5, -1, True) == 7 and seen[0] == (None, 5, -1, 1)
    text = b"structure"
    call(text, 0, 0, 0)
    assert ctypes.string_at(seen[1][0]) == text
    size, keep2 = bound(calls, "i", lambda a: (1 << 40) + a, ctypes.c_size_t)
    assert size(3) == (1 << 40) + 3


def test_the_rest_goes_to_ctypes(calls):
    seen = []
    call, keep = bound(calls, "pif", lambda *a: seen.append(a) or 0)
    value = ctypes.c_int(5)
    call(ctypes.byref(value), ctypes.c_int(6), 2)
    assert seen[0] == (ctypes.addressof(value), 6, 2.0)
    for bad in ((1, 2), (1, "two", 3.0), (1.5, 2, 3.0)):
        with pytest.raises((TypeError, ctypes.ArgumentError)):
            call(*bad)
    for kinds, result in (("px", "i"), ("p" * 29, "i"), ("fffff", "i"), ("p", "d")):
        with pytest.raises(ValueError):
            calls.bind(0, kinds, result, None)


def test_structures_are_those_of_the_header(pkg):
    """The bytes that a linear layer is called with, read back through the ctypes structure."""
    native = pkg._native
    segments = [(11, 12, 13, 14, 15), (21, 22, 23, 24, 25)]
    a = native.linear_args(1, 2, 3, 4, 5, 6, 7, 8, 9, 10, segments, 31, 32, 33, 34, 35, 1, 2, 0.5)
    if native.calls is not None:
        a = native.LinearArgs.from_buffer_copy(a)
        assert [getattr(a, n) for n, _ in native.LinearArgs._fields_ if n != "seg"] == [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 31, 32, 33, 34, 35, 2, 1, 2, 0.5]
        assert [tuple(getattr(s, n) for n, _ in native.Segment._fields_) for s in a.seg] == segments + [(None, 0, 0, 0, 0)]
        o = native.LinearOptions.from_buffer_copy(native.linear_options(1, 2, 3))
        assert [getattr(o, n) for n, _ in native.LinearOptions._fields_] == [1, 2, 3]
