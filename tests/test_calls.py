"""Calls of the C ABI through the extension module: every argument arrives, whatever the order of integers and floats and however many there
are, results keep their sign and width, and what it cannot pass on goes to the ctypes function."""
import ctypes
import importlib.machinery
import importlib.util
import pathlib
import platform
import sysconfig

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


@pytest.fixture
def builder(pkg, tmp_path, monkeypatch):
    """``build.py`` with the module's place in a folder of the test."""
    spec = importlib.util.spec_from_file_location("b2kv_build_for_test", pathlib.Path(pkg.__file__).parent / "build.py")
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    monkeypatch.setattr(module, "CALLS", tmp_path / module.CALLS.name)
    return module


def test_the_module_is_of_one_interpreter(pkg, builder):
    assert builder.CALLS.name == pkg._native.CALLS_PATH.name == "b2kv_calls" + sysconfig.get_config_var("EXT_SUFFIX")


@pytest.mark.parametrize("what", ["no compiler", "a compiler that fails", "another machine", "no headers"])
def test_the_library_is_built_where_the_module_cannot_be(builder, tmp_path, monkeypatch, capfd, what):
    if what == "another machine":
        monkeypatch.setattr(platform, "machine", lambda: "aarch64")
    if what == "no headers":
        monkeypatch.setattr(sysconfig, "get_paths", lambda: {"include": str(tmp_path)})
    monkeypatch.setenv("CC", str(tmp_path / "cc") if what == "no compiler" else "false")
    monkeypatch.setattr(builder, "up_to_date", lambda out: True)
    builder.CALLS.write_bytes(b"of an older source")
    assert builder.build_calls(force=True) is None and not builder.CALLS.exists()
    assert "ctypes" in capfd.readouterr().err
    assert builder.build() == builder.OUT


def test_calls_without_the_module(pkg, monkeypatch):
    """The same entry points, structures and refusals through ctypes alone."""
    native = pkg._native

    def refused(self, module):
        raise ImportError("of another machine")

    monkeypatch.setattr(importlib.machinery.ExtensionFileLoader, "exec_module", refused)
    monkeypatch.setattr(importlib.machinery.ExtensionFileLoader, "create_module", lambda self, spec: None)
    spec = importlib.util.spec_from_file_location("b2kv_native_for_test", native.__file__)
    other = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(other)
    assert other.calls is None and other.lib.b2kv_version() == native.lib.b2kv_version()
    args = [1 << 8, 2 << 8, 0, 0, 0, 1024, 0, 4096, 0, 0, [(3 << 8, 4096, 0, 4096, 0)], 700, 1024, 4096, 1, 0, 0, 0, 0.0]
    sizes = [n.lib.b2kv_linear_workspace_bytes(n.linear_args(*args)) for n in (native, other)]
    assert sizes[0] == sizes[1] > 0
    args[0] = 0  # no input: refused before anything is launched
    for n in (native, other):
        assert n.lib.b2kv_linear_ws(n.linear_args(*args), n.linear_options(0, 0, 0), None, 0, None, None) == -1
        with pytest.raises(IndexError):
            n.linear_args(*args[:10], args[10] * (n.MAX_SEGMENTS + 1), *args[11:])
    assert native.lib.b2kv_strerror(-1) == other.lib.b2kv_strerror(-1)
