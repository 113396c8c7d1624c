"""The generated calls of C functions: every argument arrives by the function's prototype, as through
ctypes, and wrong ones are refused."""

import ctypes

import numpy as np
import pytest

from distengine_b200.kernels import bindings, build, library

TYPES = {"P": ctypes.c_void_p, "I": ctypes.c_int, "L": ctypes.c_longlong, "F": ctypes.c_float}


def _bound(tmp_path, sig, monkeypatch):
    """(call, list of the argument tuples that arrived) of a function with this signature."""
    monkeypatch.setattr(build, "_build_dir", lambda: str(tmp_path))
    arrived = []

    def body(*args):
        arrived.append(args)
        return -7
    fn = ctypes.CFUNCTYPE(ctypes.c_int, *(TYPES[c] for c in sig))(body)
    module = bindings.load(build.build_bindings(bindings.source(["", sig])))
    return module.bind(1, ctypes.cast(fn, ctypes.c_void_p).value), arrived, fn


def test_arguments_arrive(tmp_path, monkeypatch):
    # more of each kind than there are registers for
    sig = "IPFLPIFFIPLFIIFFPFFIFPLIIPFIIPPFL"
    call, arrived, _keep = _bound(tmp_path, sig, monkeypatch)
    values = {"P": lambda i: 0x7f0000000000 + 16 * i, "I": lambda i: -i, "L": lambda i: -(1 << 40) - i,
              "F": lambda i: i + 0.25}
    args = [values[c](i) for i, c in enumerate(sig)]
    assert call(*args) == -7
    assert arrived == [tuple(args)]
    special = list(args)
    for i, c in enumerate(sig):
        special[i] = None if c == "P" else 3 if c == "F" else np.int64(i) if c == "I" else True
    assert call(*special) == -7
    assert arrived[1] == tuple(None if c == "P" else 3.0 if c == "F" else i if c == "I" else 1
                               for i, c in enumerate(sig))
    for wrong in (args[:-1], args + [0], [1.5] + args[1:], [None] + args[1:], ["1"] + args[1:],
                  args[:1] + [2.0] + args[2:], args[:2] + [None] + args[3:]):
        with pytest.raises(TypeError):
            call(*wrong)
    assert len(arrived) == 2


def test_kernel_functions_through_both():
    """A function of every library that needs no GPU, called both ways."""
    lib = library.load("gemm_f32")
    plain = lib._cdll.de_gemm_f32_form
    plain.argtypes, plain.restype = [ctypes.c_int] * 4, ctypes.c_int
    for sizes in ((1, 130, 260, 1), (8, 131, 600, 1), (1000, 2051, 772, 1), (40, 70, 51, 0)):
        assert lib.de_gemm_f32_form(*sizes) == plain(*sizes)
    with pytest.raises(AttributeError):
        lib.no_such_function


def test_without_the_interpreters_headers(tmp_path, monkeypatch):
    """No Python.h: the extension cannot be made, and the functions come through ctypes."""
    want = library.load("gemm_f32").de_gemm_f32_form(8, 131, 600, 1)
    make, folder = build.build_bindings, build._build_dir

    def make_anew(text):                     # (not the one that was made before)
        monkeypatch.setattr(build, "_build_dir", lambda: str(tmp_path))
        try:
            return make(text)
        finally:
            monkeypatch.setattr(build, "_build_dir", folder)
    monkeypatch.setattr(bindings, "include_dir", lambda: str(tmp_path))
    monkeypatch.setattr(build, "build_bindings", make_anew)
    monkeypatch.setattr(library, "_bind", None)
    monkeypatch.setattr(library, "_loaded", {})
    lib = library.load("gemm_f32")
    assert lib.de_gemm_f32_form(8, 131, 600, 1) == want
    with pytest.raises(ctypes.ArgumentError):
        lib.de_gemm_f32_form(8, 131, 600, 1.5)
    monkeypatch.setattr(build, "build_many", lambda requests, verbose: ["kernels"])
    assert build.build_all(verbose=False) == ["kernels"]
