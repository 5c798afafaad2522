"""The payload's bytes object is filled through function prototypes of the package's own: other modules
may give ctypes.pythonapi's functions, which are one object each for the whole process, other types."""
import ctypes as C
import os
import subprocess
import sys
import types

import pytest

import dynlight_gb300 as dl

HERE = os.path.dirname(os.path.abspath(__file__))
CONTENT = bytes(range(256)) * 9 + b"end"


def fake_library(content):
    """A payload of `content`, written only to an address (a prototype gone wrong hands out another object)."""
    def build(handle, length, crc):
        C.cast(length, C.POINTER(C.c_uint64))[0] = len(content)
        C.cast(crc, C.POINTER(C.c_uint32))[0] = 7
        return 0

    def read(handle, address, length):
        assert isinstance(address, int) and length == len(content)
        C.memmove(address, content, length)
        return 0

    return types.SimpleNamespace(dl_session_payload_build=build, dl_session_payload_read=read,
                                 dl_session_destroy=lambda handle: None)


@pytest.mark.parametrize("restype", [C.c_char_p, C.c_int, C.py_object, None])
def test_shared_prototypes_do_not_reach_the_payload(restype):
    shared = [C.pythonapi.PyBytes_AsString, C.pythonapi.PyBytes_FromStringAndSize]
    kept = [(f.restype, f.argtypes) for f in shared]
    session = object.__new__(dl.Session)
    session.lib, session.handle = fake_library(CONTENT), None
    try:
        for f in shared:
            f.restype, f.argtypes = restype, [C.py_object]
        payload, crc = session.encode_payload()
    finally:
        for f, (r, a) in zip(shared, kept):
            f.restype, f.argtypes = r, a
    assert payload == CONTENT and crc == 7


def test_import_leaves_the_shared_prototypes_alone():
    code = ("import ctypes as C, sys; sys.path.insert(0, sys.argv[1]); f = C.pythonapi.PyBytes_AsString; "
            "g = C.pythonapi.PyBytes_FromStringAndSize; f.restype = g.restype = C.c_char_p; f.argtypes = g.argtypes = "
            "[C.c_void_p]; import conftest; print(f.restype is C.c_char_p and g.restype is C.c_char_p and "
            "f.argtypes == g.argtypes == [C.c_void_p])")
    out = subprocess.run([sys.executable, "-c", code, HERE], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "True", out.stdout + out.stderr
