"""The payload's read to host memory (dl_session_payload_build / _read): below one piece, and shared
by several cores in pieces with a ragged end, against the host writer's bytes; and what read refuses."""
import ctypes as C
import zlib

import pytest

import dynlight_gb300 as dl
from dynlight_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,density", [(17, 2.0), (65, 4.0), (113, 4.0)])
def test_read_payload_equals_the_host_writer(grid, density):
    inp, opts = scenes.outdoor(grid=grid, chunks=2, boxes=5, point_lights=2, density=density, sun_samples=16,
                               sky_samples=16, bounce_samples=8)
    s = dl.Session(inp, opts)
    try:
        s.run()
        payload, crc = s.encode_payload()
        out = C.POINTER(dl._abi.DlBakedScene)()
        assert s.lib.dl_session_result(s.handle, C.byref(out)) == 0
        try:
            want, want_crc = dl.encode_payload(out.contents)
        finally:
            s.lib.dl_baked_scene_free(out)
        assert payload == want and crc == want_crc == zlib.crc32(want)
        data, length, crc32 = C.POINTER(C.c_uint8)(), C.c_uint64(), C.c_uint32()
        assert s.lib.dl_session_encode_payload(s.handle, C.byref(data), C.byref(length), C.byref(crc32)) == 0
        try:
            assert C.string_at(data, length.value) == want and crc32.value == want_crc
        finally:
            s.lib.dl_free(data)
        # a wrong length, and a payload that a new run has ended
        buffer = C.create_string_buffer(16)
        assert s.lib.dl_session_payload_read(s.handle, C.cast(buffer, C.c_void_p), 16) == 21
        s.run()
        assert s.lib.dl_session_payload_read(s.handle, C.cast(buffer, C.c_void_p), len(want)) == 21
        assert b"no built payload" in s.lib.dl_last_error()
    finally:
        s.close()
