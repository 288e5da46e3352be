"""Headers whose extents multiply past 2^64: the product wraps round to a number of
values that any buffer holds.  Refused on the host, before anything else is looked at."""
import ctypes
import struct

import pytest

import faz_gb300 as F
from faz_gb300.config import FazConfigStruct

import oracle.oracle as O


@pytest.fixture(scope="module")
def lib():
    from faz_gb300 import build as B
    B.build()
    return F.library()


WRAP = [(1 << 33, 1 << 31), (1 << 32, 1 << 32), (1 << 32, 1 << 32, 8), (3, 0xaaaaaaaaaaaaaaab), (1 << 22, 1 << 22, 1 << 20),
        (1 << 16, 1 << 16, 1 << 16, 1 << 16), ((1 << 64) - 1, (1 << 64) - 1)]


@pytest.mark.parametrize("dims", WRAP)
def test_payload(lib, dims):
    payload = struct.pack(f"<{len(dims)}Q", *dims) + struct.pack("<IiiddQiBiQiiBdiQ", 32, 1, 0, -1.0, -1.0, 0, 0, 0, 0, 0,
                                                                  0, 0, 2, 0.1, 32768, 0) + bytes(64)
    tm = F.api.FazTimings()
    rc = lib.faz_decompress_payload_device(len(dims), F.config.FAZ_FLOAT, payload, len(payload), ctypes.c_void_p(16),
                                           1 << 40, None, ctypes.byref(tm))
    assert rc == -4


@pytest.mark.parametrize("dims", WRAP)
def test_trailer(lib, dims):
    c = F.Config(*[4] * len(dims))
    num = 1
    for d in dims:
        num = num * d % (1 << 64)
    s = FazConfigStruct()
    good = O._config_bytes(c)
    at = 1 + 8 * len(dims)
    body = good[:1] + struct.pack(f"<{len(dims)}Q", *dims) + struct.pack("<Q", num) + good[at + 8:]
    stream = bytes(16) + body + struct.pack("<i", len(body))
    assert lib.faz_stream_info(stream, len(stream), ctypes.byref(s)) == -4
    ok = bytes(16) + good + struct.pack("<i", len(good))
    assert lib.faz_stream_info(ok, len(ok), ctypes.byref(s)) == 0


@pytest.mark.parametrize("dims", [d for d in WRAP if all(d)])
def test_configuration(lib, dims):
    s = F.Config(*[4] * len(dims)).to_struct()
    num = 1
    for i, d in enumerate(dims):
        s.dims[i] = d
        num = num * d % (1 << 64)
    s.num = num
    out, size, tm = ctypes.c_void_p(), ctypes.c_size_t(), F.api.FazTimings()
    rc = lib.faz_compress_device(ctypes.byref(s), F.config.FAZ_FLOAT, ctypes.c_void_p(16), None, ctypes.byref(out),
                                 ctypes.byref(size), ctypes.byref(tm))
    assert rc == -1
