"""Large results into fresh, unaligned and reused host memory: the same bytes as in small pieces,
and nothing written beside them."""
import ctypes as C
import mmap
import threading

import numpy as np
import pytest

from eig_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1, 65535])
@pytest.mark.parametrize("nsnp", [83055, 83056, 130001])  # 101 bytes each: around 8 MiB, and above
def test_encode_into_unaligned_memory(gpu, offset, nsnp):
    r = np.random.default_rng(nsnp)
    n = 401
    rec = r.integers(0, 256, (nsnp, 101), dtype=np.uint8)
    gpu.load_genotypes(rec, n)
    snps = np.arange(nsnp, dtype=np.int64)
    want = np.concatenate([gpu.encode_records(native.GP_OUT_PACKEDPED, s, nsamples=n)
                           for s in np.array_split(snps, 3)])  # each below the threshold
    size = nsnp * 101
    buf = np.full(offset + size + 65536, 7, np.uint8) if offset else np.empty(size + 65536, np.uint8)
    for _ in range(2):
        rc = gpu.lib.gp_encode_records(gpu.h, native.GP_OUT_PACKEDPED, None, n,
                                       snps.ctypes.data_as(native.i64p), None, nsnp,
                                       C.c_void_p(buf.ctypes.data + offset), 0)
        assert rc == native.GP_OK
        assert np.array_equal(buf[offset:offset + size], want.reshape(-1))
    if offset:
        assert np.all(buf[:offset] == 7) and np.all(buf[offset + size:] == 7)


def encode(gpu, snps, buf, offset, n):
    assert gpu.lib.gp_encode_records(gpu.h, native.GP_OUT_PACKEDPED, None, n,
                                     snps.ctypes.data_as(native.i64p), None, len(snps),
                                     C.c_void_p(buf.ctypes.data + offset), 0) == native.GP_OK


@pytest.mark.parametrize("offset", [0, 65535])
@pytest.mark.parametrize("nsnp", [166111, 166112, 330000])  # 101 bytes each: around 16 MiB, and above
def test_pages_there_or_not(gpu, offset, nsnp):
    """fresh pages, pages of which some are there, and pages that are all there: the same bytes; for
    the last no thread is started (each new thread takes a new id, a call with threads starts four)"""
    n = 401
    gpu.load_genotypes(np.random.default_rng(nsnp).integers(0, 256, (nsnp, 101), dtype=np.uint8), n)
    snps = np.arange(nsnp, dtype=np.int64)
    size = nsnp * 101
    want = np.concatenate([gpu.encode_records(native.GP_OUT_PACKEDPED, s, nsamples=n)
                           for s in np.array_split(snps, 5)]).reshape(-1)

    def new_id():
        ids = []
        t = threading.Thread(target=lambda: ids.append(threading.get_native_id()))
        t.start()
        t.join()
        return ids[0]

    for there in (0, size // 2, size):
        m = mmap.mmap(-1, size + 131072)
        buf = np.frombuffer(m, np.uint8)
        buf[:offset + there] = 7
        a = new_id()
        for _ in range(20 if there == size else 1):
            encode(gpu, snps, buf, offset, n)
        assert there < size or new_id() - a < 40
        assert np.array_equal(buf[offset:offset + size], want)
        assert np.all(buf[:offset] == (7 if offset else 0)) and not buf[offset + size:].any()
