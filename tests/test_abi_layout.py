"""Structures of the C ABI keep the layout that callers are compiled with."""
import ctypes

import perft_gpu_2026_b200 as pg


def test_statistics_write_no_more_than_their_structure():
    """pb_last_stats writes 192 bytes; later figures have entry points of their own."""
    assert ctypes.sizeof(pg.Stats) == 2 * 8 + 3 * 8 + 2 * 4 + 16 * 8 + 2 * 8 == 192
    eng = pg.Engine(device=-1)
    buf = (ctypes.c_uint8 * 512)(*([0xA5] * 512))
    fn = ctypes.CDLL(pg.LIB_PATH).pb_last_stats
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    assert fn(eng.handle, ctypes.addressof(buf)) == pg.PB_OK
    assert bytes(buf[192:]) == b"\xa5" * 320
    eng.close()
