"""What a search prepares from a pattern before its launch, on the host: the choice
of the words it is looked for by takes microseconds, whatever the pattern."""
import ctypes
import time

import numpy as np
import pytest

from oneline_b200 import _lib

SYMBOL = "_ZN2ol18search_add_patternERNS_10SearchArgsEPKhS3_jPjj"  # (args, host, dev, length, out, max_out)


@pytest.mark.parametrize("length", [12, 64, 250, 4000])
def test_preparing_a_pattern_is_quick(length):
    add = ctypes.CDLL(_lib.LIB_PATH)[SYMBOL]
    add.argtypes = [ctypes.c_void_p, ctypes.c_char_p, ctypes.c_void_p, ctypes.c_uint32, ctypes.c_void_p, ctypes.c_uint32]
    add.restype = None
    pattern = np.random.default_rng(length).integers(97, 123, length, dtype=np.uint8).tobytes()  # no rarest word ends the choice
    best = 1.0
    for _ in range(200):
        args = ctypes.create_string_buffer(1 << 14)  # a zeroed SearchArgs; the device copy is never read here
        t = time.perf_counter()
        add(args, pattern, 4096, length, None, 0)
        best = min(best, time.perf_counter() - t)
    assert best < 8e-6, best  # 20 us for 250 bytes with a library call for every byte of every word
