"""How the backward of the modulated norms cuts an image's tokens."""
import ctypes

import pytest

from dew_b200.ops import library as L


@pytest.mark.skipif(not L.exists(), reason="the library is not built")
def test_every_block_has_a_row_for_each_of_its_warps():
    slab = lambda B, n: L.load().dewb_ada_slab(ctypes.c_int(B), ctypes.c_int(n))
    for B in (1, 2, 3, 8, 64, 512):
        for n in (1, 7, 8, 9, 15, 16, 17, 129, 257, 300, 1000, 4096):
            s = slab(B, n)
            assert min(8, n) <= s <= n
            # about two blocks an SM: halved no further than that needs
            assert s == n or B * -(-n // (2 * s)) < 2 * 148
