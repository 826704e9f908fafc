"""The host's rules on which kernel a call takes: no GPU needed, only the library."""
from ctypes import c_int, c_int64, c_void_p

import pytest


@pytest.mark.parametrize("n, k, ldx, ldw, x, w, takes", [
    (2048, 2048, 2048, 2048, 0x1000, 0x2000, True), (2048, 2048, 4096, 2052, 0x1000, 0x2000, True), (2048, 2048, 0, 2048, 0x1000, 0x2000, True),
    (2048, 2048, 2048, 0, 0x1000, 0x2000, False),                  # one row for all features (an expanded weight)
    (2048, 2048, 2048, 1024, 0x1000, 0x2000, False),               # rows that overlap
    (2047, 2048, 2048, 2048, 0x1000, 0x2000, False),               # few weights
    (2048, 2080, 2080, 2080, 0x1000, 0x2000, False), (2048, 2048, 2049, 2048, 0x1000, 0x2000, False), (2048, 2048, 2048, 2048, 0x1004, 0x2000, False)])
def test_which_32_bit_products_run_on_tensor_cores(n, k, ldx, ldw, x, w, takes):
    from torchinferno_b200.kernels.library import load_library
    assert bool(load_library().tib_gemm_f32_tcgen05_takes(c_void_p(x), c_void_p(w), c_int(n), c_int(k), c_int64(ldx), c_int64(ldw))) == takes
