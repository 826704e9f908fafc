"""What can be said of the kernels without a GPU: the host's rules on which one a call takes, and rules that their sources keep."""
import re
from ctypes import c_int, c_int64, c_void_p
from pathlib import Path

import pytest

import torchinferno_b200

CSRC = Path(torchinferno_b200.__file__).parent / "csrc"


@pytest.mark.parametrize("n, k, ldx, ldw, x, w, takes", [
    (2048, 2048, 2048, 2048, 0x1000, 0x2000, True), (2048, 2048, 4096, 2052, 0x1000, 0x2000, True), (2048, 2048, 0, 2048, 0x1000, 0x2000, True),
    (2048, 2048, 2048, 0, 0x1000, 0x2000, False),                  # one row for all features (an expanded weight)
    (2048, 2048, 2048, 1024, 0x1000, 0x2000, False),               # rows that overlap
    (2047, 2048, 2048, 2048, 0x1000, 0x2000, False),               # few weights
    (2048, 2080, 2080, 2080, 0x1000, 0x2000, False), (2048, 2048, 2049, 2048, 0x1000, 0x2000, False), (2048, 2048, 2048, 2048, 0x1004, 0x2000, False)])
def test_which_32_bit_products_run_on_tensor_cores(n, k, ldx, ldw, x, w, takes):
    from torchinferno_b200.kernels.library import load_library
    assert bool(load_library().tib_gemm_f32_tcgen05_takes(c_void_p(x), c_void_p(w), c_int(n), c_int(k), c_int64(ldx), c_int64(ldw))) == takes


def test_a_timeout_code_names_one_kernel():
    """The first digit behind 0x7C00 belongs to one file, as the list in tcgen05.cuh says."""
    listed = {digit: name for digits, name in re.findall(r"((?:[0-9A-F], )*[0-9A-F]) (\w+?_\w+)", (CSRC / "tcgen05.cuh").read_text().split("first digit of xx:")[1].split("// Bounded")[0])
              for digit in digits.split(", ")}
    used = {(code, path.stem) for path in CSRC.glob("*.cu") for code in re.findall(r"0x7C00([0-9A-F])[0-9A-F]\b", path.read_text())}
    assert used and {code for code, _ in used} == set(listed)
    assert all(listed[code] == name for code, name in used), used


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.stem)
def test_dependents_are_let_in_once_tensor_memory_is_taken(path):
    """A kernel that takes tensor memory lets the next kernel's blocks in only behind that: one that was placed first, had the columns and waited for
    this kernel's end would never get it.  The products of few rows take half of the columns at most, so that two blocks have room."""
    for kernel in re.split(r"(?=__global__ void)", path.read_text())[1:]:
        taken = [m.start() for m in re.finditer(r"ft_setup\(|tcgen05\.alloc", kernel)]
        let_in = kernel.find("pdl_trigger()")
        if taken and let_in >= 0 and path.stem not in ("gemm_decode", "gemm_tcgen05"):
            assert let_in > taken[0], kernel.split("(", 3)[:3]
