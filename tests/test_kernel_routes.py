"""What can be said of the kernels without a GPU: the host's rules on which one a call takes, and rules that their sources keep."""
import re
import struct
from ctypes import c_char_p, c_int, c_int64, c_void_p
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


@pytest.mark.parametrize("name", sorted(set(re.findall(r"\b(?:lib\(\)|library)\.(tib_\w+)\(", (CSRC.parent / "kernels" / "ops.py").read_text()))))
def test_every_call_of_the_parts_is_packed_by_its_own_types(name):
    """As many slots as the function has parameters in its source, d for a floating-point number and q for anything else."""
    from torchinferno_b200.kernels.library import load_library
    slots = getattr(load_library(), name + "_slots")
    slots.restype = c_char_p
    found = [m.group(1) for path in CSRC.glob("*.cu") for m in [re.search(rf"TIB_API int {name}\(([^)]*)\)", path.read_text())] if m]
    assert len(found) == 1
    parameters = [p.strip() for p in found[0].split(",") if p.strip()]
    assert slots().decode() == "".join("d" if re.match(r"(const )?(float|double) \w+$", p) else "q" for p in parameters)


def test_packed_calls_pass_their_arguments():
    from torchinferno_b200.kernels import ops
    library = ops.lib()
    assert bool(library.tib_gemm_f32_tcgen05_takes(1 << 40, 1 << 41, 2048, 2048, 2048, 2048))           # (addresses beyond 32 bits)
    assert not library.tib_gemm_f32_tcgen05_takes((1 << 40) + 4, 1 << 41, 2048, 2048, 2048, 2048)
    assert library.tib_embedding(0, 0, 0, 1, 8, 8, 0.5, 0, 0, 0, 0, 0) == -5                              # (a refusal comes back as it is)
    with pytest.raises(struct.error):
        library.tib_plan_product(1, 2, 3)


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
