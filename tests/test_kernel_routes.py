"""What can be said of the kernels without a GPU: the host's rules on which one a call takes, and rules that their sources keep."""
import re
import struct
from ctypes import c_char_p, c_int, c_int64, c_void_p
from pathlib import Path

import pytest
import torch

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


@pytest.mark.parametrize("n, k", [(1096, 1088), (1104, 1088), (24584, 1024), (28672, 4096)])
@pytest.mark.parametrize("epilogue", ["none", "swiglu"])
def test_what_is_measured_is_what_the_kernel_takes(n, k, epilogue):
    """Every tile width and K split that is timed is one the kernel takes with the weight's own epilogue (outputs of pairs in whole eights)."""
    from torchinferno_b200.kernels import gemm, ops
    code = ops.DG_SWIGLU if epilogue == "swiglu" else ops.DG_PLAIN
    found = gemm._candidates(n, k, epilogue)
    assert all(ops.gemm_decode_supports(8, n, k, *config, code) for config in found)
    assert bool(found) == (epilogue == "none" or n % 16 == 0)


@pytest.mark.parametrize("members, size, products, distinct", [
    (1, 4, 32, 32), (1, 64, 32, 16), (3, 64, 32, 16), (16, 64, 32, 16), (20, 64, 32, 20), (1, 1000, 5, 2), (1, 1024, 4, 1), (2, 8192, 2, 2), (40, 4, 40, 40)])
def test_a_measured_walk_reads_every_weight_from_memory(members, size, products, distinct, monkeypatch):
    """Members first, copies of them behind; none is read again before TUNE_COLD bytes of them were read, or at all; the copies are smaller than that together."""
    from torchinferno_b200.kernels import gemm
    monkeypatch.setattr(gemm, "TUNE_COLD", 1024)
    monkeypatch.setattr(gemm, "TUNE_BYTES", 4096)
    own = [torch.full((size // 2, 1), float(i), dtype=torch.bfloat16) for i in range(members)]
    walk = gemm._walk_weights(own)
    places = [w.data_ptr() for w in walk]
    assert len(walk) == products and len(set(places)) == distinct and places[:members] == [w.data_ptr() for w in own]
    assert all(torch.equal(w, own[i % distinct % members]) for i, w in enumerate(walk))
    assert all(p not in places[i + 1:i + distinct] for i, p in enumerate(places))
    assert (distinct == products or distinct * size >= 1024) and (distinct - members) * size < 1024


def test_a_walk_without_room_for_copies_reads_what_there_is(monkeypatch):
    from torchinferno_b200.kernels import gemm
    clone, made = torch.Tensor.clone, []

    def limited(self):
        if len(made) == 3:
            raise torch.OutOfMemoryError("no room")
        made.append(self)
        return clone(self)

    own = [torch.zeros(8, 8, dtype=torch.bfloat16) for _ in range(2)]
    monkeypatch.setattr(torch.Tensor, "clone", limited)
    walk = gemm._walk_weights(own)
    assert len(walk) == gemm.TUNE_PRODUCTS and len({w.data_ptr() for w in walk}) == 5 and walk[0] is own[0] and walk[5] is own[0]


def test_a_stored_choice_names_how_it_was_measured(monkeypatch):
    from torchinferno_b200.kernels import gemm
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda device: "a GPU")
    keys = [gemm._choice_key(2048, 1024, torch.device("cuda", 0), epilogue) for epilogue in ("none", "swiglu")]
    for name in ("TUNE_PRODUCTS", "TUNE_BYTES", "TUNE_COLD", "TUNE_MARGIN", "TUNE_SWIGLU_US"):
        with monkeypatch.context() as patch:
            patch.setattr(gemm, name, 2 * getattr(gemm, name))
            keys.append(gemm._choice_key(2048, 1024, torch.device("cuda", 0), "none"))
    assert len(set(keys)) == 7


@pytest.mark.parametrize("few_rows, library, none, swiglu", [
    (10.0, 10.0, True, True), (10.4, 10.0, True, True), (10.5, 10.0, False, True), (12.0, 10.0, False, True), (12.1, 10.0, False, False),
    (103.0, 100.0, True, True), (104.1, 100.0, False, False), (float("nan"), 10.0, False, False)])
def test_the_line_between_the_few_rows_kernel_and_the_library(few_rows, library, none, swiglu):
    """4 % for all weights; 2 us for those whose activation is then made of fp32 sums."""
    from torchinferno_b200.kernels import gemm
    assert (gemm._few_rows_wins(few_rows, library, "none"), gemm._few_rows_wins(few_rows, library, "swiglu")) == (none, swiglu)


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
