"""Each CUDA kernel alone against a plain PyTorch reference (float64 on the CPU), at sizes other
than the engine's tiny models: widths that are no power of two, head sizes in steps of 16, odd
group sizes, page sizes from 1 up, windows, ragged batches."""
import math

import pytest
import torch

import plain_llama
from gpu_common import need_gpu

pytestmark = pytest.mark.gpu
DTYPES = [torch.float32, torch.bfloat16]


def tol(dtype):
    return dict(atol=2e-6, rtol=2e-6) if dtype == torch.float32 else dict(atol=1e-2, rtol=1.6e-2)


def dev(t, dtype=None):
    return t.to("cuda", dtype) if dtype else t.to("cuda")


def as_ref(t):
    return t.detach().cpu().double()


def rnd(*shape, dtype=torch.float32, scale=1.0, seed=0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g) * scale).to(dtype)


# ------------------------------------------------------------ elementwise
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("hidden", [100, 4096, 5000])
def test_embedding(dtype, hidden):
    need_gpu()
    from torchinferno_b200.kernels import ops
    table = rnd(37, hidden, dtype=dtype)
    ids = torch.tensor([3, 36, 0, 3, 40, -1], dtype=torch.int32)
    out = torch.empty(6, hidden, device="cuda")
    ops.embedding(dev(ids), dev(table), out)
    assert torch.equal(out[:4].cpu(), table[ids[:4].long()].float())
    assert torch.isnan(out[4:]).all()                      # ids outside the table must show


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("rows, hidden, eps", [(5, 100, 1e-5), (3, 4096, 1e-6), (2, 5000, 3e-6), (1, 24, 1e-2)])
def test_add_rmsnorm(dtype, rows, hidden, eps):
    need_gpu()
    from torchinferno_b200.kernels import ops
    res0, delta, w = rnd(rows, hidden, scale=3), rnd(rows, hidden, dtype=dtype, seed=1), 1 + 0.2 * rnd(hidden, seed=2)
    # plain norm of the residual
    res = dev(res0.clone())
    out = torch.empty(rows, hidden, dtype=dtype, device="cuda")
    ops.add_rmsnorm(None, res, dev(w), eps, out)
    want = plain_llama.rms_norm(res0.double(), w.double(), eps)
    assert torch.allclose(as_ref(out), want, **tol(dtype)) and torch.equal(res.cpu(), res0)
    # fused add: the residual is updated in 32-bit, the normed rows leave in dtype
    ops.add_rmsnorm(dev(delta), res, dev(w), eps, out)
    summed = res0 + delta.float()
    assert torch.equal(res.cpu(), summed)
    assert torch.allclose(as_ref(out), plain_llama.rms_norm(summed.double(), w.double(), eps), **tol(dtype))
    # rows: only the picked rows, residual untouched
    pick = torch.tensor([rows - 1, 0, rows - 1], dtype=torch.int32)
    out3 = torch.empty(3, hidden, dtype=dtype, device="cuda")
    before = res.clone()
    ops.add_rmsnorm(dev(delta), res, dev(w), eps, out3, rows=dev(pick))
    want3 = plain_llama.rms_norm((summed + delta.float()).double(), w.double(), eps)[pick.long()]
    assert torch.allclose(as_ref(out3), want3, **tol(dtype)) and torch.equal(res, before)
    # rows of the activation type
    x = rnd(rows, hidden, dtype=dtype, seed=5)
    ops.rmsnorm(dev(x), dev(w), eps, out)
    assert torch.allclose(as_ref(out), plain_llama.rms_norm(x.double(), w.double(), eps), **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("rows, inter", [(7, 200), (1, 14336), (33, 17)])
def test_swiglu(dtype, rows, inter):
    need_gpu()
    from torchinferno_b200.kernels import ops
    gu = rnd(rows, 2 * inter, dtype=dtype, scale=3)
    out = torch.empty(rows, inter, dtype=dtype, device="cuda")
    ops.swiglu(dev(gu), out)
    g, u = gu.double()[:, :inter], gu.double()[:, inter:]
    assert torch.allclose(as_ref(out), g / (1 + torch.exp(-g)) * u, **tol(dtype))


def test_cast_and_scatter():
    need_gpu()
    from torchinferno_b200.kernels import ops
    x = rnd(1000, 3)
    y = ops.cast(dev(x), torch.empty(1000, 3, dtype=torch.bfloat16, device="cuda"))
    assert torch.equal(y.cpu(), x.to(torch.bfloat16))
    assert torch.equal(ops.cast(y, torch.empty(1000, 3, device="cuda")).cpu(), x.to(torch.bfloat16).float())
    table = torch.full((4, 5), -1, dtype=torch.int32, device="cuda")
    ops.scatter_i32(table, dev(torch.tensor([7, 0, 19, 99], dtype=torch.int32)), dev(torch.tensor([70, 1, 190, 5], dtype=torch.int32)))
    want = torch.full((20,), -1, dtype=torch.int32)
    want[7], want[0], want[19] = 70, 1, 190
    assert torch.equal(table.cpu().view(-1), want)


# ------------------------------------------------------------------- GEMM
@pytest.mark.parametrize("m, n, k", [(1, 64, 64), (37, 129, 100), (130, 67, 257), (5, 1000, 4096)])
@pytest.mark.parametrize("wdtype", DTYPES)
def test_gemm_f32_is_true_fp32_and_row_independent(m, n, k, wdtype):
    need_gpu()
    from torchinferno_b200.kernels import ops
    x, w = rnd(m, k, scale=2), rnd(n, k, dtype=wdtype, seed=3)
    out = ops.gemm_f32(dev(x), dev(w), torch.empty(m, n, device="cuda"))
    want = x.double() @ w.double().T
    # fp32 accumulation over k terms: error far below what a tf32 or bf16 product would leave
    assert (as_ref(out) - want).abs().max() <= 4e-7 * math.sqrt(k) * (x.abs().max() * w.float().abs().max()).item() * math.sqrt(k)
    one = ops.gemm_f32(dev(x[m // 2: m // 2 + 1].contiguous()), dev(w), torch.empty(1, n, device="cuda"))
    assert torch.equal(one[0], out[m // 2])               # a row does not depend on the rows beside it


@pytest.mark.parametrize("m, n, k", [(128, 256, 64), (1, 8, 64), (200, 520, 192), (77, 1000, 4096), (300, 264, 1024), (2048, 512, 14336)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_tcgen05(m, n, k, out_dtype):
    """The TMA / tcgen05 / TMEM product against float64, with rows and columns that do not fill the
    128 x 256 tiles, a long K (many trips round the stage ring), and both output types."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    x, w = rnd(m, k, dtype=torch.bfloat16), rnd(n, k, dtype=torch.bfloat16, scale=0.05, seed=3)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = ops.gemm_tcgen05(dev(x), dev(w), torch.full((m, n), float("nan"), dtype=out_dtype, device="cuda"), err)
    assert int(err) == 0                                   # no bounded wait ran out
    want = (x.cuda().double() @ w.cuda().double().T).cpu()
    bound = (1e-2 if out_dtype == torch.bfloat16 else 2e-5) * want.abs().max() + 1e-6
    assert (as_ref(out) - want).abs().max() <= bound
    with pytest.raises(ops.KernelError, match="size"):     # K must be a multiple of 64
        ops.gemm_tcgen05(dev(rnd(4, 96, dtype=torch.bfloat16)), dev(rnd(8, 96, dtype=torch.bfloat16)), torch.empty(4, 8, dtype=out_dtype, device="cuda"))


@pytest.mark.parametrize("m, n, k", [(256, 256, 64), (1, 8, 64), (200, 520, 192), (77, 1000, 4096), (600, 264, 1024), (2048, 512, 14336),
                                     (515, 1288, 512)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_tcgen05_on_pairs_of_sms(m, n, k, out_dtype):
    """The `cta_group::2` product (two blocks per 256 x 256 tile) against float64: one tile, rows and columns that
    do not fill the tiles (among them tiles whose second block has no rows at all), a long K, more tiles than
    pairs of SMs take in one round, and both output types."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    x, w = rnd(m, k, dtype=torch.bfloat16), rnd(n, k, dtype=torch.bfloat16, scale=0.05, seed=3)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = ops.gemm_tcgen05_2cta(dev(x), dev(w), torch.full((m, n), float("nan"), dtype=out_dtype, device="cuda"), err)
    assert int(err) == 0                                   # no bounded wait ran out
    want = (x.cuda().double() @ w.cuda().double().T).cpu()
    bound = (1e-2 if out_dtype == torch.bfloat16 else 2e-5) * want.abs().max() + 1e-6
    assert (as_ref(out) - want).abs().max() <= bound
    with pytest.raises(ops.KernelError, match="size"):     # K must be a multiple of 64
        ops.gemm_tcgen05_2cta(dev(rnd(4, 96, dtype=torch.bfloat16)), dev(rnd(8, 96, dtype=torch.bfloat16)), torch.empty(4, 8, dtype=out_dtype, device="cuda"))


@pytest.mark.parametrize("m, n, k, splits", [(8, 128, 64, 0), (1, 8, 64, 1), (8, 6144, 4096, 0), (16, 4096, 4096, 4), (5, 1000, 4096, 0),
                                             (8, 4096, 14336, 8), (33, 520, 192, 3), (64, 264, 1024, 0), (17, 28672, 512, 0),
                                             (48, 136, 9472, 5)])
@pytest.mark.parametrize("w_kn", [False, True])
def test_gemm_tcgen05_swapab(m, n, k, splits, w_kn):
    """The few-rows product (weights as the 128-row operand, K split over a cluster) against float64: one tile, a
    ragged last tile, every padding of the rows, splits chosen and forced, more tiles than clusters, and the weights
    stored [out, in] (K-major operand) as well as [in, out] (MN-major operand); both output types."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    x, w = rnd(m, k, dtype=torch.bfloat16), rnd(n, k, dtype=torch.bfloat16, scale=0.05, seed=3)
    want = (x.cuda().double() @ w.cuda().double().T).cpu()
    wd = dev(w.t().contiguous()) if w_kn else dev(w)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    for out_dtype in (torch.bfloat16, torch.float32):
        out = ops.gemm_tcgen05_swapab(dev(x), wd, torch.full((m, n), float("nan"), dtype=out_dtype, device="cuda"), err,
                                      splits=splits, w_kn=w_kn)
        assert int(err) == 0                               # no bounded wait ran out
        bound = (1e-2 if out_dtype == torch.bfloat16 else 2e-5) * want.abs().max() + 1e-6
        assert (as_ref(out) - want).abs().max() <= bound
    with pytest.raises(ops.KernelError, match="size"):     # at most 64 rows
        ops.gemm_tcgen05_swapab(dev(rnd(65, 64, dtype=torch.bfloat16)), dev(rnd(8, 64, dtype=torch.bfloat16)),
                                torch.empty(65, 8, dtype=torch.bfloat16, device="cuda"))


@pytest.mark.parametrize("epilogue", ["none", "swiglu"])
def test_the_choice_of_a_shape_with_one_weight_is_measured_from_memory(epilogue, monkeypatch):
    """32 captured products in a row never read one weight twice (a hybrid model's only layer of a shape finds its weight in memory, not in the L2)."""
    need_gpu()
    from torchinferno_b200.kernels import gemm, ops
    read, product = [], ops.library_gemm
    monkeypatch.setattr(gemm, "_stored_choices", dict)
    monkeypatch.setattr(gemm, "_store_choice", lambda name, choice: None)

    def library_gemm(x, w, *args, **options):
        if torch.cuda.is_current_stream_capturing():
            read.append(w.data_ptr())
        return product(x, w, *args, **options)

    monkeypatch.setattr(ops, "library_gemm", library_gemm)
    weight = gemm.LinearWeight(dev(rnd(1104, 1088, dtype=torch.bfloat16)), few_rows_tcgen05=None, epilogue=epilogue)
    gemm.tune_few_rows()
    gemm._tuned.pop((1104, 1088, weight.tensor.device, epilogue))
    assert len(read) >= 32 and all(len(set(read[i:i + 32])) == 32 for i in range(len(read) - 31))


@pytest.mark.parametrize("choice", ["measured", "swapab", "library"])
def test_pairs_of_odd_eights_bind_and_run(choice):
    """A SwiGLU weight whose outputs are no whole eights: the few-rows kernel does not take it with its epilogue."""
    need_gpu()
    from torchinferno_b200.kernels import gemm
    n, k = 1096, 1088
    w, x = rnd(n, k, dtype=torch.bfloat16, scale=0.05), rnd(8, k, dtype=torch.bfloat16, seed=1)
    gemm.set_few_rows_choice(choice)
    try:
        weight = gemm.LinearWeight(dev(w), few_rows_tcgen05=None, epilogue="swiglu")
        gemm._tuned.pop((n, k, weight.tensor.device, "swiglu"), None)
        gemm.tune_few_rows()
        got = as_ref(gemm.linear_swiglu(dev(x), weight))
    finally:
        gemm._tuned.pop((n, k, weight.tensor.device, "swiglu"), None)
        gemm.set_few_rows_choice("measured")
    both = x.double() @ w.double().T
    gate, up = both[:, 0::2], both[:, 1::2]
    want = gate * torch.sigmoid(gate) * up
    # (gate, up and the result are rounded to bfloat16: 2^-9 each, times the slopes of the silu and the product, at most 1.1 and 1)
    assert (got - want).norm() <= 4 * 2.0 ** -9 * want.norm()


def test_few_rows_kernel_is_chosen_by_measurement_and_either_choice_is_right():
    """Weights that leave their few-rows kernel open get it from tune_few_rows (the hand-written kernel up to 0, 4, 8,
    16, 32 or 64 rows, with the tile width and K split that measured fastest): one decision per shape, kept for the
    process and on disk, the same for every weight of the shape; a slice of the weight inherits it; whichever kernel
    was chosen, and whichever is forced, the product is right at few and at many rows; and so is silu(gate) * up
    of a weight bound with the SwiGLU epilogue, fused or not."""
    need_gpu()
    from torchinferno_b200.kernels import gemm
    from torchinferno_b200.kernels.gemm import LinearWeight, linear, linear_swiglu
    n, k = 1160, 2048
    ws = [rnd(n, k, dtype=torch.bfloat16, scale=0.05, seed=i) for i in range(3)]
    open_weights = [LinearWeight(dev(w), few_rows_tcgen05=None) for w in ws]
    assert all(w.few_rows == 0 for w in open_weights)                     # the library until measured
    decisions = gemm.tune_few_rows()
    key = (n, k, open_weights[0].tensor.device, "none")
    rows, features, splits = decisions[key]
    assert rows in (0, 4, 8, 16, 32, 64) and features in (128, 256) and 0 <= splits <= 8
    assert all((w.few_rows, w.features, w.splits) == decisions[key] for w in open_weights)
    later = LinearWeight(dev(ws[0]), few_rows_tcgen05=None)
    assert gemm.tune_few_rows()[key] == decisions[key] and later.few_rows == open_weights[0].few_rows
    gemm._tuned.pop(key)                                                   # a new process reads what this one stored
    again = [LinearWeight(dev(w), few_rows_tcgen05=None) for w in ws]
    assert gemm.tune_few_rows()[key] == decisions[key] and again[0].splits == splits
    forced = [LinearWeight(dev(ws[0]), few_rows_tcgen05=True), LinearWeight(dev(ws[0]), few_rows_tcgen05=False)]
    assert [w.few_rows for w in forced] == [LinearWeight.FEW_ROWS, 0] and LinearWeight.FEW_ROWS == 64
    configured = LinearWeight(dev(ws[0]), few_rows_tcgen05=True)
    configured.features, configured.splits = 128, 4
    glu = [LinearWeight(dev(ws[0][:1152]), few_rows_tcgen05=flag, epilogue="swiglu") for flag in (True, False)]
    glu[0].splits = 1
    for m in (1, 4, 5, 8, 9, 16, 17, 33, 64, 65, 200):
        x = rnd(m, k, dtype=torch.bfloat16, seed=50 + m)
        want = x.double() @ ws[0].double().T
        for weight in (open_weights[0], later, configured, *forced):
            out = linear(dev(x), weight)
            assert (as_ref(out) - want).abs().max() <= 1e-2 * want.abs().max() + 1e-6
            part = linear(dev(x), weight.rows(64, 1096))
            assert (as_ref(part) - want[:, 64:1096]).abs().max() <= 1e-2 * want.abs().max() + 1e-6
        gate, up = want[:, 0:1152:2], want[:, 1:1152:2]
        act = gate / (1 + torch.exp(-gate)) * up
        for weight in glu:
            got = linear_swiglu(dev(x), weight)
            assert got.shape == (m, 576) and (as_ref(got) - act).abs().max() <= 1.5e-2 * act.abs().max() + 1e-6


@pytest.mark.parametrize("m, n, k", [(1, 256, 64), (8, 6144, 4096), (16, 28672, 4096), (5, 1000, 4096), (33, 520, 192), (64, 4096, 4096)])
def test_gemm_decode_every_tile_width_split_and_epilogue(m, n, k):
    """The few-rows kernel on [in, out] weights: tiles of 128 features with K shared by 1 to 8 blocks of a cluster,
    tiles of 256 features unsplit, bf16 and fp32 results, and the SwiGLU epilogue on interleaved gate/up columns,
    against float64; NaN in the output buffer beforehand shows what was not written."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    x, w = rnd(m, k, dtype=torch.bfloat16), rnd(k, n, dtype=torch.bfloat16, scale=0.05, seed=3)
    want = x.double() @ w.double()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    ran = 0
    for features in (128, 256):
        for splits in (1, 2, 3, 5, 8):
            if not ops.gemm_decode_supports(m, n, k, features, splits):
                continue
            for out_dtype in (torch.bfloat16, torch.float32):
                out = ops.gemm_decode(dev(x), dev(w), torch.full((m, n), float("nan"), dtype=out_dtype, device="cuda"),
                                      features=features, splits=splits, error_word=err)
                bound = (1e-2 if out_dtype == torch.bfloat16 else 1e-4) * want.abs().max() + 1e-6
                assert (as_ref(out) - want).abs().max() <= bound, (features, splits, out_dtype)
                ran += 1
        if n % 16 == 0:
            gate, up = want[:, 0::2], want[:, 1::2]
            act = gate / (1 + torch.exp(-gate)) * up
            out = ops.gemm_decode(dev(x), dev(w), torch.full((m, n // 2), float("nan"), dtype=torch.bfloat16, device="cuda"),
                                  features=features, splits=1, epilogue=ops.DG_SWIGLU, error_word=err)
            assert (as_ref(out) - act).abs().max() <= 1e-2 * act.abs().max() + 1e-6
    assert ran >= 4 and int(err) == 0
    assert not ops.gemm_decode_supports(65, n, k) and not ops.gemm_decode_supports(m, n, k, 256, 2)
    assert not ops.gemm_decode_supports(m, n, k, 128, 2, ops.DG_SWIGLU) and not ops.gemm_decode_supports(m, n, k + 8)
    with pytest.raises(ops.KernelError, match="size"):
        ops.gemm_decode(dev(x), dev(w), torch.empty(m, n, dtype=torch.bfloat16, device="cuda"), features=256, splits=2)


def _records(rows):
    """A record table [slots, 8] from {slot: (length, last token, seed, temperature, drawn)}."""
    import struct
    table = torch.zeros(max(rows) + 1, 8, dtype=torch.int32)
    for slot, (length, last, seed, temperature, drawn) in rows.items():
        seed &= 0xFFFFFFFFFFFFFFFF
        words = [length, last, seed & 0xFFFFFFFF, seed >> 32, struct.unpack("<I", struct.pack("<f", temperature))[0], drawn]
        table[slot, :6] = torch.tensor([w - (1 << 32) if w >= (1 << 31) else w for w in words], dtype=torch.int64).to(torch.int32)
    return table


def test_decode_inputs_come_from_the_requests_records_which_move_on():
    """The first kernel of a captured decode step: request i of the step sits in slot slots[i]; its next token and
    its position come from its record, whose length moves one on.  Records of other slots, the other words of a
    record and the tails of longer buffers stay as they are; a slot outside the table yields token -1."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    i32 = lambda xs: dev(torch.tensor(xs, dtype=torch.int32))
    table = _records({0: (4, 100, 7, 0.5, 1), 1: (9, 9, 9, 0.0, 9), 2: (511, 300, -3, 1.5, 2), 5: (0, 200, 1 << 40, 0.0, 0)})
    before, records = table.clone(), dev(table)
    tokens, positions = i32([7, 8, 9, 77]), i32([-1, -1, -1, 55])
    ops.decode_inputs(records, i32([2, 5, 0]), tokens, positions)
    assert tokens.tolist() == [300, 200, 100, 77] and positions.tolist() == [511, 0, 4, 55]
    after = records.cpu()
    assert after[:, 0].tolist() == [5, 9, 512, 0, 0, 1]
    assert torch.equal(after[:, 1:], before[:, 1:])
    ops.decode_inputs(records, i32([6, 1]), tokens, positions)           # slot 6 is outside the table
    assert tokens.tolist()[:2] == [-1, 9] and positions.tolist()[:2] == [0, 9]
    with pytest.raises(ops.KernelError, match="shorter"):
        ops.decode_inputs(records, i32([0, 1, 2]), i32([1]), positions)


def test_sampling_from_records_is_sampling_with_the_same_parameters_given_by_hand():
    """The sampler reads temperature, seed and the position of the drawn token (the request's length) from the
    record of each row's request, draws what the explicit form draws, and leaves the token in the record."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    g = torch.Generator().manual_seed(5)
    logits = dev(torch.randn(4, 1000, generator=g) * 3)
    rows = {3: (17, -1, 12345678901234567, 0.8, 0), 1: (40, 5, -99, 1.3, 7), 0: (5, 5, 3, 0.0, 2), 6: (1, 1, 1, 0.7, 0)}
    records = dev(_records(rows))
    slots = dev(torch.tensor([3, 0, 1, 6], dtype=torch.int32))
    out, history = torch.empty(4, dtype=torch.int32, device="cuda"), torch.full((6,), -1, dtype=torch.int32, device="cuda")
    ops.sample_records(logits, out, records, slots, history)
    order = [3, 0, 1, 6]
    as_i64 = lambda s: ((s & 0xFFFFFFFFFFFFFFFF) ^ (1 << 63)) - (1 << 63)
    want = ops.sample(logits, torch.empty(4, dtype=torch.int32, device="cuda"),
                      dev(torch.tensor([rows[s][3] for s in order])), dev(torch.tensor([as_i64(rows[s][2]) for s in order])),
                      dev(torch.tensor([rows[s][0] for s in order], dtype=torch.int32)))
    assert out.tolist() == want.tolist() and history.tolist() == want.tolist() + [-1, -1]
    assert out.tolist()[1] == int(logits[1].argmax())                    # temperature 0 is greedy
    after = records.cpu()
    for row, slot in enumerate(order):
        assert after[slot, 1].item() == want[row].item() and after[slot, 5].item() == rows[slot][4] + 1
        assert after[slot, 0].item() == rows[slot][0]                    # the length is the decode step's to move


@pytest.mark.parametrize("m, n, k", [(1, 72, 40), (8, 4096, 4096), (17, 1000, 264), (300, 136, 2048)])
@pytest.mark.parametrize("w_kn", [False, True])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_library_gemm_both_layouts(m, n, k, w_kn, out_dtype):
    """cuBLAS called from the engine's library (its own handle and workspace): weights stored [out, in] and
    [in, out], bf16 and fp32 results, against float64."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    x, w = rnd(m, k, dtype=torch.bfloat16), rnd(n, k, dtype=torch.bfloat16, scale=0.05, seed=3)
    ops.library_gemm_ready(torch.device("cuda", torch.cuda.current_device()))
    out = ops.library_gemm(dev(x), dev(w.t().contiguous()) if w_kn else dev(w),
                           torch.full((m, n), float("nan"), dtype=out_dtype, device="cuda"), w_kn=w_kn)
    want = x.double() @ w.double().T
    bound = (1e-2 if out_dtype == torch.bfloat16 else 2e-5) * want.abs().max() + 1e-6
    assert (as_ref(out) - want).abs().max() <= bound


# -------------------------------------------------------------- RoPE + KV
def paged_layout(n_requests, lengths, page_size, kv_heads, d, dtype, spare_pages=3, seed=0):
    """A pool with NaN everywhere, shuffled page ids, and block tables for the given lengths."""
    g = torch.Generator().manual_seed(seed)
    pages_per = [-(-n // page_size) for n in lengths]
    total = sum(pages_per) + spare_pages
    order = torch.randperm(total, generator=g).tolist()
    width = max(pages_per) + 1
    table = torch.full((n_requests + 2, width), -1, dtype=torch.int32)
    slots = torch.randperm(n_requests + 2, generator=g)[:n_requests].tolist()
    for r, slot in enumerate(slots):
        for p in range(pages_per[r]):
            table[slot, p] = order.pop()
    pool = torch.full((total, 2, kv_heads, page_size, d), float("nan"), dtype=dtype)
    return pool, table, slots


def fill_pages(pool, table, slot, k, v, start=0):
    """k, v: [kv_heads, T, d] written at positions start.. of the request in ``slot``."""
    p = pool.shape[3]
    for t in range(k.shape[1]):
        pos = start + t
        page = int(table[slot, pos // p])
        pool[page, 0, :, pos % p] = k[:, t]
        pool[page, 1, :, pos % p] = v[:, t]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads, kv_heads, d, rot, inter, page", [
    (4, 2, 16, None, False, 4), (5, 1, 48, None, False, 3), (3, 3, 80, 32, False, 16), (8, 2, 128, None, True, 16),
    (2, 1, 64, 0, False, 5)])
def test_rope_append(dtype, heads, kv_heads, d, rot, inter, page):
    need_gpu()
    from torchinferno_b200.kernels import ops
    from torchinferno_b200.parts.rope import rotary_frequencies
    rot_dim = d if rot is None else rot
    starts, lens = [0, 37, 5], [6, 1, 9]                 # three entries: a prompt start, a decode, a portion
    pool, table, slots = paged_layout(3, [s + n for s, n in zip(starts, lens)], page, kv_heads, d, dtype)
    positions = torch.tensor([s + i for s, n in zip(starts, lens) for i in range(n)], dtype=torch.int32)
    token_slot = torch.tensor([slots[e] for e, n in enumerate(lens) for _ in range(n)], dtype=torch.int32)
    n = int(positions.numel())
    qkv = rnd(n, (heads + 2 * kv_heads) * d, dtype=dtype)
    scaling = {"rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
               "original_max_position_embeddings": 16}
    inv_freq = rotary_frequencies(rot_dim, 10000.0, scaling) if rot_dim else torch.zeros(0)
    pool_d, q_out = dev(pool), torch.empty(n, heads * d, dtype=dtype, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.rope_append(dev(qkv), q_out, pool_d, dev(positions), dev(token_slot), dev(table), dev(inv_freq),
                    heads, kv_heads, d, rot_dim=rot_dim, interleaved=inter, error_word=err)
    assert int(err) == 0

    def rotate(x):                                      # x [T, H, d] float64
        if rot_dim == 0:
            return x
        ang = (positions.float()[:, None] * inv_freq[None, :]).double()      # fp32 product, as the kernel
        c, s = ang.cos()[:, None, :], ang.sin()[:, None, :]
        out = x.clone()
        if inter:
            lo, hi = x[..., 0:rot_dim:2], x[..., 1:rot_dim:2]
            out[..., 0:rot_dim:2], out[..., 1:rot_dim:2] = lo * c - hi * s, hi * c + lo * s
        else:
            h = rot_dim // 2
            lo, hi = x[..., :h], x[..., h:rot_dim]
            out[..., :h], out[..., h:rot_dim] = lo * c - hi * s, hi * c + lo * s
        return out

    q, k, v = qkv.double().split([heads * d, kv_heads * d, kv_heads * d], dim=1)
    assert torch.allclose(as_ref(q_out).view(n, heads, d), rotate(q.view(n, heads, d)), **tol(dtype))
    want_k, got = rotate(k.reshape(n, kv_heads, d)), pool_d.cpu()
    written = torch.zeros(pool.shape[0], page, dtype=torch.bool)
    for t in range(n):
        pos, slot = int(positions[t]), int(token_slot[t])
        pg = int(table[slot, pos // page])
        written[pg, pos % page] = True
        assert torch.allclose(got[pg, 0, :, pos % page].double(), want_k[t], **tol(dtype))
        assert torch.equal(got[pg, 1, :, pos % page], v.reshape(n, kv_heads, d)[t].to(dtype))
    untouched = got.permute(0, 3, 1, 2, 4)[~written]
    assert torch.isnan(untouched).all()                 # nothing else in the pool was written
    # a page id outside the pool is reported, not written
    bad = table.clone()
    bad[slots[1], 37 // page] = pool.shape[0] + 5
    ops.rope_append(dev(qkv), q_out, pool_d, dev(positions), dev(token_slot), dev(bad), dev(inv_freq),
                    heads, kv_heads, d, rot_dim=rot_dim, interleaved=inter, error_word=err)
    assert int(err) != 0


# -------------------------------------------------------------- attention
def attention_case(dtype, heads, kv_heads, d, page, entries, window=0, seed=0, standout=None, kernel="simt", splits=None):
    """entries: list of (kv_start, q_len).  Returns kernel output and the float64 reference.

    kernel "simt": the CUDA-core kernel; "mma": the tensor-core pair (portions by the prefill kernel,
    single tokens by the split decode kernel, as the engine dispatches them); "mma_prefill": the
    prefill kernel alone for every entry; "tma": as "mma" with the single tokens by the TMA decode kernel.
    ``splits`` = (num_splits, chunk) forces a split."""
    from torchinferno_b200.kernels import ops
    lengths = [s + n for s, n in entries]
    pool, table, slots = paged_layout(len(entries), lengths, page, kv_heads, d, dtype, seed=seed)
    q_rows, refs, q_start = [], [], [0]
    group = heads // kv_heads
    for e, (start, n) in enumerate(entries):
        total = start + n
        k, v = rnd(kv_heads, total, d, dtype=dtype, seed=seed + e), rnd(kv_heads, total, d, dtype=dtype, seed=seed + 50 + e)
        q = rnd(heads, n, d, dtype=dtype, seed=seed + 100 + e)
        if standout is not None and standout < total:
            # every query shares a component along u, and one far key points along u: its score
            # (about 12) stands out from the others (about N(0, 1)) for every query that may see it
            u = torch.ones(d) / math.sqrt(d)
            q = (q.float() * 0.2 + 8.0 * u).to(dtype)
            k[:, standout] = (12.0 * math.sqrt(d) / 8.0 * u).to(dtype)
            v[:, standout] = (v[:, standout].float() + 7).to(dtype)
        fill_pages(pool, table, slots[e], k, v)
        q_rows.append(q.transpose(0, 1).reshape(n, heads * d))
        full_q = torch.zeros(heads, total, d, dtype=torch.float64)
        full_q[:, start:] = q.double()
        ref = plain_llama.causal_attention(full_q, k.double(), v.double(), group, window=window or None)[:, start:]
        refs.append(ref.transpose(0, 1).reshape(n, heads * d))
        q_start.append(q_start[-1] + n)
    q_all = torch.cat(q_rows)
    out = torch.empty_like(q_all, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    i32 = lambda xs: dev(torch.tensor(xs, dtype=torch.int32))
    scale, max_q = 1.0 / math.sqrt(d), max(n for _, n in entries)
    args = (dev(q_all), dev(pool), out, i32(q_start), i32([s for s, _ in entries]), i32(slots), dev(table), len(entries))
    if kernel == "simt":
        ops.paged_attention_simt(*args, max_q, heads, kv_heads, d, scale, window=window, error_word=err)
    elif kernel == "mma_prefill":
        ops.prefill_attention(*args, max_q, heads, kv_heads, d, scale, window=window)
    elif kernel == "tcgen05_prefill":
        ops.prefill_attention_tcgen05(*args, max_q, heads, kv_heads, d, scale, window=window, error_word=err)
    else:
        out.fill_(float("nan"))
        singles = sum(1 for _, n in entries if n == 1)
        if singles < len(entries):
            ops.prefill_attention(*args, max_q, heads, kv_heads, d, scale, window=window, skip_single=singles > 0)
        if singles:
            ns, ch = splits or (None, None)
            ops.decode_attention(*args, heads, kv_heads, d, scale, max(lengths), window=window, num_splits=ns, chunk=ch,
                                 kernel="tma" if kernel == "tma" else "cp_async", error_word=err)
    assert int(err) == 0
    return out.cpu(), torch.cat(refs)


ATTN_SHAPES = [  # heads, kv_heads, d, page
    (4, 2, 16, 4), (6, 3, 32, 16), (5, 1, 48, 3), (7, 7, 80, 1), (8, 2, 128, 16), (32, 1, 64, 64), (2, 1, 256, 16),
    (14, 2, 96, 5)]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads, kv_heads, d, page", ATTN_SHAPES)
def test_paged_attention_ragged_batch(dtype, heads, kv_heads, d, page):
    need_gpu()
    entries = [(0, 70), (130, 1), (31, 2), (0, 1), (63, 33)]       # whole prompt, decode, tiny portion, first token, portion over block edges
    out, ref = attention_case(dtype, heads, kv_heads, d, page, entries)
    assert torch.isfinite(out).all()                              # NaN in unwritten slots must not leak
    assert torch.allclose(out.double(), ref, **(dict(atol=3e-6, rtol=1e-5) if dtype == torch.float32 else dict(atol=2e-2, rtol=2e-2)))


# (a portion in four rows a warp, single tokens in one row and, of groups above four, in four; heads of one, two, three and eight columns a lane)
@pytest.mark.parametrize("heads, kv_heads, d", [(4, 4, 32), (8, 2, 64), (10, 2, 72), (6, 1, 256)])
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("window", [0, 40])
def test_paged_attention_by_four_numbers_has_the_bits_of_single_ones(heads, kv_heads, d, dtype, window):
    need_gpu()
    from torchinferno_b200.kernels import ops
    i32 = lambda xs: dev(torch.tensor(xs, dtype=torch.int32))
    page, pages, contexts = 8, 40, [33, 64, 100]
    pool, table = dev(rnd(pages, 2, kv_heads, page, d, dtype=dtype)), i32(list(range(39))).view(3, 13)
    q = rnd(sum(contexts), heads * d, dtype=dtype, seed=3)

    def run(rows, starts, past, longest, shift):
        moved = torch.empty(rows.numel() + shift, dtype=dtype, device="cuda")[shift:].view(rows.shape)      # (rows off their boundaries: one number at a time)
        moved.copy_(rows)
        return ops.paged_attention_simt(moved, pool, torch.empty(rows.shape, dtype=dtype, device="cuda"), i32(starts), i32(past), i32([0, 1, 2]), table, 3, longest,
                                        heads, kv_heads, d, d ** -0.5, window=window)

    starts = [0] + [sum(contexts[:i + 1]) for i in range(3)]
    whole = run(dev(q), starts, [0, 0, 0], max(contexts), 0)
    assert torch.equal(whole, run(dev(q), starts, [0, 0, 0], max(contexts), 1))
    last = torch.tensor([e - 1 for e in starts[1:]])
    for shift in (0, 1):      # the last token of each alone: the bits it has in its portion
        assert torch.equal(run(dev(q[last]), [0, 1, 2, 3], [c - 1 for c in contexts], 1, shift), whole[last.cuda()])


@pytest.mark.parametrize("window", [1, 5, 32, 33, 100])
def test_paged_attention_window_edges(window):
    need_gpu()
    entries = [(0, 90), (200, 1), (95, 7)]
    out, ref = attention_case(torch.float32, 4, 2, 32, 16, entries, window=window, seed=3)
    assert torch.allclose(out.double(), ref, atol=3e-6, rtol=1e-5)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("standout", [0, 3, 511, 512, 700])
def test_paged_attention_finds_one_far_key_among_hundreds(dtype, standout):
    need_gpu()
    entries = [(900, 1), (640, 70)]
    out, ref = attention_case(dtype, 8, 2, 64, 16, entries, seed=5, standout=standout)
    assert ref.abs().max() > 3                                    # the far key really dominates the reference
    assert torch.allclose(out.double(), ref, **(dict(atol=2e-5, rtol=1e-5) if dtype == torch.float32 else dict(atol=6e-2, rtol=2e-2)))


def test_paged_attention_rows_do_not_depend_on_the_batch():
    need_gpu()
    alone, _ = attention_case(torch.float32, 6, 3, 32, 16, [(40, 9)], seed=9)
    # same request (same seed → same q, k, v for entry 0) with others beside it
    mixed, _ = attention_case(torch.float32, 6, 3, 32, 16, [(40, 9), (0, 50), (77, 1)], seed=9)
    assert torch.equal(alone, mixed[:9])


BF16_ATTN = dict(atol=2e-2, rtol=2e-2)
MMA_SHAPES = [(4, 2, 64, 16), (8, 2, 128, 16), (32, 8, 128, 16), (3, 1, 64, 4), (6, 6, 128, 1), (40, 2, 64, 5), (7, 1, 128, 64),
              # head sizes that do not fill the 64- or 128-wide tiles
              (5, 1, 48, 16), (4, 2, 80, 8), (6, 2, 96, 16), (3, 3, 112, 4), (4, 4, 16, 16), (8, 2, 32, 3)]


@pytest.mark.parametrize("heads, kv_heads, d, page", MMA_SHAPES)
@pytest.mark.parametrize("kernel", ["mma", "mma_prefill"])
def test_tensor_core_attention_ragged_batch(heads, kv_heads, d, page, kernel):
    need_gpu()
    # a whole prompt over several tiles, decodes at short and long contexts, portions that start and
    # end off the tile edges, a first token, a two-token portion
    entries = [(0, 150), (130, 1), (31, 2), (0, 1), (63, 66), (700, 1), (64, 1), (255, 129)]
    out, ref = attention_case(torch.bfloat16, heads, kv_heads, d, page, entries, kernel=kernel)
    assert torch.isfinite(out).all()
    assert torch.allclose(out.double(), ref, **BF16_ATTN), (out.double() - ref).abs().max()


TC_SHAPES = [(4, 2, 64, 16), (8, 2, 128, 16), (32, 8, 128, 16), (3, 1, 64, 8), (6, 6, 128, 32), (16, 2, 64, 64), (7, 1, 128, 128)]


@pytest.mark.parametrize("heads, kv_heads, d, page", TC_SHAPES)
def test_tcgen05_prefill_attention_ragged_batch(heads, kv_heads, d, page):
    need_gpu()
    entries = [(0, 150), (130, 1), (31, 2), (0, 1), (63, 66), (700, 1), (64, 1), (255, 129), (0, 300)]
    out, ref = attention_case(torch.bfloat16, heads, kv_heads, d, page, entries, kernel="tcgen05_prefill")
    assert torch.isfinite(out).all()
    assert torch.allclose(out.double(), ref, **BF16_ATTN), (out.double() - ref).abs().max()


@pytest.mark.parametrize("window", [1, 5, 128, 129, 200])
def test_tcgen05_prefill_attention_window_edges(window):
    need_gpu()
    entries = [(0, 190), (300, 1), (95, 70), (63, 1), (120, 140)]
    out, ref = attention_case(torch.bfloat16, 4, 2, 64, 16, entries, window=window, seed=3, kernel="tcgen05_prefill")
    assert torch.allclose(out.double(), ref, **BF16_ATTN), (out.double() - ref).abs().max()


@pytest.mark.parametrize("standout", [0, 3, 511, 512, 700])
def test_tcgen05_prefill_attention_finds_one_far_key(standout):
    need_gpu()
    entries = [(900, 1), (640, 70)]
    out, ref = attention_case(torch.bfloat16, 8, 2, 64, 16, entries, seed=5, standout=standout, kernel="tcgen05_prefill")
    assert ref.abs().max() > 3
    assert torch.allclose(out.double(), ref, atol=6e-2, rtol=2e-2)


@pytest.mark.parametrize("splits", [(1, 1024), (2, 512), (3, 320), (16, 64), (9, 128), (1, 0), (2, 0), (5, 0), (32, 0)])
def test_split_decode_attention_is_the_same_for_every_split(splits):
    need_gpu()
    entries = [(900, 1), (0, 1), (63, 1), (64, 1), (517, 1)]
    out, ref = attention_case(torch.bfloat16, 8, 2, 128, 16, entries, kernel="mma", splits=splits, seed=2)
    assert torch.allclose(out.double(), ref, **BF16_ATTN), (out.double() - ref).abs().max()


TMA_SHAPES = [(4, 2, 64, 16), (8, 2, 128, 16), (32, 8, 128, 16), (3, 1, 64, 8), (6, 6, 128, 32), (32, 2, 64, 64), (7, 1, 128, 8),
              (12, 4, 128, 64)]


@pytest.mark.parametrize("heads, kv_heads, d, page", TMA_SHAPES)
def test_tma_decode_attention_ragged_batch(heads, kv_heads, d, page):
    """Single tokens by the TMA kernel (portions beside them by the mma.sync prefill kernel): contexts of 1, 64, 65
    tokens, ones that end in the middle of a page and of a tile, and a long one."""
    need_gpu()
    entries = [(0, 150), (130, 1), (31, 2), (0, 1), (63, 1), (700, 1), (64, 1), (255, 129), (1000, 1), (15, 1), (16, 1), (127, 1)]
    out, ref = attention_case(torch.bfloat16, heads, kv_heads, d, page, entries, kernel="tma")
    assert torch.isfinite(out).all()
    assert torch.allclose(out.double(), ref, **BF16_ATTN), (out.double() - ref).abs().max()


@pytest.mark.parametrize("splits", [(1, 1024), (2, 512), (3, 320), (16, 64), (9, 128), (1, 0), (2, 0), (5, 0), (32, 0)])
def test_tma_decode_attention_is_the_same_for_every_split(splits):
    need_gpu()
    entries = [(900, 1), (0, 1), (63, 1), (64, 1), (517, 1)]
    out, ref = attention_case(torch.bfloat16, 8, 2, 128, 16, entries, kernel="tma", splits=splits, seed=2)
    assert torch.allclose(out.double(), ref, **BF16_ATTN), (out.double() - ref).abs().max()
    other, _ = attention_case(torch.bfloat16, 8, 2, 128, 16, entries, kernel="mma", splits=splits, seed=2)
    assert torch.allclose(out.float(), other.float(), atol=4e-3, rtol=1e-2)     # the two kernels do the same arithmetic


@pytest.mark.parametrize("window", [1, 5, 64, 65, 200])
def test_tma_decode_attention_window_edges(window):
    need_gpu()
    entries = [(300, 1), (63, 1), (64, 1), (199, 1), (200, 1), (1, 1), (777, 1)]
    out, ref = attention_case(torch.bfloat16, 4, 2, 64, 16, entries, window=window, seed=3, kernel="tma")
    assert torch.allclose(out.double(), ref, **BF16_ATTN), (out.double() - ref).abs().max()


@pytest.mark.parametrize("standout", [0, 3, 511, 512, 700])
def test_tma_decode_attention_finds_one_far_key(standout):
    need_gpu()
    entries = [(900, 1), (701, 1)]
    out, ref = attention_case(torch.bfloat16, 8, 2, 64, 16, entries, seed=5, standout=standout, kernel="tma")
    assert ref.abs().max() > 3
    assert torch.allclose(out.double(), ref, atol=6e-2, rtol=2e-2)


@pytest.mark.parametrize("heads, kv_heads, d, page, rot, inter", [(8, 2, 128, 16, 128, False), (4, 2, 64, 8, 64, False), (32, 8, 128, 16, 128, False),
                                                                  (6, 1, 64, 32, 32, True), (4, 4, 128, 64, 0, False), (3, 1, 64, 16, 48, False)])
def test_tma_decode_attention_that_rotates_and_stores_the_newest_token_itself(heads, kv_heads, d, page, rot, inter):
    """One kernel from the rows of the qkv product (rotary encoding of q and k, the write of k and v into their pages,
    attention) gives bit for bit what the rotary kernel followed by the attention kernel gives: the same output and
    the same pages, with contexts that end at the first and last slot of a page and of a tile, and with 1, 4 and 16
    context parts."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    contexts = [1, 2, 64, 65, 16, 17, 700, 128, 333, 1000]
    n = len(contexts)
    pool, table, slots = paged_layout(n, contexts, page, kv_heads, d, torch.bfloat16, seed=9)
    for e, c in enumerate(contexts):                                  # older keys and values; the newest slot stays NaN
        if c > 1:
            fill_pages(pool, table, slots[e], rnd(kv_heads, c - 1, d, dtype=torch.bfloat16, seed=e), rnd(kv_heads, c - 1, d, dtype=torch.bfloat16, seed=40 + e))
    qkv = rnd(n, (heads + 2 * kv_heads) * d, dtype=torch.bfloat16, seed=77)
    inv_freq = (1.0 / (10000.0 ** (torch.arange(0, rot, 2, dtype=torch.float32) / max(rot, 1)))) if rot else torch.zeros(0)
    i32 = lambda xs: dev(torch.tensor(xs, dtype=torch.int32))
    q_start, kv_start, slot_t, table_d = i32(list(range(n + 1))), i32([c - 1 for c in contexts]), i32(slots), dev(table)
    scale = 1.0 / math.sqrt(d)
    for splits in (1, 4, 16):
        pool_a, pool_b = dev(pool), dev(pool)
        q_rot = torch.empty(n, heads * d, dtype=torch.bfloat16, device="cuda")
        ops.rope_append(dev(qkv), q_rot, pool_a, kv_start, slot_t, table_d, dev(inv_freq), heads, kv_heads, d, rot_dim=rot, interleaved=inter)
        want = ops.decode_attention(q_rot, pool_a, torch.empty_like(q_rot), q_start, kv_start, slot_t, table_d, n, heads, kv_heads, d,
                                    scale, max(contexts), num_splits=splits, chunk=0, kernel="tma")
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        got = ops.decode_attention_rope(dev(qkv), pool_b, torch.full_like(q_rot, float("nan")), q_start, kv_start, slot_t, table_d, n,
                                        heads, kv_heads, d, scale, max(contexts), dev(inv_freq), rot_dim=rot, interleaved=inter,
                                        num_splits=splits, error_word=err)
        torch.cuda.synchronize()
        assert int(err) == 0 and torch.isfinite(got).all()
        assert torch.equal(got, want), (splits, (got.float() - want.float()).abs().max())
        a, b = pool_a.cpu(), pool_b.cpu()
        assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))
    bad = table.clone()
    bad[slots[6], 699 // page] = pool.shape[0] + 3                    # a page id outside the pool is reported, not written
    ops.decode_attention_rope(dev(qkv), dev(pool), torch.empty_like(q_rot), q_start, kv_start, slot_t, dev(bad), n, heads, kv_heads, d,
                              scale, max(contexts), dev(inv_freq), rot_dim=rot, interleaved=inter, error_word=err)
    assert int(err) != 0


def test_tma_decode_attention_refuses_other_shapes():
    need_gpu()
    from torchinferno_b200.kernels import ops
    assert not ops.decode_attention_tma_supports(96, 4, 16) and not ops.decode_attention_tma_supports(128, 32, 16)
    assert not ops.decode_attention_tma_supports(128, 4, 5) and not ops.decode_attention_tma_supports(128, 4, 128)
    with pytest.raises(ops.KernelError, match="does not take this shape"):
        attention_case(torch.bfloat16, 4, 2, 64, 4, [(10, 1)], kernel="tma")


@pytest.mark.parametrize("window", [1, 5, 64, 65, 200])
@pytest.mark.parametrize("kernel", ["mma", "mma_prefill"])
def test_tensor_core_attention_window_edges(window, kernel):
    need_gpu()
    entries = [(0, 190), (300, 1), (95, 70), (63, 1)]
    out, ref = attention_case(torch.bfloat16, 4, 2, 64, 16, entries, window=window, seed=3, kernel=kernel)
    assert torch.allclose(out.double(), ref, **BF16_ATTN), (out.double() - ref).abs().max()


@pytest.mark.parametrize("standout", [0, 3, 511, 512, 700])
def test_tensor_core_attention_finds_one_far_key_among_hundreds(standout):
    need_gpu()
    entries = [(900, 1), (640, 70)]
    out, ref = attention_case(torch.bfloat16, 8, 2, 64, 16, entries, seed=5, standout=standout, kernel="mma")
    assert ref.abs().max() > 3
    assert torch.allclose(out.double(), ref, atol=6e-2, rtol=2e-2)


def test_attention_refuses_what_it_cannot_do():
    need_gpu()
    from torchinferno_b200.kernels import ops
    i32 = lambda xs: dev(torch.tensor(xs, dtype=torch.int32))

    def call(heads, kv_heads, d):
        q = torch.zeros(4, heads * d, device="cuda")
        pool = torch.zeros(2, 2, kv_heads, 16, d, device="cuda")
        ops.paged_attention_simt(q, pool, torch.empty_like(q), i32([0, 4]), i32([0]), i32([0]), i32([[0, 1]]), 1, 4,
                                 heads, kv_heads, d, 1.0)

    call(4, 2, 256)
    with pytest.raises(ops.KernelError, match="size"):
        call(4, 2, 272)                                             # head size above 256
    with pytest.raises(ops.KernelError, match="size"):
        call(5, 2, 32)                                              # heads not a multiple of kv heads
    with pytest.raises(ops.KernelError, match="CUDA tensor"):
        ops.swiglu(torch.zeros(2, 4), torch.zeros(2, 2))            # no CPU path
    assert ops.attention_mma_supports(128, 4) and ops.attention_mma_supports(48, 4)
    assert not ops.attention_mma_supports(40, 4) and not ops.attention_mma_supports(144, 4)
    q = torch.zeros(4, 4 * 144, device="cuda", dtype=torch.bfloat16)
    pool = torch.zeros(2, 2, 2, 16, 144, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(ops.KernelError, match="size"):              # the tensor-core kernels take steps of 16 up to 128
        ops.prefill_attention(q, pool, torch.empty_like(q), i32([0, 4]), i32([0]), i32([0]), i32([[0, 1]]), 1, 4, 4, 2, 144, 1.0)


# --------------------------------------------------------------- sampling
def test_greedy_takes_the_lowest_index_among_maxima_and_nan_wins():
    need_gpu()
    from torchinferno_b200.kernels import ops
    logits = rnd(5, 3001)
    logits[0, 77] = logits[0, 2900] = 9.0
    logits[1, 3000] = 50.0
    logits[2, 1500] = float("nan")
    logits[3] = -float("inf")
    out = ops.sample(dev(logits), torch.empty(5, dtype=torch.int32, device="cuda")).cpu()
    assert out.tolist()[:4] == [77, 3000, 1500, 0] and out[4] == int(torch.argmax(logits[4]))


@pytest.mark.parametrize("vocab", [17, 1000, 128256])
def test_temperature_sampling_is_the_seeded_gumbel_max(vocab):
    need_gpu()
    from torchinferno_b200.kernels import ops
    logits = rnd(4, vocab, scale=2)
    temps, seeds, pos = [0.8, 1.5, 0.0, 0.3], [1, 2 ** 40 + 5, 3, -9], [0, 17, 5, 100000]
    i64 = torch.tensor(seeds, dtype=torch.int64)
    out = ops.sample(dev(logits), torch.empty(4, dtype=torch.int32, device="cuda"), dev(torch.tensor(temps)),
                     dev(i64), dev(torch.tensor(pos, dtype=torch.int32))).cpu().tolist()
    for r in range(4):
        if temps[r] == 0:
            assert out[r] == int(torch.argmax(logits[r]))
            continue
        scores = plain_llama.gumbel_scores(logits[r].numpy(), temps[r], seeds[r], pos[r])
        assert scores[out[r]] >= scores.max() - 1e-4        # the argmax, up to float rounding of near-ties
    # what else is in the batch does not matter
    alone = ops.sample(dev(logits[1:2].contiguous()), torch.empty(1, dtype=torch.int32, device="cuda"),
                       dev(torch.tensor(temps[1:2])), dev(i64[1:2].contiguous()), dev(torch.tensor(pos[1:2], dtype=torch.int32))).cpu()
    assert int(alone) == out[1]


def test_temperature_sampling_draws_from_the_softmax():
    need_gpu()
    from torchinferno_b200.kernels import ops
    logits = torch.tensor([[2.0, 1.0, 0.0, -1.0, 0.5]]).repeat(20000, 1)
    temp = 0.7
    out = ops.sample(dev(logits), torch.empty(20000, dtype=torch.int32, device="cuda"), dev(torch.full((20000,), temp)),
                     dev(torch.arange(20000, dtype=torch.int64)), dev(torch.zeros(20000, dtype=torch.int32))).cpu()
    freq = torch.bincount(out.long(), minlength=5).double() / 20000
    want = torch.softmax(logits[0].double() / temp, dim=0)
    assert (freq - want).abs().max() < 0.012


def test_the_library_plans_attention_and_products_for_both_ways_of_running_a_block():
    """`tib_plan_attention` and `tib_plan_product` are where the kernels of a step are chosen, for the parts and for
    the native block call: their answers on the shapes the engine meets."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    every = ops.ALLOW_PREFILL_TCGEN05 | ops.ALLOW_DECODE_ROTATES | ops.ALLOW_DECODE_TMA
    plan = ops.plan_attention
    # heads of 128 in groups of 4, pages of 16 back to back
    assert plan(128, 4, 16, True, 8, 8, 0, every) == (ops.ATTENTION_NONE, ops.ATTENTION_DECODE_TMA_ROTATES)
    assert plan(128, 4, 16, True, 9, 9, 0, every) == (ops.ATTENTION_NONE, ops.ATTENTION_DECODE_TMA)           # many requests
    assert plan(128, 4, 16, True, 8, 7, 1, every) == (ops.ATTENTION_PREFILL_TCGEN05, ops.ATTENTION_DECODE_TMA)  # a portion among them
    assert plan(128, 4, 16, True, 8, 8, 0, every & ~ops.ALLOW_DECODE_ROTATES)[1] == ops.ATTENTION_DECODE_TMA
    assert plan(128, 4, 16, False, 8, 7, 1, every) == (ops.ATTENTION_PREFILL_MMA, ops.ATTENTION_DECODE_CP_ASYNC)  # pages not back to back
    assert plan(128, 4, 16, True, 2, 0, 2, every & ~ops.ALLOW_PREFILL_TCGEN05) == (ops.ATTENTION_PREFILL_MMA, ops.ATTENTION_NONE)
    assert plan(128, 4, 3, True, 2, 1, 1, every) == (ops.ATTENTION_PREFILL_MMA, ops.ATTENTION_DECODE_CP_ASYNC)   # pages of 3 tokens
    assert plan(80, 4, 16, True, 2, 1, 1, every) == (ops.ATTENTION_PREFILL_MMA, ops.ATTENTION_DECODE_CP_ASYNC)   # heads of 80
    assert plan(72, 4, 16, True, 2, 1, 1, every) == (ops.ATTENTION_SIMT, ops.ATTENTION_SIMT)                     # heads of 72
    product = ops.plan_product
    assert product(8, 4096, 4096, True, 64, 128, 4, False, True) == ops.PRODUCT_DECODE
    assert product(8, 4096, 4096, True, 4, 128, 4, False, True) == ops.PRODUCT_LIBRARY      # more rows than the weight's bound
    assert product(8, 4096, 4096, True, 64, 128, 4, False, False) == ops.PRODUCT_LIBRARY    # operands not aligned
    assert product(8, 4096, 4096, True, 64, 128, 0, False, True) == ops.PRODUCT_SWAPAB      # no K split chosen: the older kernel
    assert product(8, 4096, 4096, False, 64, 128, 4, False, True) == ops.PRODUCT_SWAPAB     # [out, in] weights
    assert product(8, 28672, 4096, True, 64, 256, 1, True, True) == ops.PRODUCT_DECODE
    assert product(8, 28672, 4096, True, 64, 128, 2, True, True) != ops.PRODUCT_DECODE      # the activation only unsplit
    assert product(0, 4096, 4096, True, 64, 128, 4, False, True) == ops.PRODUCT_LIBRARY


def test_attention_kernels_on_random_shapes_and_batches():
    """Eighty draws of a random search over the attention kernels: head sizes, numbers of heads and groups, page
    sizes, windows, forced splits and ragged batches that no list in this file names, each against the float64
    plain attention; a shape a kernel does not take is passed over."""
    need_gpu()
    import random
    from torchinferno_b200.kernels import ops
    ran = {}
    for draw in range(80):
        rng = random.Random(77000 + draw)
        kernel = rng.choice(["simt32", "simt16", "mma", "mma_prefill", "tcgen05_prefill", "tma"])
        kv = rng.randint(1, 4)
        if kernel.startswith("simt"):
            d, group, page = rng.choice([8, 16, 24, 40, 64, 72, 96, 128, 160, 256]), rng.randint(1, 9), rng.choice([1, 2, 3, 4, 5, 8, 16, 32, 64])
        elif kernel in ("mma", "mma_prefill"):
            d, group = rng.choice([16, 32, 48, 64, 80, 96, 112, 128]), rng.choice([1, 2, 3, 4, 5, 7, 8, 12, 16, 20, 33, 64])
            page = rng.choice([1, 2, 3, 4, 5, 8, 16, 32, 64])
            if not ops.attention_mma_supports(d, group):
                continue
        else:
            d, group = rng.choice([64, 128]), rng.choice([1, 2, 3, 4, 5, 7, 8, 12, 16])
            page = rng.choice([8, 16, 32, 64, 128] if kernel == "tcgen05_prefill" else [8, 16, 32, 64])
            takes = ops.prefill_attention_tcgen05_supports if kernel == "tcgen05_prefill" else ops.decode_attention_tma_supports
            if not takes(d, group, page):
                continue
        heads = kv * group
        if heads * d > 8192:
            continue
        entries = []
        for _ in range(rng.randint(1, 6)):
            r = rng.random()
            entries.append((rng.randint(0, 900), 1) if r < 0.35 else (0, rng.randint(1, 300)) if r < 0.5 else
                           (rng.randint(0, 500), rng.randint(2, 200)))
        window = rng.choice([0, 0, 0, 1, 7, 64, 65, 130, 400])
        splits = (rng.choice([1, 2, 3, 5, 8, 16, 32]), 0) if kernel in ("mma", "tma") and rng.random() < 0.5 else None
        dtype = torch.float32 if kernel == "simt32" else torch.bfloat16
        out, ref = attention_case(dtype, heads, kv, d, page, entries, window=window, seed=draw,
                                  kernel="simt" if kernel.startswith("simt") else kernel, splits=splits)
        what = (draw, kernel, heads, kv, d, page, window, splits, entries)
        assert torch.isfinite(out).all(), what
        assert torch.allclose(out.double(), ref, **(dict(atol=3e-6, rtol=1e-5) if dtype == torch.float32 else BF16_ATTN)), what
        ran[kernel] = ran.get(kernel, 0) + 1
    assert len(ran) == 6 and min(ran.values()) >= 5, ran


def test_product_kernels_on_random_shapes():
    """Two hundred draws of a random search over the product kernels (the two tcgen05 kernels for many rows, the two
    for few rows with either weight layout, tile width, K split, ring depth and the SwiGLU epilogue, the library in
    both layouts, the 32-bit kernel), each against float64; NaN in the output beforehand shows what was not written."""
    need_gpu()
    import random
    from torchinferno_b200.kernels import ops
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    ran = {}
    for draw in range(200):
        rng = random.Random(31000 + draw)
        kind = rng.choice(["tcgen05", "2cta", "swapab", "swapab_kn", "decode", "decode_swiglu", "library", "library_kn", "f32"])
        g = torch.Generator().manual_seed(draw)
        few = kind in ("swapab", "swapab_kn", "decode", "decode_swiglu")
        m = rng.randint(1, 64) if few else rng.choice([1, 2, 7, 64, 100, 129, 256, 300, 513, 1000])
        n = rng.choice([8, 16, 24, 64, 72, 128, 136, 200, 256, 264, 512, 1000, 1024, 3072, 4104])
        k = rng.choice([64, 128, 192, 256, 320, 1024, 2048, 4096])
        out_dtype = rng.choice([torch.bfloat16, torch.float32])
        blank = lambda width, dtype: torch.full((m, width), float("nan"), dtype=dtype, device="cuda")
        if kind == "f32":
            n, k = rng.choice([1, 3, 64, 67, 129, 500]), rng.choice([1, 7, 64, 100, 257, 1000])
            x, w = torch.randn(m, k, generator=g).cuda(), torch.randn(n, k, generator=g).cuda()
            out, want, rel = ops.gemm_f32(x, w, blank(n, torch.float32)), as_ref(x) @ as_ref(w).T, 1e-5
        else:
            x = torch.randn(m, k, generator=g).to(torch.bfloat16).cuda()
            kn = kind in ("swapab_kn", "decode", "decode_swiglu", "library_kn")
            w = (torch.randn((k, n) if kn else (n, k), generator=g) * 0.05).to(torch.bfloat16).cuda()
            want = as_ref(x) @ (as_ref(w) if kn else as_ref(w).T)
            if kind in ("decode", "decode_swiglu"):
                features = rng.choice([128, 256])
                splits = rng.randint(1, 8) if features == 128 and kind == "decode" else 1
                epilogue = ops.DG_SWIGLU if kind == "decode_swiglu" else ops.DG_PLAIN
                if not ops.gemm_decode_supports(m, n, k, features, splits, epilogue):
                    continue
                if epilogue == ops.DG_SWIGLU:
                    want, out_dtype = want[:, 0::2] / (1 + torch.exp(-want[:, 0::2])) * want[:, 1::2], torch.bfloat16
                out = ops.gemm_decode(x, w, blank(want.shape[1], out_dtype), features=features, splits=splits, epilogue=epilogue,
                                      stages=rng.choice([0, 0, 1, 2, 3, 5, 9, 16]), error_word=err)
            elif kind in ("swapab", "swapab_kn"):
                if not ops.gemm_tcgen05_swapab_supports(m, n, k):
                    continue
                out = ops.gemm_tcgen05_swapab(x, w, blank(n, out_dtype), err, w_kn=kn)
            elif kind in ("library", "library_kn"):
                out = ops.library_gemm(x, w, blank(n, out_dtype), w_kn=kn)
            elif kind == "tcgen05":
                if not ops.gemm_tcgen05_supports(m, n, k):
                    continue
                out = ops.gemm_tcgen05(x, w, blank(n, out_dtype), err)
            else:
                if not ops.gemm_tcgen05_2cta_supports(m, n, k):
                    continue
                out = ops.gemm_tcgen05_2cta(x, w, blank(n, out_dtype), err)
            rel = 1.2e-2 if out.dtype == torch.bfloat16 else 2e-4
        what = (draw, kind, m, n, k, out.dtype)
        assert torch.isfinite(out).all(), what
        assert (as_ref(out) - want).abs().max() <= rel * want.abs().max() + 1e-6, what
        assert int(err) == 0, what
        ran[kind] = ran.get(kind, 0) + 1
    assert len(ran) == 9 and min(ran.values()) >= 5, ran


@pytest.mark.parametrize("m, n, k", [(1, 33, 4), (16, 48, 20), (40, 130, 64), (200, 1000, 100), (700, 2100, 36), (130, 4100, 2052)])
def test_aligned_fp32_product_has_the_plain_kernels_bits(m, n, k):
    need_gpu()
    from torchinferno_b200.kernels import ops
    x, w = dev(rnd(m, k, scale=2)), dev(rnd(n, k, seed=3))
    wide = torch.empty(m, k + 1, device="cuda")[:, :k]      # (rows off their 16-byte boundaries: the plain kernel)
    wide.copy_(x)
    plain = ops.gemm_f32(wide, w, torch.empty(m, n, device="cuda"))
    assert torch.equal(ops.gemm_f32(x, w, torch.empty(m, n, device="cuda")), plain)


# (edges of the tiles: 128 features, 16 to 80 rows, 64 k a step and 128 a sum)
@pytest.mark.parametrize("m, n, k", [(1, 8192, 512), (16, 7297, 576), (17, 512, 8192), (80, 6560, 640), (81, 2000, 2112), (161, 4100, 1024), (330, 7400, 576), (2600, 2050, 4160)])
def test_fp32_product_in_three_terms(m, n, k, monkeypatch):
    need_gpu()
    from torchinferno_b200.kernels import ops
    x, w = dev(rnd(m, k, scale=2)), dev(rnd(n, k, seed=3))
    error = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = ops.gemm_f32(x, w, torch.empty(m, n, device="cuda"), error)
    # The tensor core cuts off at most 2^-23 of a sum at each of the eight instructions over 128 k, the sums of those are added in
    # fp32, and the terms left out are below 2 * 2^-24 of a product: 2^-23 (8 + k / 256 + 1) of the products' magnitudes, and one for the small terms.
    bound = 2.0 ** -23 * (10 + k / 256) * (x.double().abs() @ w.double().abs().T)
    assert ((out.double() - x.double() @ w.double().T).abs() <= bound).all() and int(error) == 0
    # Seen: 1.4e-7 to 2.4e-7 of the result's 2-norm.  Without one of the three small groups of products it would be 1.3e-6 (a1 b1: two numbers of 2^-9
    # of theirs, evenly spread) or 2.5e-6 (a2 b0, a0 b2: one of 2^-17) or more.
    exact = x.double() @ w.double().T
    assert (out.double() - exact).norm() <= 4e-7 * exact.norm()
    for rows in (slice(m // 2, m // 2 + 1), slice(0, max(1, m - 3))):      # a row does not depend on the rows beside it
        few = x[rows].contiguous()
        assert torch.equal(ops.gemm_f32(few, w, torch.empty(len(few), n, device="cuda")), out[rows])
    monkeypatch.setattr(ops, "F32_TERMS_BYTES", 1)                         # 128 rows at a time, into a wider matrix
    wide = torch.zeros(m, n + 3, device="cuda")
    ops.gemm_f32(x, w, wide[:, :n])
    assert torch.equal(wide[:, :n], out) and not wide[:, n:].any()
    # infinities, NaN and numbers that no bf16 number reaches come out as in multiply-adds
    x[0, 5], w[3, 9], w[7, 100], x[m - 1, k - 1] = math.inf, math.nan, -math.inf, 3.4e38
    odd = torch.empty(m, k + 1, device="cuda")[:, :k]                      # (rows off their 16-byte boundaries: the plain kernel)
    odd.copy_(x)
    out, plain = (ops.gemm_f32(t, w, torch.empty(m, n, device="cuda")) for t in (x, odd))
    assert torch.equal(out.isnan(), plain.isnan()) and torch.equal(out.isinf(), plain.isinf()) and not torch.isfinite(out[:, 7]).any()


def test_calls_of_different_sizes_from_several_threads():
    """The shared memory that a kernel may take is the function's, not the thread's: one kernel at several sizes from several threads at once."""
    need_gpu()
    import threading
    from torchinferno_b200.kernels import ops
    w = dev(rnd(2048, 2048))
    heads, dim = 4, 128
    chunk = ops.linear_attention_chunk(dim, dim)
    powers = dev((torch.tensor([0.9] * heads, dtype=torch.float64)[:, None] ** torch.arange(chunk + 1, dtype=torch.float64)).float().contiguous())

    def product(m):
        x = dev(rnd(m, 2048, seed=m))
        return lambda: ops.gemm_f32(x, w, torch.empty(m, 2048, device="cuda"))

    def linear(entries):      # (a block's columns, and its shared memory, go by the number of portions)
        n = 40 * entries
        rows, state = dev(rnd(n, 3 * heads * dim, seed=entries)), dev(rnd(entries, heads, dim, dim))
        starts, slots = dev(40 * torch.arange(entries + 1, dtype=torch.int32)), dev(torch.arange(entries, dtype=torch.int32))
        q, k, v = rows.chunk(3, 1)
        return lambda: ops.linear_attention(q, k, v, torch.empty(n, heads * dim, device="cuda"), state.clone(), powers, starts, slots, entries, heads, dim, dim,
                                            silu=True, max_q_len=40)

    calls = [product(m) for m in (8, 48, 80, 300)] + [linear(entries) for entries in (8, 40)]
    want, faults = [call() for call in calls], []
    torch.cuda.synchronize()

    def work(call, ref):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(300):
                    out = call()
                assert torch.equal(out, ref)
        except Exception as error:
            faults.append(error)

    threads = [threading.Thread(target=work, args=pair) for pair in zip(calls, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not faults, faults


def test_fp32_products_of_expanded_weights():
    """One row of weights for all features, and rows that overlap: what the kernel on multiply-adds makes of them."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    x, row = dev(rnd(5, 2048)), dev(rnd(2048 + 4 * 2047))
    for w in (row[:2048].expand(2048, 2048), row.as_strided((2048, 2048), (4, 1))):
        out = ops.gemm_f32(x, w, torch.empty(5, 2048, device="cuda"))
        assert torch.equal(out[:, :512], ops.gemm_f32(x, w[:512].contiguous(), torch.empty(5, 512, device="cuda")))


# ------------------------------------------------- linear attention in runs and token by token
@pytest.mark.parametrize("lens, heads, key_dim, value_dim", [
    ([1, 1, 1], 3, 128, 128), ([32, 5, 9], 2, 64, 96),                        # token by token, to its longest portion
    ([33, 1, 64], 2, 128, 64), ([192, 7], 2, 64, 64),                                           # in chunks, to their longest portion
    ([193, 1, 64], 2, 128, 64), ([257, 128, 127, 2], 2, 64, 128), ([200, 63], 3, 128, 128)])    # in runs and at their edges
@pytest.mark.parametrize("dtype", DTYPES)
def test_linear_attention_forms_agree_with_the_recurrence(lens, heads, key_dim, value_dim, dtype):
    need_gpu()
    from torchinferno_b200.kernels import ops
    n, entries = sum(lens), len(lens)
    rows = rnd(n, heads * (2 * key_dim + value_dim) + 8, dtype=dtype)
    decay = torch.tensor([1 - 2.0 ** -(3 + i) for i in range(heads)], dtype=torch.float64)
    state = rnd(entries + 1, heads, key_dim, value_dim, seed=5)
    slots = [entries - i for i in range(entries)]

    def powers(most):
        return dev((decay[:, None] ** torch.arange(most + 1, dtype=torch.float64)).float().contiguous())

    starts = torch.tensor([sum(lens[:i]) for i in range(entries + 1)], dtype=torch.int32)
    proj, got_state = dev(rows), dev(state.clone())
    qk = heads * key_dim
    out = ops.linear_attention(proj[:, :qk], proj[:, qk:2 * qk], proj[:, 2 * qk:2 * qk + heads * value_dim],
                               torch.empty(n, heads * value_dim, device="cuda"), got_state,
                               powers(ops.linear_attention_chunk(key_dim, value_dim)), dev(starts),
                               dev(torch.tensor(slots, dtype=torch.int32)), entries, heads, key_dim, value_dim, silu=True,
                               max_q_len=max(lens), run_powers=powers(ops.linear_attention_run()))
    x = rows.double()
    act = x * torch.sigmoid(x)
    q, k = act[:, :qk].view(n, heads, key_dim), act[:, qk:2 * qk].view(n, heads, key_dim)
    v = act[:, 2 * qk:2 * qk + heads * value_dim].view(n, heads, value_dim)
    want, want_state = torch.empty(n, heads, value_dim, dtype=torch.float64), state.double().clone()
    for e, length in enumerate(lens):
        s = want_state[slots[e]].clone()
        for t in range(int(starts[e]), int(starts[e]) + length):
            s = decay[:, None, None] * s + k[t][:, :, None] * v[t][:, None, :]
            want[t] = torch.einsum("hkv,hk->hv", s, q[t])
        want_state[slots[e]] = s
    # Walk and chunks round every product of key_dim + 32 once (2^-24 of the sum).  In runs every number enters with 24 bits, what is left out of a product is
    # below 2^-24 of it, and the tensor core cuts off at most 2^-23 of a sum at each of an accumulator's 8 instructions; the last sums are fp32.  2e-6 is
    # 16 such cuts of the largest value.
    assert (as_ref(out) - want.reshape(n, -1)).abs().max() <= 2e-6 * want.abs().max()
    assert (as_ref(got_state) - want_state).abs().max() <= 2e-6 * want_state.abs().max()


@pytest.mark.parametrize("dim, value_dim", [(64, 64), (128, 128), (128, 32), (64, 40)])
@pytest.mark.parametrize("dtype", DTYPES)
def test_linear_attention_of_a_request_does_not_depend_on_its_neighbours(dim, value_dim, dtype):
    """Portions of every form, alone and in one step, bit for bit; and the launches counted are those of the forms that occur."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    lens, heads = [1, 400, 40, 1, 192, 32, 193, 2], 2
    n, entries, widths = sum(lens), len(lens), [heads * dim, heads * dim, heads * value_dim]
    decay = torch.tensor([0.9, 0.99], dtype=torch.float64)
    powers = [dev((decay[:, None] ** torch.arange(most + 1, dtype=torch.float64)).float().contiguous())
              for most in (ops.linear_attention_chunk(dim, value_dim), ops.linear_attention_run())]
    q, k, v = (dev(rnd(n, w, dtype=dtype, seed=i)) for i, w in enumerate(widths))
    held, slots = dev(rnd(entries, heads, dim, value_dim, seed=5)), dev(torch.arange(entries, dtype=torch.int32))

    def run(first, count, portions):
        rows, part = slice(sum(lens[:first]), sum(lens[:first + count])), lens[first:first + count]
        state, before = held.clone(), ops.launch_count()
        starts = dev(torch.tensor([sum(part[:i]) for i in range(count + 1)], dtype=torch.int32))
        out = ops.linear_attention(q[rows], k[rows], v[rows], torch.empty(sum(part), widths[2], device="cuda"), state, powers[0], starts,
                                   slots[first:first + count].contiguous(), count, heads, dim, value_dim, silu=True, max_q_len=max(part),
                                   run_powers=powers[1], portions={m: part.count(m) for m in part} if portions else None)
        return out, state, ops.launch_count() - before

    out, state, launches = run(0, entries, True)
    out_unnamed, state_unnamed, _ = run(0, entries, False)
    assert torch.equal(out, out_unnamed) and torch.equal(state, state_unnamed)
    new_forms, runs_from = value_dim % 32 == 0, ops.linear_attention_forms(dim, value_dim)[1]
    assert launches == (1 if not new_forms else 5 if value_dim % 64 == 0 else 2)
    for i, m in enumerate(lens):
        alone, alone_state, launches = run(i, 1, True)
        assert torch.equal(alone, out[sum(lens[:i]):sum(lens[:i + 1])]) and torch.equal(alone_state[i], state[i]), (i, m)
        assert launches == (3 if m >= runs_from and value_dim % 64 == 0 else 1)


def test_linear_attention_in_runs_has_the_same_bits_in_tiles_of_either_width():
    """Few runs go in tiles of 64 value columns, many in tiles of 128: a request alone and among others that make the step choose the other."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    heads, dim, lens = 8, 128, [385, 200, 900, 700]
    n, width, entries = sum(lens), heads * dim, len(lens)
    decay = torch.tensor([1 - 2.0 ** -(3 + i % 6) for i in range(heads)], dtype=torch.float64)
    powers = [dev((decay[:, None] ** torch.arange(most + 1, dtype=torch.float64)).float().contiguous())
              for most in (ops.linear_attention_chunk(dim, dim), ops.linear_attention_run())]
    rows, held = dev(rnd(n, 3 * width, dtype=torch.bfloat16)), dev(rnd(entries, heads, dim, dim, seed=5))

    def run(first, count):
        part = lens[first:first + count]
        own, state = rows[sum(lens[:first]):sum(lens[:first + count])], held[first:first + count].clone()
        starts = dev(torch.tensor([sum(part[:i]) for i in range(count + 1)], dtype=torch.int32))
        out = ops.linear_attention(own[:, :width], own[:, width:2 * width], own[:, 2 * width:], torch.empty(len(own), width, device="cuda"), state, powers[0],
                                   starts, dev(torch.arange(count, dtype=torch.int32)), count, heads, dim, dim, silu=True, max_q_len=max(part),
                                   run_powers=powers[1], portions={m: 1 for m in part})
        return out, state

    out, state = run(0, entries)
    for i in range(entries):
        alone, alone_state = run(i, 1)
        assert torch.equal(alone, out[sum(lens[:i]):sum(lens[:i + 1])]) and torch.equal(alone_state[0], state[i])


@pytest.mark.parametrize("key_dim", [64, 128])
@pytest.mark.parametrize("dtype", DTYPES)
def test_linear_attention_in_runs_in_tiles_of_128_columns(key_dim, dtype):
    """Enough runs and heads that the step takes its value columns 128 at a time (more than 74 tiles)."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    heads, value_dim, lens = 12, 128, [450, 200, 130]
    n, entries, qk = sum(lens), len(lens), heads * key_dim
    rows, decay = rnd(n, 2 * qk + heads * value_dim, dtype=dtype), torch.tensor([1 - 2.0 ** -(3 + i % 6) for i in range(heads)], dtype=torch.float64)
    state, starts = rnd(entries, heads, key_dim, value_dim, seed=5), [sum(lens[:i]) for i in range(entries + 1)]
    powers = [dev((decay[:, None] ** torch.arange(most + 1, dtype=torch.float64)).float().contiguous())
              for most in (ops.linear_attention_chunk(key_dim, value_dim), ops.linear_attention_run())]
    proj, got_state = dev(rows), dev(state.clone())
    out = ops.linear_attention(proj[:, :qk], proj[:, qk:2 * qk], proj[:, 2 * qk:], torch.empty(n, heads * value_dim, device="cuda"), got_state, powers[0],
                               dev(torch.tensor(starts, dtype=torch.int32)), dev(torch.arange(entries, dtype=torch.int32)), entries, heads, key_dim, value_dim,
                               silu=True, max_q_len=max(lens), run_powers=powers[1])
    act = rows.double() * torch.sigmoid(rows.double())
    q, k, v = act[:, :qk].view(n, heads, -1), act[:, qk:2 * qk].view(n, heads, -1), act[:, 2 * qk:].view(n, heads, -1)
    want, want_state = torch.empty(n, heads, value_dim, dtype=torch.float64), state.double()
    for e, length in enumerate(lens):
        s = want_state[e]
        for t in range(starts[e], starts[e] + length):
            s = decay[:, None, None] * s + k[t][:, :, None] * v[t][:, None, :]
            want[t] = torch.einsum("hkv,hk->hv", s, q[t])
        want_state[e] = s
    assert (as_ref(out) - want.reshape(n, -1)).abs().max() <= 2e-6 * want.abs().max()
    assert (as_ref(got_state) - want_state).abs().max() <= 2e-6 * want_state.abs().max()


@pytest.mark.parametrize("at_a_time", [1, 2, 3])
def test_linear_attention_in_runs_some_heads_at_a_time(at_a_time, monkeypatch):
    """With less room for the runs' states than all heads take, the same bits and no more room than that."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    lens, heads, dim = [300, 1, 200], 5, 128
    n, entries, width = sum(lens), len(lens), heads * dim
    decay = torch.tensor([1 - 2.0 ** -(3 + i) for i in range(heads)], dtype=torch.float64)
    powers = [dev((decay[:, None] ** torch.arange(most + 1, dtype=torch.float64)).float().contiguous())
              for most in (ops.linear_attention_chunk(dim, dim), ops.linear_attention_run())]
    rows, held = dev(rnd(n, 3 * width, dtype=torch.bfloat16)), dev(rnd(entries, heads, dim, dim, seed=5))
    starts, slots = dev(torch.tensor([0, 300, 301, 501], dtype=torch.int32)), dev(torch.arange(entries, dtype=torch.int32))

    def run():
        out, state = torch.empty(n, width, device="cuda"), held.clone()
        torch.cuda.reset_peak_memory_stats()
        before, launches = torch.cuda.memory_allocated(), ops.launch_count()
        ops.linear_attention(rows[:, :width], rows[:, width:2 * width], rows[:, 2 * width:], out, state, powers[0], starts, slots, entries, heads, dim,
                             dim, silu=True, max_q_len=max(lens), run_powers=powers[1], portions={300: 1, 1: 1, 200: 1})
        return out, state, torch.cuda.max_memory_allocated() - before, ops.launch_count() - launches

    out, state, _, launches = run()
    assert launches == 1 + 3
    per_head = (n // ops.linear_attention_run() + entries) * dim * dim * 4
    monkeypatch.setattr(ops, "LINEAR_ATTENTION_SCRATCH", at_a_time * per_head + 5)
    parts, parts_state, room, launches = run()
    assert torch.equal(parts, out) and torch.equal(parts_state, state)
    assert room <= at_a_time * per_head + 2 ** 20 and launches == 1 + 3 * -(-heads // at_a_time)      # (the allocator's granularity)


@pytest.mark.parametrize("lens, dim", [([400, 7, 385], 64), ([200, 450], 128), ([100, 20], 64)])      # (in runs, and in chunks)
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_linear_attention_keeps_what_is_not_finite_from_earlier_tokens(lens, dim, bad):
    """One value of one request: only its own column of its head changes, from its own token on.  One key: only its head."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    n, heads, entries = sum(lens), 2, len(lens)
    width = heads * dim
    starts = [sum(lens[:i]) for i in range(entries + 1)]
    decay = torch.tensor([0.9, 0.99], dtype=torch.float64)
    powers = [dev((decay[:, None] ** torch.arange(most + 1, dtype=torch.float64)).float().contiguous())
              for most in (ops.linear_attention_chunk(dim, dim), ops.linear_attention_run())]
    rows, held = rnd(n, 3 * width, dtype=torch.bfloat16), rnd(entries, heads, dim, dim, seed=5)

    def run(rows):
        proj, state = dev(rows), dev(held.clone())
        out = ops.linear_attention(proj[:, :width], proj[:, width:2 * width], proj[:, 2 * width:], torch.empty(n, width, device="cuda"), state,
                                   powers[0], dev(torch.tensor(starts, dtype=torch.int32)), dev(torch.arange(entries, dtype=torch.int32)), entries, heads,
                                   dim, dim, silu=False, max_q_len=max(lens), run_powers=powers[1])
        return out.cpu(), state.cpu()

    clean, clean_state = run(rows)
    for t in (0, 5, lens[0] - 1, 66):
        for column, hit in ((2 * width + dim + 3, slice(dim + 3, dim + 4)), (width + 7, slice(0, dim))):
            broken = rows.clone()
            broken[t, column] = bad
            out, state = run(broken)
            changed = torch.zeros(n, width, dtype=torch.bool)
            changed[t:lens[0], hit] = True
            assert torch.equal(out[~changed], clean[~changed]) and not torch.isfinite(out[changed]).any(), (t, column)
            assert torch.equal(state[1:], clean_state[1:])


@pytest.mark.parametrize("key_dim, value_dim", [(64, 64), (128, 128)])
@pytest.mark.parametrize("dtype", DTYPES)
def test_linear_attention_in_runs_keeps_infinities_and_the_largest_numbers(key_dim, value_dim, dtype):
    """One infinite (or, in 32 bits, very large) number of q, k, v or the state: what the formula of the runs gives in 64 bits, infinities with their signs."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    heads, n, run = 2, 400, ops.linear_attention_run()
    qk, vv = heads * key_dim, heads * value_dim
    decay = torch.tensor([0.99, 0.9], dtype=torch.float64)
    powers = [dev((decay[:, None] ** torch.arange(most + 1, dtype=torch.float64)).float().contiguous()) for most in (ops.linear_attention_chunk(key_dim, value_dim), run)]
    rows, held = rnd(n, 2 * qk + vv, dtype=dtype, scale=0.05), rnd(1, heads, key_dim, value_dim, seed=5, scale=0.05)
    held, large = held + 0.01 * held.sign(), 3.395e38      # (above the largest bf16 number)

    def reference(rows, held):
        x, s = rows.double(), held[0].double().clone()
        q, k, v = x[:, :qk].view(n, heads, -1), x[:, qk:2 * qk].view(n, heads, -1), x[:, 2 * qk:].view(n, heads, -1)
        out = torch.empty(n, heads, value_dim, dtype=torch.float64)
        for t0 in range(0, n, run):
            m = min(run, n - t0)
            for h in range(heads):
                back = decay[h] ** torch.arange(m, dtype=torch.float64)
                scores = q[t0:t0 + m, h] @ k[t0:t0 + m, h].T
                for i in range(m):
                    out[t0 + i, h] = decay[h] ** (i + 1) * (q[t0 + i, h] @ s[h]) + (scores[i, :i + 1] * back[:i + 1].flip(0)) @ v[t0:t0 + i + 1, h]
                s[h] = decay[h] ** m * s[h] + (k[t0:t0 + m, h] * back.flip(0)[:, None]).T @ v[t0:t0 + m, h]
        return out.view(n, -1).float(), s.float()

    places = [("state", (0, 1, 17, 5)), ("q", (200, key_dim + 3)), ("k", (130, qk + 7)), ("v", (255, 2 * qk + value_dim + 9)), ("k", (399, qk + key_dim + 1))]
    for what, place in places:
        for bad in (float("inf"), float("-inf"), float("nan")) + ((large,) if dtype == torch.float32 or what == "state" else ()):
            broken, state = rows.clone(), held.clone()
            (state if what == "state" else broken)[place] = bad
            want, want_state = reference(broken, state)
            proj, got_state = dev(broken), dev(state)
            out = ops.linear_attention(proj[:, :qk], proj[:, qk:2 * qk], proj[:, 2 * qk:], torch.empty(n, vv, device="cuda"), got_state, powers[0],
                                       dev(torch.tensor([0, n], dtype=torch.int32)), dev(torch.zeros(1, dtype=torch.int32)), 1, heads, key_dim, value_dim, silu=False,
                                       max_q_len=n, run_powers=powers[1], portions={n: 1})
            for got, ref in ((out.cpu(), want), (got_state[0].cpu(), want_state)):
                assert torch.equal(got.isnan(), ref.isnan()), (what, bad)
                assert torch.equal(got.sign() * got.isinf(), ref.sign() * ref.isinf()), (what, bad)
                # (fp32 sums: 2e-6 of the largest value a sum of this kind meets, as in the test of the forms; a column's or row's own where one is huge)
                fine = torch.isfinite(ref)
                size = ref.abs().where(fine, 0.).amax(-1, keepdim=True).maximum(ref.abs().where(fine, 0.).amax(-2, keepdim=True))
                assert ((got - ref).abs() <= 2e-6 * size + 2e-8)[fine].all(), (what, bad)


# ------------------------------------------------------------------------------------------------- the experts' products
@pytest.mark.parametrize("tokens, experts, top, k, n, act, by_pair, out_dtype", [
    (1, 1, 1, 8, 16, "none", True, torch.float32), (5, 4, 2, 72, 130, "relu2", True, torch.bfloat16),      # tails of k and of the features
    (40, 3, 2, 128, 96, "silu", True, torch.bfloat16), (90, 3, 2, 200, 136, "gelu", True, torch.float32),   # tiles of 64 and 96 rows
    (400, 5, 2, 192, 192, "swiglu", True, torch.bfloat16), (330, 2, 1, 64, 258, "glu_clamp", True, torch.bfloat16),      # 160, several a expert
    (64, 16, 1, 64, 128, "none", False, torch.float32), (700, 3, 2, 136, 260, "none", False, torch.float32)])            # rows already sorted
def test_expert_product_on_uneven_experts(tokens, experts, top, k, n, act, by_pair, out_dtype):
    need_gpu()
    from torchinferno_b200.kernels import ops
    pairs, gated = tokens * top, act in ("swiglu", "glu_clamp")
    scores = rnd(tokens, experts, seed=2)
    scores[:, 0] += 1.5                                   # (one expert gets many rows, some perhaps none)
    ids = scores.topk(top, -1).indices.int().contiguous()
    offsets, order, place = (torch.empty(m, dtype=torch.int32, device="cuda") for m in (experts + 1, pairs, pairs))
    ops.moe_group(dev(ids), experts, offsets, order, place)
    x, w = rnd(tokens if by_pair else pairs, k, dtype=torch.bfloat16), rnd(experts, n, k, dtype=torch.bfloat16, scale=k ** -0.5, seed=3)
    factor = rnd(pairs, seed=4).abs() if gated else None
    y = torch.full((pairs, n // 2 if gated else n), float("nan"), dtype=out_dtype, device="cuda")
    error = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.moe_expert_product(dev(x), dev(w), y, offsets, order, top, x_by_pair=by_pair, act=act, limit=2.0, alpha=1.702,
                           row_scale=None if factor is None else dev(factor), error_word=error)
    assert int(error) == 0
    order, expert_of = order.cpu().long(), ids.flatten().long()
    assert torch.equal(expert_of[order], expert_of.sort()[0])
    rows = x.double()[order // top] if by_pair else x.double()
    v = torch.einsum("sk,snk->sn", rows, w.double()[expert_of[order]])
    if factor is not None:
        v = v * factor.double()[order][:, None]
    if act == "relu2":
        v = v.clamp(min=0) ** 2
    elif act == "silu":
        v = v * torch.sigmoid(v)
    elif act == "gelu":
        v = 0.5 * v * (1 + torch.erf(v * 0.5 ** 0.5))
    elif act == "swiglu":
        v = v[:, 0::2] * torch.sigmoid(v[:, 0::2]) * v[:, 1::2]
    elif act == "glu_clamp":
        g = v[:, 0::2].clamp(max=2.0)
        v = g * torch.sigmoid(1.702 * g) * (v[:, 1::2].clamp(-2.0, 2.0) + 1)
    # exact bf16 products, fp32 sums of k of them (2^-23 of the largest partial sum each), then one rounding to the output type
    bound = (2.0 ** -8 if out_dtype == torch.bfloat16 else 0.0) * v.abs() + 4 * k * 2.0 ** -23
    assert ((as_ref(y) - v).abs() <= bound).all()


# ------------------------------------------------------------- the state-space scan in chunks, convolutions and gated norms by eight
@pytest.mark.parametrize("lens, heads, head_dim, state, groups, shift", [
    ([65, 1, 128], 4, 64, 128, 2, 0.0), ([129, 64, 256], 2, 128, 64, 1, 0.0), ([300], 4, 32, 64, 4, 0.0), ([127, 130], 2, 32, 128, 1, -6.0),
    ([200, 70], 2, 64, 128, 1, 8.0)])      # (steps near zero: nothing decays; steps of eight: everything does)
def test_scan_in_chunks_agrees_with_the_recurrence(lens, heads, head_dim, state, groups, shift):
    need_gpu()
    from torchinferno_b200.kernels import ops
    n, inner, entries = sum(lens), heads * head_dim, len(lens)
    xbc, dt = rnd(n, inner + 2 * groups * state, dtype=torch.bfloat16), rnd(n, heads, dtype=torch.bfloat16, seed=1)
    bias, a_log, skip = rnd(heads, seed=2) + shift, 0.5 * rnd(heads, seed=3), rnd(heads, seed=4)
    held, slots = rnd(entries + 1, heads * state * head_dim + 8, seed=5), [entries - i for i in range(entries)]
    starts = torch.tensor([sum(lens[:i]) for i in range(entries + 1)], dtype=torch.int32)
    y, got = torch.empty(n, inner, device="cuda"), dev(held.clone())
    ops.ssd_scan(dev(xbc), dev(dt), 0, dev(bias), dev(a_log), dev(skip), got, dev(starts), dev(torch.tensor(slots, dtype=torch.int32)), y, entries,
                 heads=heads, groups=groups, state_dim=state, head_dim=head_dim, max_q_len=max(lens))
    x = xbc[:, :inner].double().view(n, heads, head_dim)
    b, c = (xbc[:, inner + i * groups * state:inner + (i + 1) * groups * state].double().view(n, groups, state).repeat_interleave(heads // groups, 1)
            for i in range(2))
    step = torch.nn.functional.softplus(dt.double() + bias.double(), threshold=1e9)
    decay = (-a_log.double().exp() * step).exp()
    want, want_state = torch.empty(n, heads, head_dim, dtype=torch.float64), held.double().clone()
    for e, length in enumerate(lens):
        s = want_state[slots[e], :heads * state * head_dim].view(heads, state, head_dim).clone()
        for t in range(int(starts[e]), int(starts[e]) + length):
            s = decay[t][:, None, None] * s + (step[t][:, None] * b[t])[:, :, None] * x[t][:, None, :]
            want[t] = torch.einsum("hsp,hs->hp", s, c[t]) + skip.double()[:, None] * x[t]
        want_state[slots[e], :heads * state * head_dim] = s.reshape(-1)
    # everything 32-bit enters its products with 24 bits: sums of up to `state` + 128 such terms, 2^-23 of the largest value each
    for out, ref in ((y, want.reshape(n, inner)), (got, want_state)):
        assert (as_ref(out) - ref).abs().max() <= 32 * 2.0 ** -23 * ref.abs().max()


@pytest.mark.parametrize("heads, head_dim, state, groups, lens", [
    (62, 64, 128, 1, [700, 300]), (46, 64, 64, 2, [900, 257, 40]), (22, 128, 128, 1, [1100]), (80, 64, 64, 4, [650, 129])])      # (three or four a block)
def test_scan_in_chunks_with_several_heads_a_block(heads, head_dim, state, groups, lens):
    """Steps large enough that a block takes several heads (or 64-column tiles of them) of a group, the last of a group fewer: the recurrence, the bits
    that a few heads alone have (a block each), and numbers that are not finite in some of a block's heads."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    n, inner, entries = sum(lens), heads * head_dim, len(lens)
    xbc, dt = rnd(n, inner + 2 * groups * state, dtype=torch.bfloat16), rnd(n, heads, dtype=torch.bfloat16, seed=1)
    bias, a_log, skip = rnd(heads, seed=2) - 2.0, 0.5 * rnd(heads, seed=3), rnd(heads, seed=4)
    held, starts = rnd(entries, heads, state, head_dim, seed=5), torch.tensor([sum(lens[:i]) for i in range(entries + 1)], dtype=torch.int32)

    def run(xbc, of):
        """The heads ``of`` of one group (None: all of them)."""
        if of is None:
            rows, own, g = xbc, slice(None), groups
        else:
            at, g = of[0] // (heads // groups), 1
            rows = torch.cat([xbc[:, of[0] * head_dim:(of[-1] + 1) * head_dim]] + [xbc[:, inner + (i * groups + at) * state:inner + (i * groups + at + 1) * state] for i in range(2)], 1)
            own = slice(of[0], of[-1] + 1)
        count = heads if of is None else len(of)
        y, carried = torch.empty(n, count * head_dim, device="cuda"), dev(held[:, own].reshape(entries, -1).contiguous())
        error = torch.zeros(1, dtype=torch.int32, device="cuda")
        ops.ssd_scan(dev(rows.contiguous()), dev(dt[:, own].contiguous()), 0, dev(bias[own].contiguous()), dev(a_log[own].contiguous()), dev(skip[own].contiguous()), carried,
                     dev(starts), dev(torch.arange(entries, dtype=torch.int32)), y, entries, heads=count, groups=g, state_dim=state, head_dim=head_dim,
                     max_q_len=max(lens), error_word=error)
        assert int(error) == 0
        return y.cpu().view(n, count, head_dim), carried.cpu().view(entries, count, state, head_dim)

    y, carried = run(xbc, None)
    x = xbc[:, :inner].double().view(n, heads, head_dim)
    b, c = (xbc[:, inner + i * groups * state:inner + (i + 1) * groups * state].double().view(n, groups, state).repeat_interleave(heads // groups, 1)
            for i in range(2))
    step = torch.nn.functional.softplus(dt.double() + bias.double(), threshold=1e9)
    decay = (-a_log.double().exp() * step).exp()
    want, want_state = torch.empty(n, heads, head_dim, dtype=torch.float64), held.double().clone()
    for e, length in enumerate(lens):
        s = want_state[e].clone()
        for t in range(int(starts[e]), int(starts[e]) + length):
            s = decay[t][:, None, None] * s + (step[t][:, None] * b[t])[:, :, None] * x[t][:, None, :]
            want[t] = torch.einsum("hsp,hs->hp", s, c[t]) + skip.double()[:, None] * x[t]
        want_state[e] = s
    for got, ref in ((y, want), (carried, want_state)):      # (as where a block takes one head)
        assert (got.double() - ref).abs().max() <= 32 * 2.0 ** -23 * ref.abs().max()
    last = heads // groups - 1
    parts = [[0], [1, 2], [last - 1, last], [heads - 2, heads - 1]]
    for of in parts:
        few, few_state = run(xbc, of)
        assert torch.equal(few, y[:, of]) and torch.equal(few_state, carried[:, of]), of
    broken = xbc.clone()
    for h, t, bad in ((1, 5, math.inf), (2, 140, math.nan), (last, 127, -math.inf), (heads - 1, 0, math.nan), (heads - 1, lens[0] - 1, math.inf)):
        broken[t, h * head_dim + 3 + h % 32] = bad
    odd, odd_state = run(broken, None)
    bits = lambda t: t.contiguous().view(torch.int32).where(~t.isnan(), 0)
    for of in parts:
        few, few_state = run(broken, of)
        assert torch.equal(bits(few), bits(odd[:, of])) and torch.equal(bits(few_state), bits(odd_state[:, of])), of
    keep = torch.ones(n, heads, head_dim, dtype=torch.bool)
    keep[:lens[0], [1, 2, last, heads - 1]] = False
    assert torch.equal(odd[keep], y[keep]) and not odd[~keep].isfinite().all()


@pytest.mark.parametrize("lens, head_dim, state", [([300, 7, 129], 64, 128), ([140, 70], 32, 64)])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_scan_in_chunks_keeps_what_is_not_finite_from_earlier_tokens(lens, head_dim, state, bad):
    """One number of x of one request: only its own column changes, from its own token on.  One of B: the tokens from its own on;
    one of C: its own token alone."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    heads, n, entries = 2, sum(lens), len(lens)
    inner = heads * head_dim
    xbc, dt = rnd(n, inner + 2 * state, dtype=torch.bfloat16), dev(rnd(n, heads, dtype=torch.bfloat16, seed=1))
    bias, a_log, skip = dev(rnd(heads, seed=2) - 3.0), dev(rnd(heads, seed=3)), dev(rnd(heads, seed=4))
    held, starts = rnd(entries, heads * state * head_dim, seed=5), [sum(lens[:i]) for i in range(entries + 1)]

    def run(rows):
        y, carried = torch.empty(n, inner, device="cuda"), dev(held.clone())
        ops.ssd_scan(dev(rows), dt, 0, bias, a_log, skip, carried, dev(torch.tensor(starts, dtype=torch.int32)),
                     dev(torch.arange(entries, dtype=torch.int32)), y, entries, heads=heads, groups=1, state_dim=state, head_dim=head_dim,
                     max_q_len=max(lens))
        return y.cpu(), carried.cpu()

    clean, clean_state = run(xbc)
    for t in (0, 5, 15, 16, 127, 128, lens[0] - 1):
        for column, last, hit in ((head_dim + 3, lens[0], slice(head_dim + 3, head_dim + 4)), (inner + 9, lens[0], slice(0, inner)),
                                  (inner + state + 9, t + 1, slice(0, inner))):
            broken = xbc.clone()
            broken[t, column] = bad
            y, carried = run(broken)
            changed = torch.zeros(n, inner, dtype=torch.bool)
            changed[t:last, hit] = True
            assert torch.equal(y[~changed], clean[~changed]) and not torch.isfinite(y[changed]).any(), (t, column)
            assert torch.equal(carried[1:], clean_state[1:])


@pytest.mark.parametrize("head_dim, state", [(64, 128), (32, 64)])      # (on tcgen05; on mma.sync)
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_scan_in_chunks_keeps_a_step_size_that_is_not_finite_from_earlier_tokens(head_dim, state, bad):
    """One step size of one head of one request: that head's rows from the token on, whichever of its four neighbours in the scan it is."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    heads, lens = 3, [300, 129]
    n, inner = sum(lens), heads * head_dim
    xbc, steps = dev(rnd(n, inner + 2 * state, dtype=torch.bfloat16)), rnd(n, heads, dtype=torch.bfloat16, seed=1)
    bias, a_log, skip = dev(rnd(heads, seed=2) - 3.0), dev(rnd(heads, seed=3)), dev(rnd(heads, seed=4))
    held, starts = rnd(2, heads * state * head_dim, seed=5), dev(torch.tensor([0, lens[0], n], dtype=torch.int32))

    def run(dt):
        y, carried = torch.empty(n, inner, device="cuda"), dev(held.clone())
        ops.ssd_scan(xbc, dev(dt), 0, bias, a_log, skip, carried, starts, dev(torch.arange(2, dtype=torch.int32)), y, 2, heads=heads, groups=1,
                     state_dim=state, head_dim=head_dim, max_q_len=max(lens))
        return y.cpu(), carried.cpu()

    clean, clean_state = run(steps)
    for t in (0, 1, 2, 3, 5, 30, 31, 126, 127, 128, 130, lens[0] - 1):
        broken = steps.clone()
        broken[t, 1] = bad
        y, carried = run(broken)
        changed = torch.zeros(n, inner, dtype=torch.bool)
        changed[t:lens[0], head_dim:2 * head_dim] = True
        assert torch.equal(y[~changed], clean[~changed]) and torch.equal(carried[1:], clean_state[1:]), t
        if bad != bad:
            assert y[changed].isnan().all(), t


def test_scan_in_chunks_keeps_infinities_with_their_signs():
    """An infinite x or step size: its columns of the state as token by token; an infinite B: the rows of its chunk as well."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    heads, head_dim, state, n = 2, 64, 128, 200
    inner = heads * head_dim
    xbc, steps = rnd(n, inner + 2 * state, dtype=torch.bfloat16), rnd(n, heads, dtype=torch.bfloat16, seed=1)
    bias, a_log, skip = dev(rnd(heads, seed=2) - 6.0), dev(0.2 * rnd(heads, seed=3)), dev(rnd(heads, seed=4))      # (nothing decays to zero)
    held = rnd(1, heads * state * head_dim, seed=5)
    signs = lambda t: t.sign() * t.isinf()
    for what, t, column in (("x", 0, 3), ("x", 70, head_dim + 17), ("x", 127, 63), ("x", 128, 40), ("x", n - 1, 0), ("step", 65, 1), ("step", 131, 0), ("B", 0, 9), ("B", 40, 9), ("B", 150, 100)):
        for bad in (math.inf,) if what == "step" else (math.inf, -math.inf):
            rows, dt = xbc.clone(), steps.clone()
            (dt if what == "step" else rows)[t, inner + column if what == "B" else column] = bad
            results = []
            for longest in (n, None):      # (in chunks; token by token)
                y, carried = torch.empty(n, inner, device="cuda"), dev(held.clone())
                ops.ssd_scan(dev(rows), dev(dt), 0, bias, a_log, skip, carried, dev(torch.tensor([0, n], dtype=torch.int32)), dev(torch.zeros(1, dtype=torch.int32)),
                             y, 1, heads=heads, groups=1, state_dim=state, head_dim=head_dim, max_q_len=longest)
                results.append((carried.view(heads, state, head_dim).cpu(), y.cpu()))
            (got, y), (want, want_y) = results
            if what == "B":
                rows = slice(t, min(n, t // 128 * 128 + 128))
                assert (signs(y[rows]) != 0).all() and torch.equal(signs(y[rows]), signs(want_y[rows])), (what, t, bad)
            else:
                assert torch.equal(got.isnan(), want.isnan()) and torch.equal(signs(got), signs(want)) and int(got.isinf().sum()) == state * (head_dim if what == "step" else 1), (what, t, bad)


def test_scan_in_chunks_of_an_infinite_state():
    """One infinite element of a request's state: its column is infinite from then on, as in the token-by-token walk."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    heads, head_dim, state, n = 2, 64, 128, 200
    inner = heads * head_dim
    xbc, dt = dev(rnd(n, inner + 2 * state, dtype=torch.bfloat16)), dev(rnd(n, heads, dtype=torch.bfloat16, seed=1))
    bias, a_log, skip = dev(rnd(heads, seed=2) - 6.0), dev(0.2 * rnd(heads, seed=3)), dev(rnd(heads, seed=4))
    held = rnd(1, heads, state, head_dim, seed=5)
    held[0, 1, 17, 5] = float("inf")
    results = []
    for longest in (n, None):      # (in chunks; token by token)
        y, carried = torch.empty(n, inner, device="cuda"), dev(held.view(1, -1).clone())
        ops.ssd_scan(xbc, dt, 0, bias, a_log, skip, carried, dev(torch.tensor([0, n], dtype=torch.int32)), dev(torch.zeros(1, dtype=torch.int32)), y, 1,
                     heads=heads, groups=1, state_dim=state, head_dim=head_dim, max_q_len=longest)
        results.append((y.cpu(), carried.cpu()))
    for chunks, walk in zip(*results):
        assert torch.isinf(walk).any() and torch.equal(torch.where(torch.isinf(walk), walk, 0.0), torch.where(torch.isfinite(chunks), 0.0, chunks))
        fine = torch.isfinite(walk)
        assert (chunks[fine] - walk[fine]).abs().max() <= 32 * 2.0 ** -23 * walk[fine].abs().max()      # (the bound of the finite states' test)


# (the last: more segments of eight tokens than a grid is high or deep)
@pytest.mark.parametrize("lens, channels, taps", [([1, 2, 3], 8, 4), ([16, 17, 1], 1032, 3), ([50, 2], 520, 2), ([40], 16, 4), ([7, 9], 512, 4), ([8, 524300], 8, 4)])
def test_short_convolution_by_eight_channels_has_the_plain_kernels_bits(lens, channels, taps):
    need_gpu()
    from torchinferno_b200.kernels import ops
    n, entries = sum(lens), len(lens)
    rows = rnd(n, channels + 24, dtype=torch.bfloat16)
    weight, bias, state = rnd(channels, taps, seed=1), rnd(channels, seed=2), rnd(entries, (taps - 1) * channels, seed=3)
    starts = torch.tensor([sum(lens[:i]) for i in range(entries + 1)], dtype=torch.int32)
    results = []
    for shift in (8, 9):      # (columns off their 16-byte boundaries take the plain kernel)
        wide = torch.zeros(n, channels + 24, dtype=torch.bfloat16)
        wide[:, shift:shift + channels] = rows[:, 8:8 + channels]
        out, held = torch.empty(n, channels, dtype=torch.bfloat16, device="cuda"), dev(state.clone())
        ops.short_conv(dev(wide), shift, dev(weight), dev(bias), held, 0, dev(starts), dev(torch.arange(entries, dtype=torch.int32)), out,
                       entries, max(lens), silu=True)
        results.append((out, held))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("rows, width, parts", [(1, 8, 1), (3, 264, 1), (5, 2056, 1), (2, 4104, 1), (3, 8192, 4), (2, 8200, 1)])
@pytest.mark.parametrize("mode", ["gate last", "gate first", "norm and gate", "gate", "head gate"])
def test_gated_rows_by_eight_columns(rows, width, parts, mode):
    need_gpu()
    from torchinferno_b200.kernels import ops
    y, z, weight = rnd(rows, width), rnd(rows, width + 16, dtype=torch.bfloat16, seed=1), rnd(width, seed=2)
    out = torch.empty(rows, width, dtype=torch.bfloat16, device="cuda")
    v, gate = y.double(), z[:, 8:8 + width].double()
    if mode in ("gate last", "gate first"):
        ops.gated_group_norm(dev(y), dev(z), 8, dev(weight), 1e-6, out, parts, gate_last=mode == "gate last")
        v = v * gate * torch.sigmoid(gate) if mode == "gate first" else v
        v = v.view(rows, parts, -1)
        v = (v / (v.pow(2).mean(-1, keepdim=True) + 1e-6).sqrt()).reshape(rows, width) * weight.double()
        want = v * torch.sigmoid(gate) if mode == "gate last" else v
    elif mode == "norm and gate":
        ops.sigmoid_gate(dev(y), dev(z)[:, 8:8 + width], out, dev(weight), 1e-6)
        want = v / (v.pow(2).mean(-1, keepdim=True) + 1e-6).sqrt() * weight.double() * torch.sigmoid(gate)
    else:
        group = 8 if mode == "head gate" else 1
        ops.sigmoid_gate(dev(y).bfloat16(), dev(z)[:, 8:8 + width // group], out, group=group)
        want = y.bfloat16().double() * torch.sigmoid(z[:, 8:8 + width // group].double()).repeat_interleave(group, 1)
    # fp32 arithmetic (a few roundings of 2^-24), then one rounding to the eight significant bits of bfloat16 (2^-8 at most)
    assert ((as_ref(out) - want).abs() <= 1.01 * 2.0 ** -8 * want.abs() + 1e-6 * want.abs().max()).all()


# ------------------------------------------------- routers, weighted sums, appends and block means of large steps
@pytest.mark.parametrize("rows, k", [(1, 64), (8, 72), (9, 520), (33, 1020), (128, 256)])      # one, three and five rows a warp
@pytest.mark.parametrize("dtype", DTYPES)
def test_router_logits_of_large_steps_have_the_bits_of_small_ones(rows, k, dtype):
    need_gpu()
    from torchinferno_b200.kernels import ops
    tokens = 8 * 148 + 5
    x, w, bias = dev(rnd(tokens, (k + 7) // 8 * 8, dtype=dtype))[:, :k], dev(rnd(rows, k, seed=1)), dev(rnd(rows, seed=2))
    out = ops.router_logits(x, w, torch.empty(tokens, rows, device="cuda"), bias)
    parts = [ops.router_logits(x[i:i + 400], w, torch.empty(len(x[i:i + 400]), rows, device="cuda"), bias) for i in range(0, tokens, 400)]
    assert torch.equal(out, torch.cat(parts))
    want = as_ref(x) @ as_ref(w).T + as_ref(bias)
    assert (as_ref(out) - want).abs().max() <= k * 2.0 ** -23 * want.abs().max()      # fp32 sums of k products


@pytest.mark.parametrize("tokens, width, top", [(1, 8, 1), (7, 520, 3), (300, 2056, 2)])
@pytest.mark.parametrize("shared, handed_on", [(False, False), (True, False), (True, True)])
def test_weighted_sums_by_eight_columns_have_the_plain_kernels_bits(tokens, width, top, shared, handed_on):
    need_gpu()
    from torchinferno_b200.kernels import ops
    y, weights = rnd(tokens * top, width), rnd(tokens, top, seed=1).abs()
    place = dev(torch.randperm(tokens * top, generator=torch.Generator().manual_seed(2)).int().view(tokens, top))
    options = {}
    if shared:
        options = dict(shared=dev(rnd(tokens, width, dtype=torch.bfloat16, seed=3)), gate=dev(rnd(tokens, 1, seed=4))[:, 0])
    if handed_on:
        ids = torch.arange(tokens * top, dtype=torch.int32).view(tokens, top) % 5
        options.update(ids=dev(ids), identity_from=3, x=dev(rnd(tokens, width, dtype=torch.bfloat16, seed=5)))
    results = []
    for shift in (0, 1):      # (rows off their 16-byte boundaries take the plain kernel)
        rows = torch.empty(y.numel() + shift, device="cuda")[shift:].view(y.shape).copy_(dev(y))
        results.append(ops.moe_combine(rows, place, dev(weights), torch.empty(tokens, width, dtype=torch.bfloat16, device="cuda"), **options))
    assert torch.equal(*results)


def page_views(pages, kv_heads, page, dim, vdim, dtype):
    """One layer's key and value pages side by side in one buffer, zeroed."""
    both = torch.zeros(pages, kv_heads * page * (dim + vdim), dtype=dtype, device="cuda")
    cut = kv_heads * page * dim
    return both[:, :cut].view(pages, kv_heads, page, dim), both[:, cut:].view(pages, kv_heads, page, vdim)


@pytest.mark.parametrize("tokens, heads, kv_heads, dim, vdim, rot, turned", [
    (3, 2, 1, 64, 32, 64, True), (70, 5, 2, 36, 20, 12, True), (33, 4, 4, 256, 256, 128, True), (9, 3, 1, 8, 6, 4, False)])
def test_append_with_one_table_of_angles_agrees_with_the_plain_kernel(tokens, heads, kv_heads, dim, vdim, rot, turned):
    need_gpu()
    from torchinferno_b200.kernels import ops
    total, page = heads * dim + kv_heads * (dim + vdim), 8
    pages = -(-tokens // page) + 1
    rows, q_bias = rnd(tokens, total, dtype=torch.bfloat16), dev(rnd(heads * dim, seed=1))
    freq = dev(1e4 ** (-torch.arange(rot // 2) / (rot // 2)))
    vfreq = dev(1e4 ** (-torch.arange(vdim // 2) / (vdim // 2))) if turned else None
    table = dev(torch.randperm(pages, generator=torch.Generator().manual_seed(3)).int().view(1, pages))
    results = []
    for shift in (2, 1):      # (columns off their 4-byte boundaries take the plain kernel)
        wide = torch.zeros(tokens, total + 2, dtype=torch.bfloat16)
        wide[:, shift:shift + total] = rows
        keys, values = page_views(pages, kv_heads, page, dim, vdim, torch.bfloat16)
        q = torch.empty(tokens, heads * dim, dtype=torch.bfloat16, device="cuda")
        ops.rotary_kv_append(dev(wide), shift, shift + heads * dim,
                             shift + (heads + kv_heads) * dim, q, keys, values, dev(torch.arange(tokens, dtype=torch.int32)),
                             torch.zeros(tokens, dtype=torch.int32, device="cuda"), table, freq, vfreq, heads, kv_heads, dim, vdim,
                             rot_dim=rot, amplitude=1.25, q_bias=q_bias)
        results.append((q, keys, values))
    for got, plain in zip(*results):
        assert torch.equal(got, plain)      # (the same turns and sums in fp32, each rounded once to bfloat16)


# (297 tokens are the fewest that go in pieces of 16 bytes, 2,049 go two a block; halves of eight elements, heads that are turned whole or not at all, more
# pieces than threads; three requests that begin on odd rows, so that a block holds tokens of two)
@pytest.mark.parametrize("tokens", [297, 2049])
@pytest.mark.parametrize("missing", [False, True])
@pytest.mark.parametrize("heads, kv_heads, dim, vdim, rot, turned, bias", [
    (3, 1, 64, 64, 64, True, True), (5, 2, 32, 16, 16, True, False), (24, 8, 128, 128, 32, True, True), (2, 2, 48, 80, 0, False, True), (4, 4, 256, 256, 128, True, False)])
def test_append_in_pieces_agrees_with_the_plain_kernel(tokens, missing, heads, kv_heads, dim, vdim, rot, turned, bias):
    """``missing``: the first page of the request that begins on a block's second token is out of range: it is reported, the first token is stored."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    page, lens, pasts = 8, [tokens // 3 | 1, tokens // 4 * 2, 0], [5, 800, 30]
    lens[2] = tokens - lens[0] - lens[1]
    total, per = heads * dim + kv_heads * (dim + vdim), -(-max(n + p for n, p in zip(lens, pasts)) // page)
    pages = 3 * per
    rows, biases = rnd(tokens, total, dtype=torch.bfloat16), [dev(rnd(w, seed=i)) if bias else None for i, w in enumerate((heads * dim, kv_heads * dim, kv_heads * vdim))]
    freq = dev(1e4 ** (-torch.arange(rot // 2) / max(rot // 2, 1)))
    vfreq = dev(1e4 ** (-torch.arange(vdim // 2) / (vdim // 2))) if turned else None
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(3)).int().view(3, per)
    if missing:
        table[1, pasts[1] // page] = pages
    positions = torch.cat([p + torch.arange(n) for n, p in zip(lens, pasts)]).int()
    token_slot = torch.cat([torch.full((n,), i) for i, n in enumerate(lens)]).int()
    assert lens[0] % 2 == 1 and pasts[1] % page == 0
    results = []
    for shift in (8, 1):      # (columns off their boundaries take the plain kernel)
        wide = torch.zeros(tokens, total + 8, dtype=torch.bfloat16)
        wide[:, shift:shift + total] = rows
        keys, values = page_views(pages, kv_heads, page, dim, vdim, torch.bfloat16)
        q = torch.empty(tokens, heads * dim, dtype=torch.bfloat16, device="cuda")
        turns = torch.empty(tokens, vdim // 2, 2, device="cuda") if turned else None
        error = torch.zeros(1, dtype=torch.int32, device="cuda")
        ops.rotary_kv_append(dev(wide), shift, shift + heads * dim, shift + (heads + kv_heads) * dim, q, keys, values,
                             dev(positions), dev(token_slot), dev(table), freq, vfreq, heads,
                             kv_heads, dim, vdim, rot_dim=rot, amplitude=1.25, q_bias=biases[0], k_bias=biases[1], v_bias=biases[2], turns=turns, error_word=error)
        assert (int(error) != 0) == missing
        results.append((q, keys, values) + ((turns,) if turned else ()))
    for got, plain in zip(*results):
        assert torch.equal(got, plain)      # (the same turns and sums in fp32, each rounded once to bfloat16)


@pytest.mark.parametrize("dim, keep, pool", [(64, 0, 16), (128, 0, 64), (128, 40, 0)])
@pytest.mark.parametrize("gated", [False, True])
def test_window_attention_with_the_appends_turns_has_the_bits_of_its_own(dim, keep, pool, gated):
    """Two portions whose tiles begin and end off the window's, the blocks' and the kept tokens' edges."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    heads, kv_heads, page, window, lens, pasts = 4, 2, 16, 150, [130, 260], [333, 0]
    n, per = sum(lens), 32
    ints = lambda v: dev(torch.tensor(list(v), dtype=torch.int32))
    keys, values = (dev(rnd(2 * per, kv_heads, page, dim, dtype=torch.bfloat16, seed=i)) for i in range(2))
    means = [dev(rnd(4, kv_heads, page, dim, dtype=torch.bfloat16, seed=5 + i)) for i in range(2)] if pool else [None, None]
    table, blocks = ints(range(2 * per)).view(2, per), ints(range(4)).view(2, 2)
    q, gate = dev(rnd(n, heads * dim, dtype=torch.bfloat16)), dev(rnd(n, heads * dim, dtype=torch.bfloat16, seed=9)) if gated else None
    freq = dev(5e5 ** (-torch.arange(dim // 2) / (dim // 2)))
    positions = torch.cat([p + torch.arange(m) for m, p in zip(lens, pasts)])
    angle = dev(positions.float())[:, None] * freq
    turns = torch.stack([angle.cos(), angle.sin()], -1).contiguous()
    own = torch.empty_like(turns)
    pool_keys, pool_values = page_views(60, kv_heads, page, dim, dim, torch.bfloat16)
    ops.rotary_kv_append(q[:, :2 * kv_heads * dim].repeat(1, 2).contiguous(), 0, 0, 0, torch.empty(n, kv_heads * dim, dtype=torch.bfloat16, device="cuda"), pool_keys, pool_values,
                         dev(positions.int()), torch.zeros(n, dtype=torch.int32, device="cuda"), ints(range(60)).view(1, 60), freq, freq, kv_heads, kv_heads, dim, dim,
                         rot_dim=dim, turns=own)
    assert (own - turns).abs().max() <= 2.0 ** -22      # (cosines and sines to an ulp or two of one)
    run = lambda turns: ops.pooled_window_attention(q, torch.empty_like(q), ints([0, lens[0], n]), ints(pasts), ints(range(2)), keys, values, table, *means,
                                                    blocks if pool else None, 2, max(lens), heads, kv_heads, window=window, pool=pool, scale=dim ** -0.5, keep=keep,
                                                    value_freq=freq, gate=gate, turns=turns)
    assert torch.equal(run(own), run(None))


GATES = [float("nan"), float("inf"), float("-inf"), 0.0, -20.0, 60.0, -86.0, -87.5, -88.5]      # (the last: a sigmoid below the normal numbers)


def test_gates_of_window_attention_on_prompts():
    """A prompt's gates against those of the kernel for few tokens: NaN stays NaN, the smallest ones do not become zero."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    heads, kv_heads, page, dim, n = 2, 1, 16, 64, 140
    ints = lambda v: dev(torch.tensor(list(v), dtype=torch.int32))
    per = -(-n // page)
    keys, values = (dev(rnd(per, kv_heads, page, dim, dtype=torch.bfloat16, seed=i)) for i in range(2))
    q, gate = dev(rnd(n, heads * dim, dtype=torch.bfloat16)), rnd(n, heads * dim, seed=9)
    for i, g in enumerate(GATES):
        gate[3 + 13 * i, 5 * i:5 * i + 60] = g
    gate = dev(gate, torch.bfloat16)
    run = lambda gate: ops.pooled_window_attention(q, torch.empty_like(q), ints([0, n]), ints([0]), ints([0]), keys, values, ints(range(per)).view(1, per), None, None,
                                                   None, 1, n, heads, kv_heads, window=100, pool=0, scale=dim ** -0.5, gate=gate).cpu()
    plain, got = run(None).double(), run(gate)
    want = plain * torch.sigmoid(gate.cpu().double())
    assert torch.equal(got.isnan(), want.isnan()) and not got.isinf().any()
    # a rounding to bf16 is off by at most 2^-8 of the value (eight significant bits), and the rows without gates are rounded and these again
    assert ((got.double() - want).abs() <= 2.0 ** -6.9 * want.abs() + 2.0 ** -133)[~want.isnan()].all()


@pytest.mark.parametrize("per_head", [False, True])
def test_gates_of_latent_attention_on_prompts(per_head):
    need_gpu()
    from torchinferno_b200.kernels import ops
    heads, dim, rot, n = 4, 64, 64, 140
    rows = 256
    ints = lambda v: dev(torch.tensor(list(v), dtype=torch.int32))
    q = dev(rnd(n, heads * (dim + rot), dtype=torch.bfloat16))
    kv, rotated = dev(rnd(rows, heads * 2 * dim, dtype=torch.bfloat16, seed=1)), dev(rnd(rows, rot, dtype=torch.bfloat16, seed=2))
    gate = rnd(n, heads * (1 if per_head else dim), seed=9)
    for i, g in enumerate(GATES):
        gate[3 + 13 * i, i % 4 if per_head else slice(20 * i, 20 * i + 60)] = g
    gate = dev(gate, torch.bfloat16)
    run = lambda gate: ops.latent_prefill(q, kv, rotated, torch.empty(n, heads, dim, dtype=torch.bfloat16, device="cuda"), ints([0, n]), ints([0]), 1, n, heads, dim, dim,
                                          (dim + rot) ** -0.5, gate=gate, gate_per_head=per_head).cpu()
    plain, got = run(None).double(), run(gate)
    want = plain * torch.sigmoid(gate.cpu().double()).view(n, heads, -1)
    assert torch.equal(got.isnan(), want.isnan()) and not got.isinf().any()
    assert ((got.double() - want).abs() <= 2.0 ** -6.9 * want.abs() + 2.0 ** -133)[~want.isnan()].all()


@pytest.mark.parametrize("tokens, kv_heads, dim, vdim, pool", [(65, 1, 64, 64, 4), (97, 2, 40, 24, 8), (300, 2, 128, 96, 32), (130, 1, 16, 8, 1)])
@pytest.mark.parametrize("dtype", DTYPES)
def test_block_means_of_large_steps_have_the_bits_of_small_ones(tokens, kv_heads, dim, vdim, pool, dtype):
    need_gpu()
    from torchinferno_b200.kernels import ops
    page, pages = 16, -(-tokens // 16)
    count = tokens // pool
    keys, values = page_views(pages, kv_heads, page, dim, vdim, dtype)
    keys.copy_(rnd(*keys.shape)), values.copy_(rnd(*values.shape, seed=1))
    table, b_pages = dev(torch.arange(pages, dtype=torch.int32).flip(0).contiguous().view(1, pages)), -(-count // page) + 1
    b_table = dev(torch.arange(b_pages, dtype=torch.int32).view(1, b_pages))
    positions, slots = dev(torch.arange(tokens, dtype=torch.int32)), torch.zeros(tokens, dtype=torch.int32, device="cuda")
    results = []
    for run in (tokens, 50):
        b_keys, b_values = page_views(b_pages, kv_heads, page, dim, vdim, dtype)
        for i in range(0, tokens, run):
            ops.pool_blocks(keys, values, table, b_keys, b_values, b_table, positions[i:i + run], slots[i:i + run], pool)
        results.append((b_keys, b_values))
    for large, small, rows in zip(*results, (keys, values)):
        assert torch.equal(large, small)
        flat = as_ref(rows).flip(0).transpose(1, 2).reshape(pages * page, kv_heads, -1)[:count * pool]
        want = flat.view(count, pool, kv_heads, -1).mean(1)
        got = as_ref(large).transpose(1, 2).reshape(b_pages * page, kv_heads, -1)[:count]
        # fp32 sums of `pool` numbers, then one rounding to the element type
        assert (got - want).abs().max() <= ((2.0 ** -8 if dtype == torch.bfloat16 else 0.0) + (pool + 1) * 2.0 ** -23) * want.abs().max() + pool * 2.0 ** -23


@pytest.mark.parametrize("contexts, heads, rank", [([1, 64, 65, 1000], 3, 64), ([4000], 16, 512), ([129, 700], 20, 200)])
@pytest.mark.parametrize("sink", [False, True])
def test_merged_latent_rows_in_bfloat16_are_the_fp32_rows_rounded_once(contexts, heads, rank, sink):
    need_gpu()
    from torchinferno_b200.kernels import ops
    n, page, rot = len(contexts), 16, 16
    per = -(-max(contexts) // page)
    keys = dev(rnd(n * per, 1, page, rank + rot, dtype=torch.bfloat16, scale=0.7))
    table = dev(torch.randperm(n * per, generator=torch.Generator().manual_seed(4)).int().view(n, per))
    ints = lambda v: dev(torch.tensor(list(v), dtype=torch.int32))
    args = (ints(range(n + 1)), ints(c - 1 for c in contexts), ints(range(n)), table, n, 1, heads, rank, rot, 0.11)
    options = dict(max_kv_len=max(contexts), sink=dev(rnd(heads, seed=2)) if sink else None)
    folded = dev(rnd(n, heads, rank + rot, scale=0.3, seed=1))
    out = ops.latent_attention(folded, keys, torch.empty(n, heads, rank, device="cuda"), *args, **options)
    merged = torch.empty(n, heads, rank, dtype=torch.bfloat16, device="cuda")
    rows = ops.latent_attention(folded, keys, torch.zeros_like(out), *args, merged=merged, **options)
    assert torch.equal(rows.bfloat16(), out.bfloat16())
    assert rows is merged


# (runs of 32 keys: 50, 63, 24, 25, 9 and 8 of them: the merge has nine to 24 on their way at once; a context of one run beside them)
@pytest.mark.parametrize("contexts, heads, rank, rot", [([1600, 33], 3, 64, 16), ([2010], 16, 512, 64), ([768, 1, 700], 2, 96, 0), ([800], 5, 40, 8), ([288, 90], 4, 64, 64), ([256, 17], 3, 512, 64)])
@pytest.mark.parametrize("sink", [False, True])
@pytest.mark.parametrize("simt", [False, True])
def test_latent_single_tokens_over_many_runs(contexts, heads, rank, rot, sink, simt):
    """Against the formula in 64 bits."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    n, page, width, scale = len(contexts), 16, rank + rot, 0.11
    per = -(-max(contexts) // page)
    keys, table = rnd(n * per, 1, page, width, dtype=torch.bfloat16, scale=0.7), torch.randperm(n * per, generator=torch.Generator().manual_seed(4)).int().view(n, per)
    folded, sinks = rnd(n, heads, width, scale=0.3, seed=1).bfloat16().float(), rnd(heads, seed=2) if sink else None      # (no rounding of the queries)
    ints = lambda v: dev(torch.tensor(list(v), dtype=torch.int32))
    assert ops.lib().tib_latent_attention_splits(n, heads, max(contexts)) == -(-max(contexts) // 32)
    out = as_ref(ops.latent_attention(dev(folded), dev(keys), torch.empty(n, heads, rank, device="cuda"), ints(range(n + 1)), ints(c - 1 for c in contexts),
                                      ints(range(n)), dev(table), n, 1, heads, rank, rot, scale, max_kv_len=max(contexts), force_simt=simt,
                                      sink=None if sinks is None else dev(sinks)))
    for i, c in enumerate(contexts):
        rows = keys[table[i].long(), 0].reshape(-1, width)[:c].double()
        scores = scale * folded[i].double() @ rows.T
        beside = scores if sinks is None else torch.cat([scores, sinks.double()[:, None]], 1)
        want = (beside.softmax(1)[:, :c]) @ rows[:, :rank]
        # a score's error: its `width` products rounded as they are added; a weight's twice that, and two bf16 terms of it (2^-17) on tensor cores;
        # the sums over c keys and up to 64 runs in fp32
        wrong = width * 2.0 ** -24 * scale * (folded[i].double().abs() @ rows.abs().T).max()
        bound = (2 * wrong + 2.0 ** -16 + (c + 64 + 8) * 2.0 ** -24) * rows[:, :rank].abs().max()
        assert (out[i] - want).abs().max() <= bound


# (rows wider than the queries' registers hold, in whole and odd steps; heads beyond a block's 16; contexts split and, with many entries, whole)
@pytest.mark.parametrize("heads, rank, rot, entries", [(17, 512, 128, 3), (5, 512, 80, 150), (16, 384, 16, 2), (33, 64, 16, 160), (4, 192, 112, 1)])
@pytest.mark.parametrize("sink", [False, True])
def test_latent_single_tokens_on_tensor_cores(heads, rank, rot, entries, sink):
    need_gpu()
    from torchinferno_b200.kernels import ops
    page, width = 16, rank + rot
    contexts = [(1, 64, 65, 127, 200, 129)[i % 6] + 64 * (i % 2) for i in range(entries)]
    per = -(-max(contexts) // page)
    keys = dev(rnd(entries * per, 1, page, width, dtype=torch.bfloat16, scale=0.7))
    table = dev(torch.randperm(entries * per, generator=torch.Generator().manual_seed(4)).int().view(entries, per))
    ints = lambda v: dev(torch.tensor(list(v), dtype=torch.int32))
    folded = dev(rnd(entries, heads, width, scale=0.3, seed=1).bfloat16().float())      # (no rounding of the queries between the two kernels)
    error = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, plain = (ops.latent_attention(folded, keys, torch.empty(entries, heads, rank, device="cuda"), ints(range(entries + 1)), ints(c - 1 for c in contexts),
                                       ints(range(entries)), table, entries, 1, heads, rank, rot, 0.11, error, max_kv_len=max(contexts),
                                       sink=dev(rnd(heads, seed=2)) if sink else None, force_simt=simt) for simt in (False, True))
    # the weights enter as two bf16 terms (2^-17 of each), everything else is fp32 sums of at most `width` or 264 numbers
    assert (out - plain).abs().max() <= (2.0 ** -16 + 640 * 2.0 ** -23) * plain.abs().max() and int(error) == 0


@pytest.mark.parametrize("heads, rank, rot, entries", [(17, 512, 224, 3), (5, 512, 256, 150), (16, 384, 384, 2)])
@pytest.mark.parametrize("shift", [0, 1])
def test_latent_single_tokens_of_the_widest_rows_on_tensor_cores(heads, rank, rot, entries, shift):
    """Rows too wide for the sixteen warps' shared memory, and queries off their 16-byte boundaries, take the kernel of four warps: its sums are not the CUDA cores'."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    page, width = 16, rank + rot
    contexts = [(1, 64, 65, 127, 200, 129)[i % 6] + 64 * (i % 2) for i in range(entries)]
    per = -(-max(contexts) // page)
    keys = dev(rnd(entries * per, 1, page, width, dtype=torch.bfloat16, scale=0.7))
    table = dev(torch.randperm(entries * per, generator=torch.Generator().manual_seed(4)).int().view(entries, per))
    ints = lambda v: dev(torch.tensor(list(v), dtype=torch.int32))
    room = torch.empty(entries * heads * width + shift, device="cuda")
    folded = room[shift:].view(entries, heads, width)
    folded.copy_(rnd(entries, heads, width, scale=0.3, seed=1).bfloat16().float())
    error = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, plain = (ops.latent_attention(folded, keys, torch.empty(entries, heads, rank, device="cuda"), ints(range(entries + 1)), ints(c - 1 for c in contexts),
                                       ints(range(entries)), table, entries, 1, heads, rank, rot, 0.11, error, max_kv_len=max(contexts), force_simt=simt) for simt in (False, True))
    assert (out - plain).abs().max() <= (2.0 ** -16 + 900 * 2.0 ** -23) * plain.abs().max() and int(error) == 0
    assert not torch.equal(out, plain)


@pytest.mark.parametrize("tokens, experts, kept, top, groups, keep", [(1, 1, 1, 1, 1, 1), (31, 40, 33, 3, 4, 2), (64, 300, 300, 8, 1, 1), (65, 64, 64, 2, 8, 3)])
def test_choices_and_sorting_in_one_launch(tokens, experts, kept, top, groups, keep):
    """Some choices name no expert (``kept`` of ``experts`` are ones): their place is -1."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    logits, results = dev(rnd(tokens, experts)), []
    for together in (True, False):
        ids, weights = torch.empty(tokens, top, dtype=torch.int32, device="cuda"), torch.empty(tokens, top, device="cuda")
        offsets, order, place = (torch.full((m,), -7, dtype=torch.int32, device="cuda") for m in (kept + 1, tokens * top, tokens * top))
        ops.moe_route(logits, experts, top, ids, weights, groups=groups, keep=keep, sort=(kept, offsets, order, place) if together else None)
        if not together:
            ops.moe_group(ids, kept, offsets, order, place)
        results.append((ids, weights, offsets))
        flat, total = ids.flatten().cpu(), int((ids < kept).sum())
        assert torch.equal(offsets.cpu().long(), torch.cat([torch.zeros(1, dtype=torch.long), torch.bincount(flat[flat < kept].long(), minlength=kept).cumsum(0)]))
        assert torch.equal(flat[order[:total].cpu().long()], flat[flat < kept].sort()[0])
        assert torch.equal(place[order[:total].long()].cpu(), torch.arange(total, dtype=torch.int32)) and (place.cpu()[flat >= kept] == -1).all()
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("missing", [0, 128, 256])
def test_gathered_latent_rows_stay_within_their_buffer(missing):
    """Two entries of 200 and 129 keys need 512 rows; with fewer, what is missing is reported and nothing is written behind the last."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    rank, rot, page, lens = 16, 8, 16, (200, 129)
    pool = dev(rnd(32, 1, page, rank + rot, dtype=torch.bfloat16))
    table = dev(torch.arange(32, dtype=torch.int32).view(2, 16))
    latent_room, rotated_room = (torch.full((512 + 8, w), 7.0, dtype=torch.bfloat16, device="cuda") for w in (rank, rot))
    rows, error = 512 - missing, torch.zeros(1, dtype=torch.int32, device="cuda")
    ints = lambda v: dev(torch.tensor(v, dtype=torch.int32))
    ops.latent_gather(pool, table, ints([0, 50, 51]), ints([150, 128]), ints([0, 1]), 2, 200, latent_room[:rows], rotated_room[:rows], error)
    want = torch.zeros(512, rank + rot, dtype=torch.bfloat16)
    for first, n, at in ((0, lens[0], 0), (256, lens[1], 16)):
        want[first:first + n] = pool[at:at + 16].cpu().view(256, rank + rot)[:n]
    got = torch.cat([latent_room, rotated_room], 1).cpu()
    assert torch.equal(got[:rows], want[:rows]) and (got[rows:] == 7.0).all()
    assert int(error) == (0x60001 if missing else 0)


@pytest.mark.parametrize("rows, width, wide, dtypes, shift", [
    (1, 8, 8, (torch.bfloat16, torch.bfloat16, torch.bfloat16), 0), (7, 520, 1040, (torch.float32, torch.bfloat16, None), 8),
    (296, 2056, 2056, (torch.bfloat16, None, torch.float32), 0), (5, 516, 520, (torch.bfloat16, torch.float32, torch.bfloat16), 0),
    (3, 64, 96, (torch.bfloat16, torch.bfloat16, torch.bfloat16), 1)])      # (the last two: not by eight)
def test_sums_of_two_outputs(rows, width, wide, dtypes, shift):
    """residual += a + b, every sum in 32 bits: the same numbers as torch's, bit for bit."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    a, b = (rnd(rows, wide + shift, dtype=t, seed=s)[:, shift:shift + width] if t else None for s, t in enumerate(dtypes[:2]))
    residual = rnd(rows, width, seed=5)
    copy = torch.empty(rows, width, dtype=dtypes[2], device="cuda") if dtypes[2] else None
    got = dev(residual)
    on = [t if t is None else dev(t._base if t._base is not None else t)[:, shift:shift + width] for t in (a, b)]
    ops.add_pair(got, on[0], on[1], copy)
    want = residual + (a.float() if b is None else a.float() + b.float())
    assert torch.equal(got.cpu(), want)
    assert copy is None or torch.equal(copy.cpu(), want.to(copy.dtype))


@pytest.mark.parametrize("tokens, heads, dim, rank, rot, n_freq, half_pairs, in_place", [
    (1, 1, 8, 8, 8, 4, False, True), (3, 2, 64, 520, 16, 5, False, False), (5, 3, 16, 1032, 24, 8, True, True), (2, 16, 128, 512, 64, 32, True, False),
    (296, 2, 8, 72, 16, 8, True, False), (297, 3, 8, 264, 16, 8, True, True), (301, 5, 24, 512, 64, 32, False, True), (299, 2, 16, 264, 8, 0, False, False)])
def test_latent_rows_in_pieces_are_those_element_by_element(tokens, heads, dim, rank, rot, n_freq, half_pairs, in_place):
    """To the bit, whichever kernel stores a row: the sum of squares is added in one order.  Without a cache nothing is stored; a token whose page is
    out of range is reported, and its neighbours are stored."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    page, width, slots = 16, rank + rot, 3
    per_slot = -(-tokens // slots)
    table = torch.randperm(slots * -(-per_slot // page) + 2, generator=torch.Generator().manual_seed(1))[:slots * -(-per_slot // page)]
    table = dev(table.to(torch.int32).view(slots, -1))
    positions = dev(torch.tensor([t // slots for t in range(tokens)], dtype=torch.int32))
    token_slot = dev(torch.tensor([t % slots for t in range(tokens)], dtype=torch.int32))
    dkv_rows, q_rows = rnd(tokens, width, dtype=torch.bfloat16), rnd(tokens, heads * (dim + rot), dtype=torch.bfloat16, seed=1)
    weight, freq = dev(1 + 0.1 * rnd(rank, seed=2)), dev(rnd(n_freq, seed=3).abs())
    bad = table.clone()
    bad[tokens % slots, 0] = 1 << 20      # (the first page of one slot)
    last = int(table.max()) + 1
    results = []
    for shift in (8, 7):      # (rows off their 16-byte boundaries are taken element by element)
        dkv = dev(torch.zeros(tokens, width + 8, dtype=torch.bfloat16))
        dkv[:, shift:shift + width] = dev(dkv_rows)
        for pages in (table, bad, None):
            q = dev(q_rows.clone())
            keys = None if pages is None else torch.full((last, 1, page, width), -7.0, dtype=torch.bfloat16, device="cuda")
            folded = None if in_place else torch.full((tokens, heads, width), -7.0, device="cuda")
            error = torch.zeros(1, dtype=torch.int32, device="cuda")
            ops.latent_append(dkv[:, shift:shift + width], q, folded, keys, positions, token_slot, pages, weight, 1e-6, freq, heads, dim, rank, rot,
                              half_pairs=half_pairs, error_word=error)
            results.append((keys, q, folded))
            assert (int(error) >> 16 == 2) == (pages is bad and bool((token_slot == tokens % slots).any()))
    for got, want in zip(results[:3], results[3:]):
        for x, y in zip(got, want):
            assert (x is None and y is None) or torch.equal(x, y)
    for cached in results[1:3]:      # (the queries do not depend on the cache)
        assert torch.equal(cached[1], results[0][1]) and (in_place or torch.equal(cached[2], results[0][2]))


@pytest.mark.parametrize("tokens, rows, k", [(2859, 7, 260), (1187, 37, 64), (331, 61, 1028), (157, 129, 2056)])
@pytest.mark.parametrize("dtype", DTYPES)
def test_router_logits_of_six_rows_a_warp_have_the_bits_of_one(tokens, rows, k, dtype):
    need_gpu()
    from torchinferno_b200.kernels import ops
    x, w, bias = dev(rnd(tokens, (k + 7) // 8 * 8, dtype=dtype))[:, :k], dev(rnd(rows, k, seed=1)), dev(rnd(rows, seed=2))
    out = ops.router_logits(x, w, torch.empty(tokens, rows, device="cuda"), bias)
    parts = [ops.router_logits(x[i:i + 100], w, torch.empty(len(x[i:i + 100]), rows, device="cuda"), bias) for i in range(0, tokens, 100)]
    assert tokens * rows >= 20000 > 100 * rows and torch.equal(out, torch.cat(parts))


@pytest.mark.parametrize("entries, dim", [(28, 128), (37, 100), (30, 32)])      # (448 to 592 blocks of heads of 65 to 128: the form with four blocks an SM)
@pytest.mark.parametrize("dtype", DTYPES)
def test_attention_on_cuda_cores_of_many_single_tokens_has_the_bits_of_a_few(entries, dim, dtype):
    need_gpu()
    from torchinferno_b200.kernels import ops
    heads, page, contexts = 16, 16, [1 + 37 * i % 90 for i in range(entries)]
    ints = lambda v: dev(torch.tensor(list(v), dtype=torch.int32))
    pool = dev(rnd(6 * entries, 2, heads, page, dim, dtype=dtype))
    table, q = ints(torch.randperm(6 * entries, generator=torch.Generator().manual_seed(2)).tolist()).view(entries, 6), dev(rnd(entries, heads * dim, dtype=dtype, seed=1))

    def run(first, last):
        n = last - first
        return ops.paged_attention_simt(q[first:last], pool, torch.empty(n, heads * dim, dtype=dtype, device="cuda"), ints(range(n + 1)),
                                        ints(c - 1 for c in contexts[first:last]), ints(range(first, last)), table, n, 1, heads, heads, dim, scale=dim ** -0.5)

    assert torch.equal(run(0, entries), torch.cat([run(0, 15), run(15, entries)]))


# (two and four blocks on the fullest SM and bf16 rows, more than one and fp32 rows: the form with fewer registers; the last the form of large steps)
@pytest.mark.parametrize("tokens, rows, dtype", [(501, 16, torch.bfloat16), (1180, 16, torch.bfloat16), (2049, 9, torch.bfloat16), (603, 9, torch.bfloat16),
                                                 (1183, 16, torch.float32), (1301, 7, torch.float32), (1184, 9, torch.float32)])
def test_router_logits_have_the_bits_of_a_few_tokens_alone(tokens, rows, dtype):
    need_gpu()
    from torchinferno_b200.kernels import ops
    x, w = dev(rnd(tokens, 1032, dtype=dtype)), dev(rnd(rows, 1032, seed=1))
    out = ops.router_logits(x, w, torch.empty(tokens, rows, device="cuda"))
    parts = [ops.router_logits(x[i:i + 100], w, torch.empty(len(x[i:i + 100]), rows, device="cuda")) for i in range(0, tokens, 100)]
    assert tokens * rows < 20000 and torch.equal(out, torch.cat(parts))


def test_router_logits_of_more_rows_than_a_grid_is_high():
    need_gpu()
    from torchinferno_b200.kernels import ops
    x, w = dev(rnd(1, 4)), dev(rnd(36 * 65535 + 1, 4, seed=1))
    out = ops.router_logits(x, w, torch.empty(1, len(w), device="cuda"))
    want = x.double() @ w.double().T
    assert (out.double() - want).abs().max() <= 4 * 2.0 ** -24 * (x.abs().double() @ w.abs().double().T).max()      # (four products, rounded as they are added)


@pytest.mark.parametrize("experts, top", [(1, 1), (31, 4), (32, 32), (33, 3), (64, 6), (65, 8), (256, 8)])
@pytest.mark.parametrize("sigmoid, normalize, corrected", [(False, True, False), (True, False, True)])
def test_choices_of_few_experts_are_the_general_forms(experts, top, sigmoid, normalize, corrected):
    """The same logits beside experts that are never chosen (more than 256 take the general form); equal logits among them."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    tokens, wide = 67, 300
    z = rnd(tokens, experts)
    z[::3, 1::2] = z[::3, 0:2 * (experts // 2):2]                      # (pairs of equals)
    beside = torch.full((tokens, wide - experts), -float("inf"))
    correction = 0.1 * rnd(experts, seed=1) if corrected else None
    results = []
    for logits, extra in ((z, 0), (torch.cat([z, beside], dim=1), wide - experts)):
        ids, weights = torch.empty(tokens, top, dtype=torch.int32, device="cuda"), torch.empty(tokens, top, device="cuda")
        c = None if correction is None else dev(torch.cat([correction, torch.full((extra,), -100.0)]))
        ops.moe_route(dev(logits), logits.shape[1], top, ids, weights, sigmoid_scores=sigmoid, normalize=normalize, norm_eps=1e-20, correction=c)
        results.append((ids, weights))
    assert torch.equal(results[0][0], results[1][0])
    # (the softmax's sum takes the same numbers in the same lanes; zeros change nothing)
    assert torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("pairs, experts", [(1, 1), (1023, 32), (1025, 3), (8191, 256), (8192, 32), (8192, 31), (9001, 256), (16384, 60), (16385, 60), (9000, 257)])
def test_pairs_are_sorted_by_expert(pairs, experts):
    need_gpu()
    from torchinferno_b200.kernels import ops
    ids = torch.randint(-1, experts + 1, (pairs,), generator=torch.Generator().manual_seed(pairs), dtype=torch.int32)      # (some have no expert here)
    offsets, order, place = (torch.full((n,), -9, dtype=torch.int32, device="cuda") for n in (experts + 1, pairs, pairs))
    ops.moe_group(dev(ids), experts, offsets, order, place)
    inside = (ids >= 0) & (ids < experts)
    counts = torch.bincount(ids[inside].long(), minlength=experts)
    assert offsets.tolist() == [0] + counts.cumsum(0).tolist()
    order, place = order.cpu().long(), place.cpu().long()
    assert (place[~inside] == -1).all()
    held = order[:int(inside.sum())]
    assert torch.equal(held.sort().values, inside.nonzero().flatten())                       # every pair once
    assert torch.equal(place[held], torch.arange(len(held))) and (ids[held].long().diff() >= 0).all()


@pytest.mark.parametrize("n, k, many", [(512, 8192, 700), (2048, 4096, 2100), (2050, 2112, 1500), (8190, 2048, 300)])
def test_fp32_product_in_parts_of_k_has_one_order(n, k, many):
    """Parts that blocks of their own sum, and parts that one block sums one after the other: the same bits."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    x, w = dev(rnd(many, k)), dev(rnd(n, k, seed=3))
    apart = [ops.lib().tib_gemm_f32_tcgen05_partial(m, n, k, m) for m in (8, 130, many)]
    assert apart[0] > 0                                                    # (few rows: blocks of their own)
    out = ops.gemm_f32(x, w, torch.empty(many, n, device="cuda"))
    for m in (8, 130):
        assert torch.equal(ops.gemm_f32(x[:m], w, torch.empty(m, n, device="cuda")), out[:m])
    whole = torch.empty(130, n, device="cuda")
    scratch = torch.empty(3 * 130 * k, dtype=torch.bfloat16, device="cuda")
    launches = torch.zeros(1, dtype=torch.int32)
    assert ops.lib().tib_gemm_f32_tcgen05(x.data_ptr(), w.data_ptr(), whole.data_ptr(), 130, n, k, k, k, n, scratch.data_ptr(), 130, 0, 0, 0,
                                          launches.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0      # (no room for the parts' sums)
    assert torch.equal(whole, out[:130]) and int(launches) == 2
    exact = x[:130].double() @ w.double().T
    assert (whole.double() - exact).norm() <= 4e-7 * exact.norm()          # (the bound of the products in one part)


@pytest.mark.parametrize("lens", [[129, 641], [512, 100, 513]])      # (chunks of a request: fewer than four, four, and one more)
def test_scan_of_many_states_folds_each_request_as_alone(lens):
    """Where states are enough for five blocks an SM a thread has four chunks on their way instead of eight: the same chain, to the bit."""
    need_gpu()
    from torchinferno_b200.kernels import ops
    heads, head_dim, state, n = 64, 64, 128, sum(lens)
    blocks = heads * head_dim * state // 1024
    assert blocks * len(lens) >= 5 * 148 > blocks
    inner = heads * head_dim
    xbc, dt = dev(rnd(n, inner + 2 * state, dtype=torch.bfloat16)), dev(rnd(n, heads, dtype=torch.bfloat16, seed=1))
    bias, a_log, skip = dev(rnd(heads, seed=2)), dev(0.2 * rnd(heads, seed=3)), dev(rnd(heads, seed=4))
    held = rnd(len(lens), heads * state * head_dim, seed=5)

    def scan(first, lens, held):
        rows = slice(first, first + sum(lens))
        y, carried = torch.empty(sum(lens), inner, device="cuda"), dev(held.clone())
        starts = dev(torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32))
        ops.ssd_scan(xbc[rows], dt[rows], 0, bias, a_log, skip, carried, starts, dev(torch.arange(len(lens), dtype=torch.int32)), y, len(lens),
                     heads=heads, groups=1, state_dim=state, head_dim=head_dim, max_q_len=max(lens))
        return y, carried

    y, carried = scan(0, lens, held)
    for i, length in enumerate(lens):
        if length <= 128:      # (alone it would not go in chunks)
            continue
        first = sum(lens[:i])
        own, own_state = scan(first, [length], held[i:i + 1])
        assert torch.equal(own, y[first:first + length]) and torch.equal(own_state, carried[i:i + 1])
