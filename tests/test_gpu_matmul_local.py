"""The GEMM without a gather through its native call: tile widths, K splits of a short last wave, the three
epilogues, ragged edges; and calls on several streams at once."""
import pytest
import torch


def _operands(M, N, K, dtype=torch.bfloat16):
    gen = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, generator=gen, device="cuda") * 0.5
    b = torch.randn(N, K, generator=gen, device="cuda") * 0.1
    return a.to(dtype), b.to(dtype)


def _run(a, b, out=None, epilogue=0, residual=None, block_n=0, splits=0, sms=0):
    from symm_mem_recipes_b200._ext import C

    return C.matmul_local(a, b, out, epilogue, residual, block_n, sms, True, 0, 2_000_000_000, splits)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (17, 520, 1024), (129, 1280, 2048), (300, 264, 4104), (2049, 272, 1000)])
@pytest.mark.parametrize("block_n,sms", [(0, 0), (128, 64), (192, 0), (256, 24), (224, 0)])
def test_tiles_splits_and_residual(M, N, K, block_n, sms):
    from symm_mem_recipes_b200.parallel import symm_mem
    from symm_mem_recipes_b200.utils.testing import guarded_empty

    a, b = _operands(M, N, K)
    ref = a.float() @ b.float().t()
    res = (torch.randn(M, N, device="cuda")).to(torch.bfloat16)
    for r in (None, res):
        if r is not None and block_n == 224:
            continue                                     # the launcher refuses it: no whole boxes of C
        c, intact = guarded_empty((M, N), torch.bfloat16, "cuda")
        for _ in range(2):                               # the second call finds the scratch as the first left it
            c.fill_(float("nan"))
            assert _run(a, b, c, residual=r, block_n=block_n, sms=sms) is not None
        symm_mem.check_status("cuda")
        want = ref if r is None else ref + r.float()
        assert bool(((c.float() - want).abs() <= want.abs() * 2.0 ** -6 + 2e-2).all())
        assert intact(), "the kernel stored outside its output"


@pytest.mark.gpu
@pytest.mark.parametrize("M,F,K", [(1, 8, 64), (130, 1000, 2048), (700, 3584, 1024), (2048, 3584, 512)])
def test_swiglu_of_separate_and_interleaved_halves(M, F, K):
    from symm_mem_recipes_b200.ops import interleave_gate_up
    from symm_mem_recipes_b200.parallel import symm_mem

    a, b = _operands(M, 2 * F, K)
    g, u = (a.float() @ b.float().t()).split(F, dim=1)
    want = torch.nn.functional.silu(g) * u
    outs = [_run(a, b, epilogue=2)]
    if F % 128 == 0:
        outs.append(_run(a, interleave_gate_up(b[:F], b[F:]), epilogue=1))
    symm_mem.check_status("cuda")
    for c in outs:
        assert bool(((c.float() - want).abs() <= want.abs() * 2.0 ** -6 + 2e-2).all())


@pytest.mark.gpu
@pytest.mark.parametrize("M,F,K", [(129, 7168, 2048), (509, 3584, 2048), (385, 6984, 1032)])
def test_swiglu_in_narrower_tiles(M, F, K):
    """Sizes at which tiles of 112 gate and 112 up columns fill the pairs better; the last one ends inside a tile."""
    from symm_mem_recipes_b200._ext import C
    from symm_mem_recipes_b200.parallel import symm_mem
    from symm_mem_recipes_b200.utils.testing import guarded_empty

    assert C.matmul_plan(M, 2 * F, K, epilogue=2) == (224, 1, 0)
    a, b = _operands(M, 2 * F, K)
    g, u = (a.float() @ b.float().t()).split(F, dim=1)
    want = torch.nn.functional.silu(g) * u
    c, intact = guarded_empty((M, F), torch.bfloat16, "cuda")
    c.fill_(float("nan"))
    assert _run(a, b, c, epilogue=2) is not None
    symm_mem.check_status("cuda")
    assert bool(((c.float() - want).abs() <= want.abs() * 2.0 ** -6 + 2e-2).all())
    assert intact(), "the kernel stored outside its output"


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,sms,units,left", [
    (256, 1024, 5120, 4, 2, 0),       # one wave of units, nothing left
    (511, 1520, 5128, 8, 4, 4),       # a ragged row and column; a wave of single tiles after the units
    (700, 2320, 5184, 8, 12, 6),      # three rows of ten columns, the last one 16 wide
    (1290, 2304, 5120, 8, 24, 6),     # nine columns: the odd one comes last, and its last two tiles are the tail
    (769, 1296, 6200, 4, 12, 0),      # the last row of tiles with one row of C, the last column 16 wide
])
def test_two_tiles_at_a_time(M, N, K, sms, units, left):
    """Uncut, the same products in the same order as one tile at a time: the same bits.  And with the tail cut in two."""
    from symm_mem_recipes_b200._ext import C
    from symm_mem_recipes_b200.parallel import symm_mem
    from symm_mem_recipes_b200.utils.testing import guarded_empty

    a, b = _operands(M, N, K)
    ref = a.float() @ b.float().t()
    res = (torch.randn(M, N, device="cuda")).to(torch.bfloat16)
    gate, up = ref.split(N // 2, dim=1)
    tail = left % (sms // 2)
    for epilogue, residual, want in [(0, None, ref), (0, res, ref + res.float()), (2, None, torch.nn.functional.silu(gate) * up)]:
        def plan(sms, splits):
            return C.matmul_plan(M, N, K, 2, epilogue, 256, sms, splits, residual is not None)

        one = _run(a, b, epilogue=epilogue, residual=residual, block_n=256, sms=64, splits=1)
        assert plan(64, 1) == (256, 1, 0)                # 32 pairs: no whole wave of units
        for splits in (1, -2):
            c, intact = guarded_empty(tuple(want.shape), torch.bfloat16, "cuda")
            c.fill_(float("nan"))
            assert plan(sms, splits) == (256, 2 if splits < 0 and tail else 1, units)
            assert _run(a, b, c, epilogue=epilogue, residual=residual, block_n=256, sms=sms, splits=splits) is not None
            symm_mem.check_status("cuda")
            # a bf16 rounding is 2^-9 of the value (two with a residual); the sums of 5000 products of 0.05 differ by 1e-4
            assert bool(((c.float() - want).abs() <= want.abs() * 2.0 ** -6 + 2e-2).all())
            assert intact(), "the kernel stored outside its output"
            assert splits < 0 or torch.equal(c, one)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,epilogue", [
    (509, 1280, 8192, None),          # narrow tiles, all cut along K
    (1240, 8192, 3584, None),         # 192 columns, three rounds
    (2048, 5120, 5120, None), (2048, 5120, 5120, "swiglu"), (1100, 8200, 5120, None),   # two tiles at a time
])
def test_a_record_is_of_the_kernel_that_runs(M, N, K, epilogue):
    """The CTAs and pieces of work in a timing record are those of the plan, and the result is the same to the bit."""
    import symm_mem_recipes_b200 as smr
    from symm_mem_recipes_b200._ext import C
    from symm_mem_recipes_b200.ops.ag_matmul import TRACE_FIELDS

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    pairs = sms // 2
    width, parts, units = C.matmul_plan(M, N, K, epilogue=1 if epilogue else 0, num_sms=sms)
    assert (units > 0) == (K == 5120)
    a, b = _operands(M, N, K)
    trace = torch.zeros(sms, len(TRACE_FIELDS), dtype=torch.int64, device="cuda")
    got = smr.matmul(a, b, epilogue=epilogue, trace=trace)
    assert torch.equal(got, smr.matmul(a, b, epilogue=epilogue))
    tiles = -(-M // 256) * -(-N // width)
    cut = tiles % pairs if parts > 1 else 0
    record = dict(zip(TRACE_FIELDS, trace.cpu().unbind(1)))
    assert int((record["start"] > 0).sum()) == 2 * (tiles * parts if cut == tiles else min(tiles, pairs))
    assert int(record["tiles"].sum()) == 2 * (tiles - cut + cut * parts)
    ran = record["start"] > 0
    assert bool((record["end"] >= record["tiles_done"])[ran].all()) and bool((record["tiles_done"] > record["start"])[ran].all())


@pytest.mark.gpu
def test_split_calls_on_several_streams():
    """Calls whose tiles are cut along K share no scratch across streams."""
    from symm_mem_recipes_b200.parallel import symm_mem

    from symm_mem_recipes_b200._ext import C

    cases = [_operands(M, 1280, 4096) for M in (64, 200, 250)]
    assert all(C.matmul_plan(*a.shape[:1], 1280, 4096, num_sms=48)[1] > 1 for a, _ in cases)
    want = [a.float() @ b.float().t() for a, b in cases]
    streams = [torch.cuda.Stream() for _ in cases]
    torch.cuda.synchronize()
    got = []
    for _ in range(4):
        for (a, b), st in zip(cases, streams):
            with torch.cuda.stream(st):
                got.append(_run(a, b, sms=48))           # three of them fit the GPU side by side
    torch.cuda.synchronize()
    symm_mem.check_status("cuda")
    for i, c in enumerate(got):
        ref = want[i % len(cases)]
        assert bool(((c.float() - ref).abs() <= ref.abs() * 2.0 ** -6 + 2e-2).all())


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 16, 17, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("N,K", [(16, 8), (1280, 2048), (2816, 600), (4096, 72), (8192, 520)])
def test_few_rows(M, N, K):
    """Where the weights are streamed past a few rows: paddings of the batch, K splits, partial tiles, the three ends."""
    from symm_mem_recipes_b200.ops import interleave_gate_up
    from symm_mem_recipes_b200.parallel import symm_mem
    from symm_mem_recipes_b200.utils.testing import guarded_empty

    a, b = _operands(M, N, K)
    ref = a.float() @ b.float().t()
    res = torch.randn(M, N, device="cuda").to(torch.bfloat16)
    g, u = ref.split(N // 2, dim=1)
    swiglu = torch.nn.functional.silu(g) * u
    runs = [(b, 0, None, ref), (b, 0, res, ref + res.float()), (b, 2, None, swiglu)]
    if N % 256 == 0:
        runs.append((interleave_gate_up(b[: N // 2], b[N // 2:]), 1, None, swiglu))
    for w, epilogue, r, want in runs:
        c, intact = guarded_empty(tuple(want.shape), torch.bfloat16, "cuda")
        for _ in range(2):
            c.fill_(float("nan"))
            assert _run(a, w, c, epilogue=epilogue, residual=r) is not None
        symm_mem.check_status("cuda")
        assert bool(((c.float() - want).abs() <= want.abs() * 2.0 ** -6 + 2e-2).all())
        assert intact(), "the kernel stored outside its output"
