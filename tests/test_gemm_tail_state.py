"""What a GEMM whose tiles are cut along K keeps between calls: where it comes from, and the state in which a call finds it."""
import pathlib
import re
import threading

import pytest
import torch

CSRC = pathlib.Path(__file__).resolve().parent.parent / "symm_mem_recipes_b200" / "csrc"
M, N, K = 200, 1280, 4096                          # 10 tiles of 128 columns on 74 pairs: every tile is cut


def test_tail_needs_no_state_and_no_waits():
    """The parts of a cut tile do not wait for one another, so nothing has to be cleared, kept between calls or resident at
    the same time: the GEMM without a gather holds no wait on global memory."""
    source = (CSRC / "kernels" / "ag_matmul_2cta_sm100.cu").read_text()
    waits = re.findall(r"\b(wait_\w+|ld_acquire_\w+|await_\w+)\(", source)
    assert waits == ["wait_reached_acquire_sys"]       # a gathered block of a peer
    assert not re.search(r"counters|marks", (CSRC / "bindings.cpp").read_text())


def test_launches_of_a_cut_gemm_are_counted():
    """What bench.py reports as its launches: 896 tiles on 74 pairs leave 8, which are cut; 74 x 12 tiles leave none."""
    from symm_mem_recipes_b200._ext import C

    assert all(C.gemm_kernels(16384, 3584, 8192, 2, 148, gather) == 2 for gather in (False, True))
    assert all(C.gemm_kernels(74 * 256, 12 * 256, 8192, 2, 148, gather) == 1 for gather in (False, True))
    assert C.gemm_kernels(256, 64, 128, 2, 148, False) == 1      # too short a K to cut


def test_calls_that_are_alive_at_once_share_no_scratch():
    import importlib

    ag = importlib.import_module("symm_mem_recipes_b200.ops.ag_matmul")
    config = ag.AgMatmulConfig(num_sms=148, split_k_tail=True)
    first, second = (ag._tail_buffer(torch.device("cpu"), config) for _ in range(2))
    assert first.data_ptr() != second.data_ptr()
    assert first.nbytes == 74 * 2 * 128 * 256 * 4      # a 256 x 256 fp32 partial on every one of 74 pairs
    kept = [k for k, v in vars(ag).items() if isinstance(v, dict) and "scratch" in k]
    assert not kept, "state that symm_mem.reset() does not know of"
    assert ag._tail_buffer(torch.device("cpu"), ag.AgMatmulConfig(num_sms=148, split_k_tail=False)) is None


def _operands():
    gen = torch.Generator(device="cuda").manual_seed(7)
    a = (torch.randn(M, K, generator=gen, device="cuda") * 0.5).to(torch.bfloat16)
    b = (torch.randn(N, K, generator=gen, device="cuda") * 0.1).to(torch.bfloat16)
    return a, b, a.float() @ b.float().t()


def _cut_gemm(a, b):
    from symm_mem_recipes_b200._ext import C

    return C.matmul_local(a, b, None, 0, None, 0, 0, True, 0, 2_000_000_000, 0)


def _matches(c, want):
    return bool(((c.float() - want).abs() <= want.abs() * 2.0 ** -6 + 2e-2).all())


@pytest.mark.gpu
def test_first_cut_call_on_a_stream_while_the_default_stream_is_busy():
    from symm_mem_recipes_b200.parallel import symm_mem

    a, b, want = _operands()
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):                # what the allocator hands out next on this stream is not zero
        poison = [torch.full((n,), 0x01010101, dtype=torch.int32, device="cuda") for n in (1024, 1 << 20, 4 << 20) for _ in range(4)]
        del poison
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)                 # about 50 ms on the default stream
    with torch.cuda.stream(stream):
        got = [_cut_gemm(a, b) for _ in range(3)]
    torch.cuda.synchronize()
    symm_mem.check_status("cuda")
    assert all(_matches(c, want) for c in got)


@pytest.mark.gpu
def test_cut_call_while_another_thread_captures():
    a, b, want = _operands()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):                # kernels loaded, output and scratch in the allocator's cache
        _cut_gemm(a, b)                            # (without torch.cuda.graph below, which would empty it)
    torch.cuda.synchronize()
    x = torch.ones(16, device="cuda")
    out, errors = [], []

    def call():
        try:
            with torch.cuda.stream(stream):
                out.append(_cut_gemm(a, b))
        except Exception as e:  # noqa: BLE001 - reported by the assertion below
            errors.append(e)

    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        graph.capture_begin(capture_error_mode="global")
        y = x + 1
        t = threading.Thread(target=call)
        t.start()
        t.join()
        y = y * 2
        graph.capture_end()
    assert not errors, errors
    graph.replay()
    torch.cuda.synchronize()
    assert bool((y == 4).all()) and _matches(out[0], want)


@pytest.mark.gpu
@pytest.mark.parametrize("traced", [False, True])
def test_calls_in_a_row_and_replayed(traced):
    """Both bindings, again and again on one scratch, eagerly and from a graph."""
    import symm_mem_recipes_b200 as smr
    from symm_mem_recipes_b200._ext import C
    from symm_mem_recipes_b200.parallel import symm_mem

    a, b, want = _operands()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    trace = torch.zeros(sms, 12, dtype=torch.int64, device="cuda") if traced else None
    scratch = torch.empty(sms * 128 * 256 * 4, dtype=torch.uint8, device="cuda")

    def call():
        if not traced:
            return smr.matmul(a, b)
        c = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")          # the binding of the gather, with a record
        C.ag_matmul(a, b, c, 0, None, 0, None, 128, sms, 2_000_000_000, scratch, 0, trace)
        return c

    graph = torch.cuda.CUDAGraph()
    call()
    with torch.cuda.graph(graph):
        c = call()
    for _ in range(3):
        c.zero_()
        graph.replay()
        assert _matches(c, want) and _matches(call(), want)
    symm_mem.check_status("cuda")


@pytest.mark.gpu
def test_cut_calls_of_two_priorities_at_once():
    """Cut GEMMs as wide as the GPU on streams of two priorities, started while another kernel holds some of the SMs."""
    from symm_mem_recipes_b200.parallel import symm_mem

    a, b, want = _operands()
    low, high = torch.cuda.Stream(priority=0), torch.cuda.Stream(priority=-1)
    filler = torch.randn(2048, 2048, device="cuda")
    torch.cuda.synchronize()
    got = []
    for _ in range(20):
        filler = (filler @ filler).clamp_(-1, 1)   # on the default stream: its end frees SMs one after the other
        for stream in (low, high, low, high):
            with torch.cuda.stream(stream):
                got.append(_cut_gemm(a, b))
    torch.cuda.synchronize()
    symm_mem.check_status("cuda")
    assert all(_matches(c, want) for c in got)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,block_n,sms,epilogue,dtype", [
    (129, 136, 1024, 128, 0, 0, torch.bfloat16), (300, 1000, 2048, 192, 0, 0, torch.bfloat16),
    (257, 520, 4096, 256, 0, 0, torch.bfloat16), (130, 464, 1160, 224, 0, 0, torch.bfloat16),
    (300, 2000, 1024, 256, 0, 2, torch.bfloat16), (300, 768, 1024, 0, 0, 1, torch.bfloat16),
    (129, 144, 4096, 128, 0, 0, torch.float8_e4m3fn), (300, 976, 2064, 192, 0, 0, torch.float8_e4m3fn),
    (600, 464, 4096, 224, 0, 0, torch.float8_e4m3fn)])
@pytest.mark.parametrize("splits", [2, 3, 8])
def test_cut_tiles_equal_uncut_ones(m, n, k, block_n, sms, epilogue, dtype, splits):
    """Every width, end and type of the cut path at ragged edges, cut into as many parts as asked for or as there are
    pairs (K 1160 in eight: the last part is empty).  The same products in another order of fp32 sums: a
    result may round to the neighbouring bf16 (2^-8 of it) or e4m3 (2^-3) number, and beside that differ by what
    cancels, k * 2^-24 of a sum of k terms of 0.05."""
    from symm_mem_recipes_b200._ext import C
    from symm_mem_recipes_b200.parallel import symm_mem
    from symm_mem_recipes_b200.utils.testing import guarded_empty

    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = (torch.randn(m, k, generator=gen, device="cuda") * 0.5).to(dtype)
    b = (torch.randn(n, k, generator=gen, device="cuda") * 0.1).to(dtype)
    n_out, es = n // 2 if epilogue else n, a.element_size()
    width = block_n or 256
    tiles, pairs = -(-m // 256) * -(-n_out // (width // 2 if epilogue else width)), torch.cuda.get_device_properties(0).multi_processor_count // 2
    parts = min(splits, pairs // tiles)            # every tile is cut: they are fewer than half of the pairs
    assert C.matmul_plan(m, n, k, es, epilogue, block_n, 2 * pairs, -splits) == (width, parts, 0) and parts >= 2
    residuals = [None]
    if dtype == torch.bfloat16 and not epilogue and block_n != 224:
        residuals.append(torch.randn(m, n, generator=gen, device="cuda").to(dtype))
    for residual in residuals:
        if dtype == torch.bfloat16:
            c, intact = guarded_empty((m, n_out), dtype, "cuda")
            c.fill_(float("nan"))
        else:
            c, intact = torch.empty(m, n_out, dtype=dtype, device="cuda"), lambda: True
        whole = C.matmul_local(a, b, None, epilogue, residual, block_n, sms, False, 0, 2_000_000_000, 1)
        assert C.matmul_local(a, b, c, epilogue, residual, block_n, sms, True, 0, 2_000_000_000, -splits) is not None
        symm_mem.check_status("cuda")
        ulp = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -3
        x, y = c.float(), whole.float()
        product = torch.maximum(x.abs(), y.abs())
        if residual is not None:                   # rounded before the residual is added, and once more after
            product = torch.maximum(product, torch.maximum((x - residual.float()).abs(), (y - residual.float()).abs())) * 2
        assert bool(((x - y).abs() <= product * ulp + 0.05 * k * 2.0 ** -22).all())
        assert intact(), "the kernel stored outside its output"
