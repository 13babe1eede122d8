"""What a GEMM whose tiles are cut along K keeps between calls: where it comes from, and the state in which a call finds it."""
import pathlib
import re
import threading

import pytest
import torch

CSRC = pathlib.Path(__file__).resolve().parent.parent / "symm_mem_recipes_b200" / "csrc"
M, N, K = 200, 1280, 4096                          # 10 tiles of 128 columns on 74 pairs: every tile is cut


def test_marks_are_not_cleared_on_the_legacy_stream():
    """cudaMemset runs on the legacy stream: it is not ordered before a kernel on a non-blocking stream, and it waits
    behind whatever the default stream has queued."""
    source = (CSRC / "bindings.cpp").read_text()
    assert not re.findall(r"cudaMemset\([^;]*(counters|marks)", source)
    assert not re.findall(r"cudaMalloc\([^;]*(counters|marks)", source)


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
    from symm_mem_recipes_b200._ext import C
    from symm_mem_recipes_b200.parallel import symm_mem

    a, b, want = _operands()
    C.release_tail_marks()
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):                # what the allocator hands out next on this stream is not zero
        poison = [torch.full((1024,), 0x01010101, dtype=torch.int32, device="cuda") for _ in range(32)]
        del poison
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)                 # about 50 ms on the default stream
    with torch.cuda.stream(stream):
        got = [_cut_gemm(a, b) for _ in range(3)]
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):                # and nothing that was queued late has touched the marks
        got.append(_cut_gemm(a, b))
    torch.cuda.synchronize()
    symm_mem.check_status("cuda")
    assert all(_matches(c, want) for c in got)


@pytest.mark.gpu
def test_first_cut_call_while_another_thread_captures():
    """The buffers that a first call makes do not break a capture in progress elsewhere in the process."""
    from symm_mem_recipes_b200._ext import C

    a, b, want = _operands()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):                # kernels loaded, output and scratch in the allocator's cache
        _cut_gemm(a, b)                            # (without torch.cuda.graph below, which would empty it)
    torch.cuda.synchronize()
    C.release_tail_marks()
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
def test_call_after_one_that_gave_up(traced):
    """Whatever part of its marks a call that gave up has left, the next one waits for its own parts."""
    import symm_mem_recipes_b200 as smr
    from symm_mem_recipes_b200._ext import C
    from symm_mem_recipes_b200.parallel import symm_mem

    a, b, want = _operands()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    trace = torch.zeros(sms, 12, dtype=torch.int64, device="cuda") if traced else None   # a record takes the other binding
    C.release_tail_marks()
    for left in (lambda w: w.zero_(), lambda w: w.fill_(int(w.max())), lambda w: w[::2].zero_(), lambda w: w[1::3].sub_(1)):
        assert _matches(smr.matmul(a, b, trace=trace), want)
        (words,) = C.tail_marks_in_use()
        assert int(words.max()) > 0, "the call was not cut"
        left(words)
        assert _matches(smr.matmul(a, b, trace=trace), want)
    symm_mem.check_status("cuda")
    symm_mem.reset()
    assert C.tail_marks_in_use() == []


@pytest.mark.gpu
def test_captured_cut_call_replays():
    from symm_mem_recipes_b200.parallel import symm_mem

    a, b, want = _operands()
    _cut_gemm(a, b)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        c = _cut_gemm(a, b)
    for _ in range(3):
        c.zero_()
        graph.replay()
        assert _matches(c, want) and _matches(_cut_gemm(a, b), want)
    symm_mem.check_status("cuda")
