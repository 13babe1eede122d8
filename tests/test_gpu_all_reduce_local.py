"""One-shot all-reduce in a world of one: edges of its chunks and of its streaming stores."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("numel", [8, 8192 - 8, 8192 + 8, (1 << 24) - 8, (1 << 24), (1 << 25) + 8 * 1025])
@pytest.mark.parametrize("write_back", [False, True])
def test_adds_zero_and_nothing_else(numel, write_back):
    import symm_mem_recipes_b200 as smr
    from symm_mem_recipes_b200.parallel import symm_mem
    from symm_mem_recipes_b200.utils.testing import guarded_empty

    t = symm_mem.empty(numel, dtype=torch.bfloat16, device="cuda")
    t.copy_(torch.randn(numel, device="cuda"))
    t[::7] = -0.0
    symm_mem.rendezvous(t)
    want = t.clone() + 0.0
    out, intact = guarded_empty((numel,), torch.bfloat16, "cuda")
    smr.one_shot_all_reduce(t, out=out, write_back=write_back)
    symm_mem.check_status("cuda")
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))
    assert not write_back or torch.equal(t.view(torch.int16), want.view(torch.int16))
    assert intact(), "the kernel stored outside its output"
    symm_mem.free(t)
