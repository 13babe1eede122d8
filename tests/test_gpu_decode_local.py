"""The rank-local GEMV and the decode step built on it, at the edges of their tilings."""
import pytest
import torch


def _normal(gen, *shape, std=1.0):
    return (torch.randn(*shape, generator=gen) * std).to(torch.bfloat16).cuda()


@pytest.mark.gpu
@pytest.mark.parametrize("nk", [True, False])
@pytest.mark.parametrize("B,K,N", [(1, 8, 8), (2, 72, 136), (16, 8192, 1280), (5, 1000, 328), (7, 4096, 520),
                                   (16, 200, 20008), (1, 3584, 8192)])
def test_gemv_tile_edges(B, K, N, nk):
    import symm_mem_recipes_b200 as smr
    from symm_mem_recipes_b200.parallel import symm_mem
    from symm_mem_recipes_b200.utils.testing import guarded_empty

    gen = torch.Generator().manual_seed(B + K + N)
    x, w = _normal(gen, B, K), _normal(gen, N, K, std=0.05)
    out, intact = guarded_empty((B, N), torch.bfloat16, "cuda")
    ref = x.double() @ w.double().t()
    for _ in range(2):                     # back to back: the second starts under the first
        out.fill_(float("nan"))
        smr.gemv(x, w, out, weights_nk=True) if nk else smr.gemv(x, w.t().contiguous(), out)
    symm_mem.check_status("cuda")
    assert intact(), "the kernel stored outside its output"
    assert bool(((out.double() - ref).abs() <= ref.abs() * 2.0 ** -7 + 2e-2).all())
