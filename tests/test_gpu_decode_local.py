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


@pytest.mark.gpu
@pytest.mark.parametrize("B,hidden,heads,kv,D,ffn,s_max,pos", [
    (1, 512, 4, 1, 64, 512, 32, 0), (3, 512, 8, 1, 128, 520, 40, 15), (16, 1024, 8, 2, 128, 1544, 300, 257),
    (5, 264, 3, 1, 64, 264, 4096, 4095), (2, 8192, 8, 1, 128, 3584, 2048, 1000)])
def test_decode_step_matches_the_composition(B, hidden, heads, kv, D, ffn, s_max, pos):
    """Five fused launches against the layer composed of library GEMMs and PyTorch attention."""
    from symm_mem_recipes_b200.models.llama_tp_layer import LlamaTPConfig, LlamaTPDecoderLayer
    from symm_mem_recipes_b200.parallel import symm_mem

    dev = torch.device("cuda", 0)
    cfg = LlamaTPConfig(hidden=hidden, n_heads=heads, n_kv_heads=kv, head_dim=D, ffn=ffn)
    layer = LlamaTPDecoderLayer(cfg, dev, seed=3)
    gen = torch.Generator().manual_seed(B + hidden + pos)
    x = _normal(gen, B, hidden, std=0.5)
    kc, vc = _normal(gen, B, s_max, kv, D), _normal(gen, B, s_max, kv, D)
    ka, va, kb, vb = kc.clone(), vc.clone(), kc.clone(), vc.clone()
    got = layer.decode_local(x, None, ka, va, pos)
    assert got is not None, "these shapes are meant for the fused step"
    again = layer.decode_local(x, None, ka, va, torch.tensor([pos], dtype=torch.int32, device=dev))
    want = layer.decode(x, kb, vb, pos, fused=False)
    symm_mem.check_status(dev)
    assert torch.equal(got[0], again[0]) and torch.equal(got[1].sum(0)[:B], again[1].sum(0)[:B])
    assert (got[0].float() - want.float()).norm() < 1e-2 * want.float().norm()
    assert torch.allclose(got[1].sum(0)[:B], got[0].float().pow(2).sum(1), rtol=1e-4)
    assert torch.allclose(va.float(), vb.float(), rtol=2e-2, atol=2e-2)
    assert torch.allclose(ka.float(), kb.float(), rtol=2e-2, atol=2e-2)
    other = torch.ones(s_max, dtype=torch.bool, device=dev)
    other[pos] = False
    assert torch.equal(ka[:, other], kc[:, other]) and torch.equal(va[:, other], vc[:, other]), "only the new position may change"
