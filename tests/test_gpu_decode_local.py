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
@pytest.mark.parametrize("n_layers,B,hidden,heads,kv,D,ffn,s_max,pos", [
    (1, 1, 512, 4, 1, 64, 512, 32, 0), (2, 3, 512, 8, 1, 128, 576, 40, 15), (1, 16, 1024, 8, 2, 128, 1536, 300, 257),
    (3, 5, 256, 3, 1, 64, 320, 4096, 4095), (1, 16, 512, 64, 16, 64, 512, 64, 40), (9, 2, 512, 4, 1, 128, 512, 64, 33),
    (2, 2, 8192, 8, 1, 128, 3584, 2048, 1000),
    (1, 16, 512, 8, 1, 128, 512, 4100, 4097), (1, 16, 512, 2, 1, 64, 512, 4100, 4090)])   # five tiles of positions a warp
def test_decode_step_matches_the_composition(n_layers, B, hidden, heads, kv, D, ffn, s_max, pos):
    """The persistent step against the layers composed of library GEMMs and PyTorch attention."""
    from symm_mem_recipes_b200.models.llama_tp_layer import LlamaTPConfig, LlamaTPDecoderLayer, decode_local
    from symm_mem_recipes_b200.parallel import symm_mem

    dev = torch.device("cuda", 0)
    cfg = LlamaTPConfig(hidden=hidden, n_heads=heads, n_kv_heads=kv, head_dim=D, ffn=ffn)
    layers = [LlamaTPDecoderLayer(cfg, dev, seed=3 + i) for i in range(n_layers)]
    gen = torch.Generator().manual_seed(B + hidden + pos)
    x = _normal(gen, B, hidden, std=0.5)
    caches = [(_normal(gen, B, s_max, kv, D), _normal(gen, B, s_max, kv, D)) for _ in layers]
    mine, theirs = ([(k.clone(), v.clone()) for k, v in caches] for _ in range(2))
    got = decode_local(layers, mine, x, pos)
    symm_mem.check_status(dev)
    assert got is not None, "these shapes are meant for the persistent step"
    again = decode_local(layers, mine, x, torch.tensor([pos], dtype=torch.int32, device=dev))
    symm_mem.check_status(dev)
    assert torch.equal(got, again)
    want = x
    for layer, (kc, vc) in zip(layers, theirs):
        want = layer.decode(want, kc, vc, pos, fused=False)
    assert (got.float() - want.float()).norm() < 1e-2 * want.float().norm()
    other = torch.ones(s_max, dtype=torch.bool, device=dev)
    other[pos] = False
    for (ka, va), (kb, vb), (kc, vc) in zip(mine, theirs, caches):
        for a, b, c in ((ka, kb, kc), (va, vb, vc)):
            assert (a.float() - b.float()).norm() < 1e-2 * b.float().norm()
            assert torch.equal(a[:, other], c[:, other]), "only the new position may change"
