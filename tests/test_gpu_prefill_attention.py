"""The short-prompt attention of the rank-local prefill, at the edges of its 16-row tiles and its warps' turns."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("B,S,hq,hkv,D", [(1, 1, 1, 1, 64), (3, 15, 4, 2, 128), (1, 16, 8, 1, 128), (2, 17, 3, 3, 64),
                                          (1, 64, 8, 2, 128), (1, 65, 16, 1, 128), (2, 509, 8, 1, 128), (1, 2048, 2, 1, 64)])
def test_matches_fp32_attention(B, S, hq, hkv, D):
    from symm_mem_recipes_b200._ext import C

    gen = torch.Generator().manual_seed(S + hq)
    qkv = torch.randn(B * S, (hq + 2 * hkv) * D, generator=gen).to(torch.bfloat16).cuda()
    q, k, v = (t.transpose(1, 2) for t in qkv.float().view(B, S, hq + 2 * hkv, D).split([hq, hkv, hkv], dim=2))
    ref = torch.nn.functional.scaled_dot_product_attention(q, k, v, is_causal=True, enable_gqa=True)
    ref = ref.transpose(1, 2).reshape(B * S, hq * D)
    got = C.prefill_attention(qkv, B, S, hq, hkv).float()
    assert (got - ref).norm() <= 4e-3 * ref.norm()
    assert bool(((got - ref).abs() <= ref.abs() * 2.0 ** -6 + 2e-2).all())
