"""Attention of the token counts where both kernels are launched and the mask decides which one works, with the KV range of the per-token one
uncut, cut into clusters, and cut for the combine pass; prompts (whose tokens share their cells), tokens with cells of their own, and masks with
values beside 0 and -inf; against f64.

Tolerance: f16 inputs are exact in f64, Q is rounded to f16 here as there; what is left are f32 sums and P as an f16 pair (2^-22)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# heads, KV heads, tokens, cells: clusters of 3; two splits beyond one wave; one; 9 query heads per KV head (not for the tiled kernel) in clusters of 2
@pytest.mark.parametrize("H,Hkv,Nq,n_kv", [(8, 1, 128, 2048), (8, 2, 140, 1536), (8, 8, 200, 1024), (16, 8, 130, 1024), (18, 2, 30, 1280), (9, 1, 60, 1024)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("kind", ["prompt", "own", "soft"])
def test_both_kernels_launched(H, Hkv, Nq, n_kv, D, kind):
    from cactus_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(H + Nq + D)
    q = torch.randn((Nq, H, D), device="cuda", generator=g)
    k, v = (torch.randn((n_kv, Hkv, D), device="cuda", generator=g).half() for _ in range(2))
    cell, tok = torch.arange(n_kv, device="cuda")[None], torch.arange(Nq, device="cuda")[:, None]
    mask = torch.full((Nq, n_kv), float("-inf"), dtype=torch.float16, device="cuda")
    if kind == "prompt":
        mask[cell <= n_kv - Nq + tok] = 0
    elif kind == "own":
        mask[cell // 8 % (n_kv // 8) == tok * 7 % (n_kv // 8)] = 0          # a few cells of its own each, spread over the range
        mask[cell % n_kv == (tok * 37 + 5) % n_kv] = 0
    else:
        mask = torch.randn((Nq, n_kv), device="cuda", generator=g).half()
        mask[cell > n_kv - Nq + tok] = float("-inf")
    out = ops.flash_attn_ext(q, k, v, mask, D ** -0.5)
    s = torch.einsum("jhd,chd->jhc", q.half().double(), k.double().repeat_interleave(H // Hkv, 1)) * D ** -0.5 + mask.double()[:, None]
    want = torch.einsum("jhc,chd->jhd", torch.softmax(s, -1), v.double().repeat_interleave(H // Hkv, 1))
    assert float((out - want).abs().max() / want.abs().max()) < 2e-5
