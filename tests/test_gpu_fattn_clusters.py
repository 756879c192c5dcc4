"""KV splits as clusters of 2 to 8 CTAs whose result is quantised, and with two groups of query heads per KV head: against f64, and the quantised
form against the quantiser on the f32 result, byte for byte (a column tile's padding included).

Tolerance: f16 inputs are exact in f64, Q is rounded to f16 here as there; what is left are f32 sums and P as an f16 pair (2^-22)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# 8 KV heads in 4096 cells: 7, 6, 5, 4, 3, 2 splits and no longer any; two groups of heads (9 and 16 query heads per KV head): 8, 3 and 2 splits
@pytest.mark.parametrize("H,Hkv,Nq", [(32, 8, 6), (16, 8, 7), (32, 8, 8), (32, 8, 10), (8, 8, 13), (32, 8, 27), (32, 8, 37), (18, 2, 5), (18, 2, 30), (64, 4, 23)])
@pytest.mark.parametrize("D", [64, 128])
def test_quantised_clusters(H, Hkv, Nq, D):
    from cactus_b200._lib import check, lib
    L, n_kv = lib(), 4096
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(H + Nq + D)
    q = torch.randn((Nq, H, D), device="cuda", generator=g)
    k, v = (torch.randn((n_kv, Hkv, D), device="cuda", generator=g).half() for _ in range(2))
    lens = torch.randint(1, n_kv + 1, (Nq, 1), device="cuda", generator=g)
    lens[0] = 1        # one split that holds anything, seven that hold nothing
    lens[Nq - 1] = n_kv
    mask = torch.full((Nq, n_kv), float("-inf"), dtype=torch.float16, device="cuda")
    mask[torch.arange(n_kv, device="cuda")[None] < lens] = 0
    index = torch.empty(L.b200_mask_index_bytes(Nq, n_kv), dtype=torch.uint8, device="cuda")
    check(L.b200_mask_index_build(mask.data_ptr(), n_kv * 2, Nq, n_kv, index.data_ptr(), index.numel(), st))
    scratch = torch.empty(max(256, L.b200_flash_attn_scratch_bytes(D, H, Hkv, Nq, n_kv)), dtype=torch.uint8, device="cuda")
    args = (D, H, Hkv, Nq, n_kv, q.data_ptr(), H * D * 4, D * 4, k.data_ptr(), Hkv * D * 2, D * 2, v.data_ptr(), Hkv * D * 2, D * 2,
            mask.data_ptr(), n_kv * 2, index.data_ptr(), D ** -0.5, 0.0, 0.0)
    out = torch.empty((Nq, H * D), device="cuda")
    check(L.b200_flash_attn_ext_indexed(*args, out.data_ptr(), scratch.data_ptr(), scratch.numel(), st))
    s = torch.einsum("jhd,chd->jhc", q.half().double(), k.double().repeat_interleave(H // Hkv, 1)) * D ** -0.5 + mask.double()[:, None]
    want = torch.einsum("jhc,chd->jhd", torch.softmax(s, -1), v.double().repeat_interleave(H // Hkv, 1)).reshape(Nq, H * D)
    assert float((out - want).abs().max() / want.abs().max()) < 2e-5
    acts = [torch.full((L.b200_act_bytes(H * D, Nq),), fill, dtype=torch.uint8, device="cuda") for fill in (0x11, 0xAB)]
    check(L.b200_quantize_activations(out.data_ptr(), H * D * 4, H * D, Nq, acts[0].data_ptr(), acts[0].numel(), 0, st))
    check(L.b200_flash_attn_ext_quant(*args, None, acts[1].data_ptr(), acts[1].numel(), 0, scratch.data_ptr(), scratch.numel(), st))
    torch.cuda.synchronize()
    assert torch.equal(*acts)
