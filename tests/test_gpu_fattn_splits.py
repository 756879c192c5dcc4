"""Attention of a few tokens, whose KV range is cut: tokens of one word (one split) beside tokens of many, at the cache sizes where
the number of splits changes; the result in f32 against f64, and as the pass that adds the splits quantises it.

Tolerance: f16 inputs are exact in f64, Q is rounded to f16 here as there; what is left are f32 sums and P as an f16 pair (2^-22)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_kv,lens", [(768, (1, 65, 768)), (1024, (1, 64, 128, 129, 1000)), (1280, (1280,)), (4096, (3, 130, 4096, 64, 2000, 700, 1, 128, 4000))])
@pytest.mark.parametrize("D", [64, 128])
def test_one_word_beside_many(n_kv, lens, D):
    from cactus_b200._lib import check, lib
    L, H, Hkv, Nq = lib(), 8, 2, len(lens)
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(n_kv + D)
    q = torch.randn((Nq, H, D), device="cuda", generator=g)
    k, v = (torch.randn((n_kv, Hkv, D), device="cuda", generator=g).half() for _ in range(2))
    mask = torch.full((Nq, n_kv), float("-inf"), dtype=torch.float16, device="cuda")
    for j, n in enumerate(lens):
        mask[j, :n] = 0
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


@pytest.mark.parametrize("Nq", [1, 5])
@pytest.mark.parametrize("softcap", [0.0, 20.0])
def test_values_in_the_mask(Nq, softcap):
    """A mask with values beside 0 and -inf (with the slopes of ALiBi) and one without, which takes the walk that does not read it."""
    from cactus_b200._lib import check, lib
    L, n_kv, D, H, Hkv, bias = lib(), 1024, 64, 8, 2, 4.0
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(Nq)
    q = torch.randn((Nq, H, D), device="cuda", generator=g)
    k, v = (torch.randn((n_kv, Hkv, D), device="cuda", generator=g).half() for _ in range(2))
    slopes = torch.tensor([2.0 ** (-bias / H * (h + 1)) for h in range(H)], dtype=torch.float64, device="cuda")
    for soft in (0.0, 1.0):
        mask = (soft * torch.randn((Nq, n_kv), device="cuda", generator=g)).half()
        mask[torch.rand((Nq, n_kv), device="cuda", generator=g) < 0.4] = float("-inf")
        mask[:, 7] = 0
        index = torch.empty(L.b200_mask_index_bytes(Nq, n_kv), dtype=torch.uint8, device="cuda")
        check(L.b200_mask_index_build(mask.data_ptr(), n_kv * 2, Nq, n_kv, index.data_ptr(), index.numel(), st))
        scratch = torch.empty(max(256, L.b200_flash_attn_scratch_bytes(D, H, Hkv, Nq, n_kv)), dtype=torch.uint8, device="cuda")
        out = torch.empty((Nq, H * D), device="cuda")
        check(L.b200_flash_attn_ext_indexed(D, H, Hkv, Nq, n_kv, q.data_ptr(), H * D * 4, D * 4, k.data_ptr(), Hkv * D * 2, D * 2, v.data_ptr(), Hkv * D * 2, D * 2,
                                            mask.data_ptr(), n_kv * 2, index.data_ptr(), D ** -0.5, bias, softcap, out.data_ptr(), scratch.data_ptr(), scratch.numel(), st))
        s = torch.einsum("jhd,chd->jhc", q.half().double(), k.double().repeat_interleave(H // Hkv, 1)) * D ** -0.5
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        s = s + slopes[None, :, None] * mask.double()[:, None]
        want = torch.einsum("jhc,chd->jhd", torch.softmax(s, -1), v.double().repeat_interleave(H // Hkv, 1)).reshape(Nq, H * D)
        torch.cuda.synchronize()
        assert float((out - want).abs().max() / want.abs().max()) < 2e-5, soft
