"""The mask index (one pass per row, plan, vote) and the token-by-token walk of tiles that share few cells, at their edges."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _mask(lens, prompt, cells, aligned):
    nq = len(lens) + prompt
    m = torch.full((nq, cells + (0 if aligned else 1)), float("-inf"), dtype=torch.float16)[:, : cells]
    at = 0
    for j, n in enumerate(lens):
        m[j, at:at + n] = 0
        at += n
    for j in range(prompt):
        m[len(lens) + j, at:at + j + 1] = 0
    return m


# decode tokens of the given lengths first, then a prompt; cells; head size, heads; a mask row that starts on 16 bytes or not
CASES = [([1, 2047, 33, 64, 5], 131, 4096, 128, 32, True), ([700] * 17, 111, 16384, 64, 32, True), ([31, 32, 33], 126, 1000, 128, 16, False),
         (list(range(1, 49)), 230, 8191, 64, 16, False), ([1], 127, 136, 128, 32, True)]


@pytest.mark.parametrize("lens,prompt,cells,D,H,aligned", CASES)
@pytest.mark.parametrize("soft", [False, True])
def test_mixed_ubatch(lens, prompt, cells, D, H, aligned, soft):
    from cactus_b200 import ops
    g = torch.Generator().manual_seed(7)
    mask = _mask(lens, prompt, cells, aligned)
    if soft:
        mask[0, 0] = -0.5
    nq, hkv = mask.shape[0], 8
    q, k, v = torch.randn((nq, H, D), generator=g), torch.randn((cells, hkv, D), generator=g).half(), torch.randn((cells, hkv, D), generator=g).half()
    dev = torch.empty_strided(mask.shape, mask.stride(), dtype=mask.dtype, device="cuda").copy_(mask)
    got = ops.flash_attn_ext(q.cuda(), k.cuda(), v.cuda(), dev, D ** -0.5).cpu()
    s = torch.einsum("nhd,chd->nhc", q.half().float(), k.float().repeat_interleave(H // hkv, 1)) * D ** -0.5 + mask.float()[:, None]
    ref = torch.einsum("nhc,chd->nhd", torch.softmax(s, -1), v.float().repeat_interleave(H // hkv, 1))
    assert (got - ref).abs().max() < 2e-4 * ref.abs().max()
