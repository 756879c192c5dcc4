"""How many KV splits attention cuts a cache into, read off the scratch it asks for (no GPU).  Where the range is cut is part of the result's
last bits, and the product behind it quantises them: the counts are what they were before, for a step's logits to be."""
import pytest


@pytest.mark.parametrize("Nq,H,Hkv,D,n_kv,want", [
    (1, 32, 8, 64, 512, 1), (1, 32, 8, 64, 1023, 1), (1, 32, 8, 64, 1024, 2), (1, 32, 8, 128, 2048, 4), (1, 32, 8, 128, 4096, 8), (1, 32, 8, 128, 16384, 32),
    (1, 32, 8, 128, 65536, 37), (2, 32, 8, 64, 1024, 2), (3, 32, 8, 64, 16384, 13), (7, 32, 8, 128, 16384, 6), (7, 32, 8, 128, 1280, 2), (12, 32, 8, 128, 65536, 4),
    (36, 32, 8, 128, 65536, 2), (37, 32, 8, 128, 65536, 1), (1, 8, 1, 128, 65536, 64), (4, 16, 1, 64, 3000, 5)])
def test_split_counts(Nq, H, Hkv, D, n_kv, want):
    from cactus_b200._lib import lib
    L = lib()
    part = L.b200_flash_attn_scratch_bytes(D, H, Hkv, Nq, n_kv) - L.b200_mask_index_bytes(Nq, n_kv)
    per = Nq * H * (D + 2) * 4
    assert part == (0 if want == 1 else (per * want + 255) // 256 * 256)
