"""The product of the stacked wq, wk, wv rows that rotates and stores by itself: bit-identical to the product followed by b200_rope_store_angles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one and two columns (dp4a kernel; large: streaming), up to 8 (streaming), 9 (two launches); heads of every size, rotated dims short of the
# head, row tiles that do not divide among the SMs, fewer of them than SMs, K that no longer fits the streaming kernel's shared memory
@pytest.mark.parametrize("wtype", [2, 8])
@pytest.mark.parametrize("K,D,H,Hkv,n_dims,Ns", [(2048, 64, 32, 8, 64, (1, 2, 3, 8, 9)), (4096, 128, 32, 8, 128, (1, 2, 7)), (8192, 128, 64, 8, 64, (1, 5)),
                                                 (256, 256, 1, 1, 128, (1, 2, 3)), (160, 64, 7, 1, 32, (2, 5, 8)), (22016, 64, 2, 1, 64, (1, 3))])
def test_same_as_two_calls(wtype, K, D, H, Hkv, n_dims, Ns):
    from cactus_b200._lib import check, lib
    from cactus_b200.engine import random_blocks
    from cactus_b200.ops import QWeight
    L, cells, M = lib(), 32, (H + 2 * Hkv) * D
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(K + D)
    w = QWeight.from_blocks(wtype, K, M, random_blocks(wtype, M, K, g))
    for N in Ns:
        x = torch.randn((N, K), device="cuda", generator=g)
        act = torch.empty(L.b200_act_bytes(K, N), dtype=torch.uint8, device="cuda")
        check(L.b200_quantize_activations(x.data_ptr(), K * 4, K, N, act.data_ptr(), act.numel(), 0, st))
        pos = torch.randint(0, 5000, (N,), device="cuda", generator=g, dtype=torch.int32)
        slots = torch.randperm(cells, device="cuda", generator=g)[:N].to(torch.int32)
        angles = torch.empty((N, n_dims), device="cuda")
        check(L.b200_rope_angles(angles.data_ptr(), N, n_dims, pos.data_ptr(), None, 500000.0, 1.0, 1.0, st))
        ws = torch.empty(max(256, L.b200_mul_mat_workspace_bytes(wtype, K, M, N)), dtype=torch.uint8, device="cuda")
        out = [torch.full((N, M + 2), 7.0, device="cuda") for _ in range(2)]
        kv = [torch.zeros((cells, Hkv * D), dtype=torch.float16, device="cuda") for _ in range(4)]
        s = (M + 2) * 4
        check(L.b200_mul_mat_q_prequant(wtype, w.data.data_ptr(), K, M, act.data_ptr(), N, out[0].data_ptr(), s, ws.data_ptr(), ws.numel(), st))
        check(L.b200_rope_store_angles(out[0].data_ptr(), D * 4, s, out[0][:, H * D:].data_ptr(), D * 4, s, out[0][:, (H + Hkv) * D:].data_ptr(), s, D, H, Hkv, N, n_dims,
                                       angles.data_ptr(), slots.data_ptr(), kv[0].data_ptr(), Hkv * D * 2, kv[1].data_ptr(), Hkv * D * 2, st))
        check(L.b200_mul_mat_qkv_rope(wtype, w.data.data_ptr(), K, act.data_ptr(), N, out[1].data_ptr(), s, D, H, Hkv, n_dims, angles.data_ptr(), slots.data_ptr(),
                                      kv[2].data_ptr(), Hkv * D * 2, kv[3].data_ptr(), Hkv * D * 2, ws.data_ptr(), ws.numel(), st))
        torch.cuda.synchronize()
        assert torch.equal(out[0][:, :H * D], out[1][:, :H * D]), N
        assert torch.equal(kv[0], kv[2]) and torch.equal(kv[1], kv[3]), N
        assert bool((out[1][:, M:] == 7.0).all())
