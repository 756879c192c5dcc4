"""A product that is enqueued right behind the kernel which writes its weights, with nothing waited for in between: an upload as the
direct predecessor, the one-row quantiser (which lets the next kernel in before its own wait) between the two, a stacking copy.

Calls are ordered on their stream, so the result is that of the new weights to the last bit, whatever the buffer held before."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _two_weights(wtype, K, M):
    from cactus_b200.engine import random_blocks
    g = torch.Generator(device="cuda").manual_seed(K + M)
    return [random_blocks(wtype, M, K, g) for _ in range(2)], g


# dp4a (layers and, Q8_0 at two columns, a short head), streaming (heads and 3 to 8 columns), tiled mma.sync
@pytest.mark.parametrize("wtype,K,M,N", [(2, 2048, 8192, 1), (2, 4096, 20480, 1), (8, 1024, 65536, 2), (2, 1024, 65536, 1), (8, 1024, 65536, 1), (2, 1024, 65536, 2), (2, 2048, 8192, 3), (2, 4096, 4096, 8), (8, 2048, 4096, 5), (2, 2048, 8192, 24)])
@pytest.mark.parametrize("quantiser_between", [False, True])
def test_product_behind_an_upload(wtype, K, M, N, quantiser_between):
    from cactus_b200._lib import check, lib
    L = lib()
    st = torch.cuda.current_stream().cuda_stream
    blocks, g = _two_weights(wtype, K, M)
    x = torch.randn((N, K), device="cuda", generator=g)
    w = torch.empty(L.b200_weight_bytes(wtype, K, M), dtype=torch.uint8, device="cuda")
    act = torch.empty(L.b200_act_bytes(K, N), dtype=torch.uint8, device="cuda")
    ws = torch.empty(max(256, L.b200_mul_mat_workspace_bytes(wtype, K, M, N)), dtype=torch.uint8, device="cuda")

    def upload(b):
        check(L.b200_weight_upload(wtype, K, M, b.data_ptr(), w.data_ptr(), 0, M, st))

    def quantise():
        check(L.b200_quantize_activations(x.data_ptr(), K * 4, K, N, act.data_ptr(), act.numel(), 0, st))

    def product():
        out = torch.empty((N, M), device="cuda")
        check(L.b200_mul_mat_q_prequant(wtype, w.data_ptr(), K, M, act.data_ptr(), N, out.data_ptr(), M * 4, ws.data_ptr(), ws.numel(), st))
        return out
    want = []
    for b in blocks:
        upload(b)
        quantise()
        torch.cuda.synchronize()
        want.append(product())
        torch.cuda.synchronize()
    assert not torch.equal(*want)
    for i in range(8):
        upload(blocks[i & 1])
        if quantiser_between:
            quantise()
        got = product()
        assert torch.equal(got, want[i & 1]), i


@pytest.mark.parametrize("N", [1, 4])
def test_product_behind_a_stacking_copy(N):
    from cactus_b200 import ops
    K, M = 1024, 32768   # stacked: an output head's rows
    blocks, g = _two_weights(2, K, M)
    parts = [ops.QWeight.from_blocks(2, K, M, b) for b in blocks]
    x = torch.randn((N, K), device="cuda", generator=g)
    want = [ops.mul_mat(ops.QWeight.from_blocks(2, K, 2 * M, torch.cat([blocks[i], blocks[1 - i]])), x) for i in range(2)]
    for i in range(8):
        w = ops.QWeight.cat([parts[i & 1], parts[1 - (i & 1)]])   # (its memory is that of the last turn's weight)
        assert torch.equal(ops.mul_mat(w, x), want[i & 1]), i
        del w
