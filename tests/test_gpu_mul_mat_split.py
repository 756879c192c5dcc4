"""The K cuts of the streaming product (3 to 8 columns) are those of the tiled one (9 to 16): a column's result does not depend on which of
the two works, to the last bit.  Shapes for each way to deal K out: whole, in clusters, through partial sums, and the stream-K deals."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (type, rows, K): clusters of 8; 13 partial sums; fewer row groups than SMs and a ragged last one; one block; heads and tails (both types, a short
# and a ragged K); the even deal; one part for all of K; K beyond the streaming kernel's shared memory
SHAPES = [(2, 6144, 4096), (2, 4096, 14336), (8, 2048, 2048), (2, 700, 1056), (8, 33, 64), (2, 28672, 4096), (8, 28672, 2048), (2, 30208, 1056), (2, 44544, 416),
          (2, 57344, 2048), (8, 60032, 512), (2, 65408, 160), (2, 20480, 96), (2, 16384, 256), (2, 160, 20480), (2, 32, 32768)]


@pytest.mark.parametrize("wtype,M,K", SHAPES)
def test_columns_do_not_depend_on_the_kernel(wtype, M, K):
    from cactus_b200 import ops
    from cactus_b200._lib import check, lib
    from cactus_b200.engine import random_blocks
    L = lib()
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(M + K)
    w = ops.QWeight.from_blocks(wtype, K, M, random_blocks(wtype, M, K, g))
    x = torch.randn((16, K), device="cuda", generator=g)
    want = ops.mul_mat(w, x)
    for N in (3, 5, 8):
        assert torch.equal(ops.mul_mat(w, x[:N]), want[:N]), N

    def without_workspace(N):   # the deals that need one are out of reach
        act = torch.empty(L.b200_act_bytes(K, N), dtype=torch.uint8, device="cuda")
        out = torch.empty((N, M), device="cuda")
        check(L.b200_quantize_activations(x.data_ptr(), K * 4, K, N, act.data_ptr(), act.numel(), 0, st))
        check(L.b200_mul_mat_q_prequant(wtype, w.data.data_ptr(), K, M, act.data_ptr(), N, out.data_ptr(), M * 4, None, 0, st))
        torch.cuda.synchronize()
        return out
    assert torch.equal(without_workspace(7), without_workspace(16)[:7])


# layers of 32768 tiles and more; a row tile short of an output head; a head one block group short of 32768 tiles, and one of a short K at two columns
@pytest.mark.parametrize("wtype,M,K,Ns", [(2, 28672, 4096, (1, 2)), (8, 16384, 4096, (1, 2)), (2, 65520, 1024, (1, 2)), (2, 65536, 896, (1, 2)), (8, 65536, 1920, (2,))])
def test_one_and_two_columns_of_a_layer(wtype, M, K, Ns):
    """A layer's product of one or two columns is the dp4a kernel's whatever its size: the rows of two parts of a row split, which only that
    kernel stores, are the same to the last bit."""
    import ctypes as C

    from cactus_b200 import ops
    from cactus_b200._lib import check, lib
    from cactus_b200.engine import random_blocks
    L = lib()
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(M + K)
    w = ops.QWeight.from_blocks(wtype, K, M, random_blocks(wtype, M, K, g))
    first = M // 32 * 16
    rows, cols = (C.c_int64 * 2)(first, M - first), (C.c_int64 * 2)(0, first)
    flags = torch.zeros(64, dtype=torch.int32, device="cuda")   # (a world of one: nobody is waited for)
    for N in Ns:
        x = torch.randn((N, K), device="cuda", generator=g)
        act = torch.empty(L.b200_act_bytes(K, N), dtype=torch.uint8, device="cuda")
        check(L.b200_quantize_activations(x.data_ptr(), K * 4, K, N, act.data_ptr(), act.numel(), 0, st))
        want = torch.empty((N, M), device="cuda")
        check(L.b200_mul_mat_q_rowsplit_stacked(wtype, w.data.data_ptr(), K, M, act.data_ptr(), N, 0, 1, (C.c_void_p * 1)(want.data_ptr()), M * 4, 2, rows, cols, None, 0,
                                                (C.c_void_p * 1)(flags.data_ptr()), st))
        assert torch.equal(ops.mul_mat(w, x), want), N
