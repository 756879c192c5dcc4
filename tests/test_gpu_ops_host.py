"""The native host path of the single-op entry points: what its failures look like to the caller."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_an_allocation_that_fails_raises_torchs_out_of_memory_error():
    """A result that does not fit what the process may take raises torch.OutOfMemoryError, as a torch op does (callers
    catch it to free memory and try again), and the op works once there is room.  The limit is the caching allocator's own
    (set_per_process_memory_fraction): nothing large is allocated on the device."""
    from cactus_b200 import ops
    K, M, N = 32, 1 << 20, 512                       # a result of 2 GiB from operands of 20 MB
    w = ops.QWeight.from_blocks(ops.Q4_0, K, M, np.zeros((M, 18), np.uint8))
    x = torch.ones((N, K), device="cuda")
    q = torch.zeros((1 << 15, 32, 64), device="cuda")    # 256 MB, and as much for the result
    kv = torch.zeros((256, 8, 64), dtype=torch.float16, device="cuda")
    torch.cuda.empty_cache()
    room = torch.cuda.memory_reserved() + (64 << 20)
    torch.cuda.set_per_process_memory_fraction(room / torch.cuda.get_device_properties(0).total_memory)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            ops.mul_mat(w, x)
        with pytest.raises(torch.OutOfMemoryError):
            ops.flash_attn_ext(q, kv, kv, None, 0.125)
        assert not ops.mul_mat(w, x[:1]).any()       # 4 MB: fits
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    del q
    assert ops.mul_mat(w, x[:32]).shape == (32, M)
