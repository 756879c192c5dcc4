"""The product of up to 8 columns whose weights go straight to registers, at the edges of its split, against the oracle.

Only the order and the rounding of the fp32 sums differ from the reference.  Bound, of the largest result: a sum of n terms of
which each is rounded to 2^-24 is some sqrt(n) 2^-25 away, the oracle's as much; over 672 blocks (K 21504) 2 x 7.7e-7 in the mean
of the largest of them, and 5e-6 leaves three times that for the largest difference."""
import numpy as np
import pytest
import torch

from gpu_util import rel_max_err

pytestmark = pytest.mark.gpu

# (type, rows, K, columns): one block; a row tile and a bit; more CTAs than row tiles; chunks that do not come out even; a warp's
# last tiles; K where the activations and partial tiles just fit into shared memory, and where they no longer do
CASES = [(2, 16, 32, 3), (2, 17, 160, 8), (8, 33, 64, 5), (2, 700, 1056, 7), (8, 272, 2080, 4), (2, 2400, 544, 8), (8, 5000, 256, 6), (2, 48, 20480, 8),
         (2, 32, 21504, 3), (2, 32, 32768, 8),
         (2, 65536, 1024, 1), (2, 65530, 1024, 2), (8, 65536, 1000 // 32 * 32, 1)]   # one and two columns from 32768 tiles on (and just below)


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c)))
def test_few_columns_against_the_oracle(oracle, case):
    from cactus_b200 import ops
    wtype, M, K, N = case
    rng = np.random.default_rng(M + K + N)
    wq = oracle.quantize_weights(wtype, (rng.standard_normal((M, K)) * 0.02).astype(np.float32))
    x = rng.standard_normal((N, K)).astype(np.float32)
    ref, _ = oracle.mul_mat(wtype, wq, x)
    w, xd = ops.QWeight.from_blocks(wtype, K, M, wq), torch.from_numpy(x).cuda()
    wide = torch.full((N, M + 3), -7.0, device="cuda")          # a destination whose rows are neither packed nor 16-byte aligned
    got = ops.mul_mat(w, xd, out=wide[:, 1:M + 1])
    assert rel_max_err(got.cpu().numpy(), ref) < 5e-6
    assert bool((wide[:, 0] == -7).all()) and bool((wide[:, M + 1:] == -7).all())
    assert torch.equal(got, ops.mul_mat(w, xd))                 # the split does not depend on timing
