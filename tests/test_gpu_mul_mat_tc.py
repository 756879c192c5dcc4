"""The tcgen05 (tensor-memory accumulator) mul_mat kernel against the oracle and against f64.

B200_MMQ_TC=1 takes it for every Q4_0 product of at least 9 columns, which is read once per process: the cases run in a
child interpreter, which also reports the library's kernel status (non-zero after a bounded barrier wait gave up)."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def run_child(code):
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, B200_MMQ_TC="1"), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    res = json.loads(r.stdout.strip().splitlines()[-1])
    assert res["status"] == 0
    return res


CHILD = r"""
import json, sys
sys.path.insert(0, {here!r}); sys.path.insert(0, {root!r})
import numpy as np, torch
from oracle.binding import Oracle, Q4_0, Q8_0
from cactus_b200 import ops, _lib
o = Oracle()
L = _lib.lib()
err, routed = [], []
for (wtype, M, K, N) in {cases!r}:
    rng = np.random.default_rng(M + K + N)
    wq = o.quantize_weights(wtype, (rng.standard_normal((M, K)) * 0.02).astype(np.float32))
    x = rng.standard_normal((N, K)).astype(np.float32)
    ref, _ = o.mul_mat(wtype, wq, x)
    got = ops.mul_mat(ops.QWeight.from_blocks(wtype, K, M, wq), torch.from_numpy(x).cuda()).cpu().numpy()
    err.append(float(np.abs(got - ref).max() / np.abs(ref).max()))
    routed.append(L.b200_mul_mat_scratch_bytes(wtype, K, M, N) != L.b200_act_bytes(K, N) + L.b200_mul_mat_workspace_bytes(wtype, K, M, N))
print(json.dumps({{"err": err, "routed": routed, "status": int(L.b200_kernel_status())}}))
"""

# full and ragged tiles: rows not a multiple of 16, 128 or 256, columns not a multiple of 8 or 64, blocks not a multiple of 4; one to
# four column chunks; the K range whole, cut by a cluster, cut in equal shares
CASES = [(2, 128, 128, 64), (2, 80, 512, 9), (2, 80, 512, 16), (2, 1000, 4096, 50), (2, 130, 160, 40), (2, 48, 14336, 20), (2, 300, 1024, 65),
         (2, 256, 256, 200), (2, 272, 2048 + 96, 128), (2, 4096, 4096, 64)]


def test_sums_are_within_fp32_rounding_of_the_oracle():
    """Only the order and the rounding of the fp32 sums differ from the reference.  Of the largest result: the kernel is within
    2.5e-7 (2-norm, below), the oracle's own fp32 sums as much; the largest of 10^5 differences is some five times that."""
    res = run_child(CHILD.format(here=HERE, root=ROOT, cases=CASES))
    assert all(res["routed"])
    assert max(res["err"]) < 2e-6, list(zip(CASES, res["err"]))


def test_q8_0_weights_keep_the_mma_sync_kernel():
    cases = [(8, 130, 160, 40), (8, 80, 512, 33), (8, 4096, 1024, 130)]
    res = run_child(CHILD.format(here=HERE, root=ROOT, cases=cases))
    assert not any(res["routed"])
    assert max(res["err"]) < 2e-6, list(zip(cases, res["err"]))


F64_CHILD = r"""
import json, sys
sys.path.insert(0, {root!r})
import torch
from cactus_b200 import ops, _lib
from cactus_b200.engine import random_blocks
gen = torch.Generator(device="cuda").manual_seed(1)
out = []
for (wtype, M, K, N) in {cases!r}:
    blocks = random_blocks(wtype, M, K, gen)
    b = blocks.view(M, K // 32, -1)
    q = torch.cat([(b[..., 2:] & 15).double() - 8, (b[..., 2:] >> 4).double() - 8], -1)
    w = (q * b[..., :2].contiguous().view(torch.float16).double()).view(M, K)
    x = torch.randn((N, K), device="cuda", generator=gen)
    a = ops.quantize_row_q8_0(x).view(N, K // 32, 34)
    a = (a[..., 2:].contiguous().view(torch.int8).double() * a[..., :2].contiguous().view(torch.float16).double()).view(N, K)
    want = a @ w.T
    got = ops.mul_mat(ops.QWeight.from_blocks(wtype, K, M, blocks), x).double()
    out.append(float((got - want).norm() / want.norm()))
print(json.dumps({{"err": out, "status": int(_lib.lib().b200_kernel_status())}}))
"""


def test_sums_are_as_close_to_f64_as_exact_dots_and_fp32_sums_are():
    """Against the product of the quantised operands in f64 (2-norm).  Bound: the mma.sync kernel, whose block dots are exact and
    whose sums round to nearest, is 0.7e-7 to 3.8e-7 away over these sizes.  The tensor core truncates when it accumulates, at
    most one part in 2^23 and half of that in the mean: 8 times per block group are 8 x 2^-24 / 2 = 2.4e-7 on a sum that grows
    evenly; 16 block groups in one accumulator, as it was once, 2.3e-6."""
    cases = [(2, 256, 128, 33), (2, 2048, 1024, 77), (2, 4096, 4096, 512), (2, 1040, 14336, 512), (2, 28672, 4096, 64)]
    res = run_child(F64_CHILD.format(root=ROOT, cases=cases))
    assert max(res["err"]) < 3.8e-7, list(zip(cases, res["err"]))
