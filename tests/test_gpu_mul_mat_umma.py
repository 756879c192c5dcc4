"""The folded-scale tcgen05 mul_mat kernel at the edges of its tiles, and where a folded operand leaves the fp16 range.

B200_MMQ_TC=1 takes it for every Q4_0 product of at least 9 columns, which is read once per process: the cases run in a child
interpreter.  (The Q8_0 cases run the mma.sync kernel: the same edges, the same bounds.)"""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

CHILD = r"""
import json, sys
sys.path.insert(0, {here!r}); sys.path.insert(0, {root!r})
import numpy as np, torch
from oracle.binding import Oracle
from cactus_b200 import ops, _lib
o = Oracle()
out = []
for (wtype, M, K, N, wscale, xscale) in {cases!r}:
    rng = np.random.default_rng(M + K + N)
    w = (rng.standard_normal((M, K)) * 0.02).astype(np.float32)
    x = rng.standard_normal((N, K)).astype(np.float32)
    w[M // 2] *= wscale
    x[N // 3] *= xscale
    wq = o.quantize_weights(wtype, w)
    ref, _ = o.mul_mat(wtype, wq, x)
    wt, xd = ops.QWeight.from_blocks(wtype, K, M, wq), torch.from_numpy(x).cuda()
    got, again = ops.mul_mat(wt, xd), ops.mul_mat(wt, xd)
    g = got.cpu().numpy()
    scale = np.linalg.norm(x.astype(np.float64), axis=1)[:, None] * np.linalg.norm(w.astype(np.float64), axis=1)[None] * 3 / np.sqrt(K)   # about the largest result of a row and column
    out.append(dict(err=float((np.abs(g - ref) / scale).max()), finite=bool(np.isfinite(g).all()), same=bool(torch.equal(got, again))))
print(json.dumps(dict(res=out, status=int(_lib.lib().b200_kernel_status()))))
"""

# (type, rows, K, columns, scale of one weight row, scale of one column)
CASES = [(2, 256, 128, 33, 1, 1), (2, 16, 32, 64, 1, 1), (2, 129, 4096, 65, 1, 1), (2, 700, 1056, 77, 1, 1), (2, 4097, 512, 129, 1, 1), (8, 272, 2080, 40, 1, 1),
         (8, 1000, 256, 200, 1, 1), (2, 38400, 256, 96, 1, 1),        # many tiles: equal shares, tiles of two and three parts
         (2, 300, 512, 40, 2e6, 1), (8, 300, 512, 72, 1, 3e5)]        # |scale x quant| beyond 65504 in a weight row, in a column


def test_edges_and_values_beyond_fp16():
    env = dict(os.environ, B200_MMQ_TC="1")
    code = CHILD.format(here=HERE, root=ROOT, cases=CASES)
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    res = json.loads(r.stdout.strip().splitlines()[-1])
    assert res["status"] == 0
    for c, v in zip(CASES, res["res"]):
        assert v["finite"] and v["same"] and v["err"] < 5e-5, (c, v)
