"""Multinomial sub-label pass where its staged rows and its static arrays together pass the 48 KB that a launch gets
without asking (Dp = 352 and 672).  Each D in a process of its own: a larger limit asked for by another D would hide it."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = r"""
import sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from dpmmsubclusters_gpu_b200 import CudaKernel, prior_type
D, K, N = int(sys.argv[2]), 3, 700
rng = np.random.default_rng(D)
x = rng.poisson(0.7, size=(N, D)).astype(np.float64)
z = rng.integers(0, K, size=N)
ck = CudaKernel(prior_type.Multinomial, k_max=8).init(N, x, 1, points_major=True)
lt = np.log(rng.dirichlet(np.ones(D), size=(K, 3)))
ck.set_multinomial_params(lt[:, 0], None, lt[:, 1:], np.full((K, 2), 0.5))
ck.set_labels((z + 1).astype(np.int32))
ck.create_subclusters_labels(K, uniforms=rng.random(2 * N, dtype=np.float32))
sub = ck.get_sub_labels()
cnt, sm, _ = ck.create_sufficient_statistics(np.arange(K))
for k in range(K):
    for s in (1, 2):
        m = (z == k) & (sub == s)
        assert cnt[k, s] == m.sum()
        np.testing.assert_array_equal(sm[k, s], x[m].sum(0))
print("OK")
"""


@pytest.mark.parametrize("D", [330, 352, 641, 672])
def test_stage_next_to_the_default_limit(D):
    out = subprocess.run([sys.executable, "-c", CHILD, ROOT, str(D)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and "OK" in out.stdout, out.stdout + out.stderr
