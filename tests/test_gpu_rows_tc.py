"""The persistent gather kernels (csrc/dpmm_rows_tc.cu) where a CTA walks several short chunks: more clusters than
SMs, one to three tiles each, so that the operand buffers of the chunks and the slots of the tiles come
round in every phase.  Sub-cluster log-likelihoods and sub-labels equal those of the one-block-per-chunk fused
pass bit for bit, and the labels equal the oracle's draw on the GPU's own log-likelihoods (margins below
1e-4 aside, the bound of the FP32 two-way softmax)."""
import numpy as np
import pytest

from conftest import uniforms
from dpmmsubclusters_gpu_b200 import LL_TC_BF16X3, CudaKernel, prior_type
from dpmmsubclusters_gpu_b200.capi import check, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [17, 32, 33, 64])
@pytest.mark.parametrize("K,lo,hi", [(250, 1, 300), (3, 1, 129), (160, 128, 129)])
def test_short_chunks(D, K, lo, hi):
    rng = np.random.default_rng(D + K)
    sizes = rng.integers(lo, hi + 1, size=K)
    z = rng.permutation(np.repeat(np.arange(K), sizes))
    N = z.size
    mus = rng.normal(size=(K, D)) * 3
    x = mus[z] + rng.normal(size=(N, D))
    A = rng.normal(size=(K, 2, D, D)) * 0.3 / np.sqrt(D) + np.eye(D)
    inv_lr = A @ np.swapaxes(A, -1, -2)
    ld_lr = -np.linalg.slogdet(inv_lr)[1]
    mu_lr = mus[:, None] + 0.5 * rng.normal(size=(K, 2, D))
    lrw = rng.dirichlet([2, 2], size=K)
    u = uniforms(2 * N, D)
    got = []
    for fused in (1, 0):
        ck = CudaKernel(prior_type.Gaussian, loglik_mode=LL_TC_BF16X3).init(N, x, 3, points_major=True)
        check(lib().dpmm_set_fused_sub_stats(ck.ctx, fused))
        ck.set_gaussian_params(mus, np.repeat(np.eye(D)[None], K, 0), np.zeros(K), np.full(K, 1.0 / K), mu_lr, inv_lr, ld_lr,
                               lrw)
        ck.set_labels((z + 1).astype(np.int32))
        r = ck.create_subclusters_labels(K, uniforms=u, return_loglik=True)
        got.append((np.asarray(r), ck.get_sub_labels()))
        ck.release()
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][1], got[1][1])
    r = got[1][0].astype(np.float64) + np.log(lrw[z])
    p = np.exp(r - r.max(1, keepdims=True))
    p /= p.sum(1, keepdims=True)
    u = u.reshape(N, 2).astype(np.float64)
    col = (u[:, 0] * 1.999999 + 1).astype(int)
    y = 2 * p[np.arange(N), col - 1]
    want = np.where((y < 1) & (y < u[:, 1]), 3 - col, col)
    margin = np.minimum(np.abs(y - u[:, 1]), np.abs(y - 1))
    bad = got[1][1] != want
    assert np.all(margin[bad] < 1e-4), int(bad.sum())
