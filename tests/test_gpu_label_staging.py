"""The FP32 label kernel where a launch of many blocks stages fewer clusters at a time than one of few (and the last
group is a partial one): a data set made of repeated copies of a small one gets its log-likelihoods bit for bit, and
with the same uniforms its labels.  The points are multiples of 1/8 that sum to zero, so that both have shift 0."""
import numpy as np
import pytest

from conftest import uniforms
from dpmmsubclusters_gpu_b200 import LL_FP32, CudaKernel, prior_type

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,K", [(3, 200), (8, 119), (8, 120), (16, 40), (16, 121), (32, 63), (64, 9)])
def test_many_blocks_equal_few(D, K):
    rng = np.random.default_rng(D + K)
    M, copies = 700, 160
    half = np.round(rng.normal(size=(M // 2, D)) * 16) / 8
    x = np.stack([half, -half], 1).reshape(M, D)
    mus = rng.normal(size=(K, D))
    A = rng.normal(size=(K, D, D)) * 0.2 / np.sqrt(D) + np.eye(D)
    inv = A @ np.swapaxes(A, -1, -2)
    u = uniforms(2 * M, K).reshape(M, 2)
    params = (mus, inv, -np.linalg.slogdet(inv)[1], rng.dirichlet(np.full(K, 3.0)))

    def run(c):
        ck = CudaKernel(prior_type.Gaussian, loglik_mode=LL_FP32, k_max=K + 1).init(c * M, np.tile(x, (c, 1)), 1, points_major=True)
        ck.set_gaussian_params(*params)
        r = np.asarray(ck.create_clusters_labels(K, uniforms=np.tile(u, (c, 1)), return_loglik=True))
        lab = ck.get_labels()
        ck.release()
        return r.reshape(c, M, K), lab.reshape(c, M)
    r, lab = run(copies)
    r1, lab1 = run(1)
    np.testing.assert_array_equal(r, np.broadcast_to(r1, r.shape))
    np.testing.assert_array_equal(lab, np.broadcast_to(lab1, lab.shape))
