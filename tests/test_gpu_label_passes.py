"""The dense tensor-core label kernel at the cluster counts where its tiles and launches change (two or four
clusters a tile, 256 a launch) and at both operand widths, drawn and argmax, against the FP64 oracle."""
import numpy as np
import pytest

import parity as P
from conftest import uniforms
from dpmmsubclusters_gpu_b200 import LL_TC_BF16X3, CudaKernel, prior_type
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [20, 32, 64])
@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 7, 255, 256, 257, 300, 513])
def test_cluster_counts(D, K):
    rng = np.random.default_rng(D * 1000 + K)
    N = 700
    mus = rng.normal(size=(K, D))
    x = mus[rng.integers(0, K, size=N)] + rng.normal(size=(N, D))
    A = rng.normal(size=(K, D, D)) * 0.2 / np.sqrt(D) + np.eye(D)
    inv = A @ np.swapaxes(A, -1, -2)
    ld = -np.linalg.slogdet(inv)[1]
    w = rng.dirichlet(np.full(K, 3.0))
    ck = CudaKernel(prior_type.Gaussian, loglik_mode=LL_TC_BF16X3, k_max=520).init(N, x, 1, points_major=True)
    ck.set_gaussian_params(mus, inv, ld, w)
    u = uniforms(2 * N, K)
    r = ck.create_clusters_labels(K, uniforms=u, return_loglik=True)
    r64 = np.stack([O.gauss_loglik(x, mus[k], inv[k], ld[k], w[k]) for k in range(K)], 1)
    P.gauss_ll(r, r64, D, ld, np.log(w), "tc", f"label passes D={D} K={K}")
    lab, mg = O.sample_labels(np.asarray(r, np.float64), u.reshape(N, 2).astype(np.float64))
    bad = ck.get_labels() != lab
    assert np.all(mg[bad] < 1e-4)
    r = np.asarray(ck.create_clusters_labels(K, True, return_loglik=True))
    np.testing.assert_array_equal(ck.get_labels(), r.argmax(1) + 1)
    ck.release()
