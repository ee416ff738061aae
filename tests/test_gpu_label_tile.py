"""The FP32 SIMT label kernel at the cluster counts where its staging changes (one cluster more or less than a stage
holds, the largest counts of each block size), at every padded width, with ragged blocks, against the FP64 oracle."""
import numpy as np
import pytest

import parity as P
from conftest import uniforms
from dpmmsubclusters_gpu_b200 import LL_FP32, CudaKernel, prior_type
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,K", [(3, 255), (3, 256), (3, 257), (8, 1), (8, 63), (8, 64), (8, 65), (8, 400), (8, 800),
                                 (13, 15), (13, 16), (13, 17), (13, 33), (13, 420), (32, 3), (32, 4), (32, 5),
                                 (50, 1), (50, 2), (50, 300), (65, 7), (80, 3), (81, 9), (100, 3), (113, 2), (128, 40), (128, 300)])
@pytest.mark.parametrize("N", [1, 300])
def test_stages(D, K, N):
    rng = np.random.default_rng(D * 1000 + K)
    mus = rng.normal(size=(K, D))
    x = mus[rng.integers(0, K, size=N)] + rng.normal(size=(N, D))
    A = rng.normal(size=(K, D, D)) * 0.2 / np.sqrt(D) + np.eye(D)
    inv = A @ np.swapaxes(A, -1, -2)
    ld = -np.linalg.slogdet(inv)[1]
    w = rng.dirichlet(np.full(K, 3.0))
    ck = CudaKernel(prior_type.Gaussian, loglik_mode=LL_FP32, k_max=K + 1).init(N, x, 1, points_major=True)
    ck.set_gaussian_params(mus, inv, ld, w)
    u = uniforms(2 * N, K)
    r = ck.create_clusters_labels(K, uniforms=u, return_loglik=True)
    r64 = np.stack([O.gauss_loglik(x, mus[k], inv[k], ld[k], w[k]) for k in range(K)], 1)
    row_err = P.gauss_ll(r, r64, D, ld, np.log(w), "fp32", f"label tile D={D} K={K}")
    P.labels_vs_fp64(ck.get_labels(), r64, u.reshape(N, 2).astype(np.float64), row_err, f"label tile draws D={D} K={K}")
    r = np.asarray(ck.create_clusters_labels(K, True, return_loglik=True))
    np.testing.assert_array_equal(ck.get_labels(), r.argmax(1) + 1)
    ck.release()
