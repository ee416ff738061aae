"""The FP32 sub-cluster pass (draws and statistics) at every padded width on clusters of 1 to 300 points: one tile
and a bit, ragged windows, sides that are empty in a window.  Against the FP64 oracle; the statistics' bound: runs of
at most 33 products of once-rounded differences, 38 roundings of 2^-24 on the sum of their absolute values."""
import numpy as np
import pytest

import parity as P
from conftest import uniforms
from dpmmsubclusters_gpu_b200 import LL_FP32, CudaKernel, prior_type
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [2, 4, 7, 8, 13, 16, 32, 60, 65, 80, 81, 97, 112, 113, 128])
@pytest.mark.parametrize("K,lo,hi", [(9, 1, 300), (4, 127, 129), (5, 31, 33), (1, 1, 1)])
def test_tiles(D, K, lo, hi):
    rng = np.random.default_rng(100 * D + K)
    sizes = rng.integers(lo, hi + 1, size=K)
    z = rng.permutation(np.repeat(np.arange(K), sizes))
    N = z.size
    mus = (rng.normal(size=(K, D)) * 3).astype(np.float32).astype(np.float64)
    x = (mus[z] + rng.normal(size=(N, D))).astype(np.float32).astype(np.float64)
    A = rng.normal(size=(K, 2, D, D)) * 0.3 / np.sqrt(D) + np.eye(D)
    inv_lr = A @ np.swapaxes(A, -1, -2)
    ld_lr = -np.linalg.slogdet(inv_lr)[1]
    mu_lr = mus[:, None] + 0.5 * rng.normal(size=(K, 2, D))
    lrw = rng.dirichlet([2, 2], size=K)
    ck = CudaKernel(prior_type.Gaussian, loglik_mode=LL_FP32).init(N, x, 3, points_major=True)
    ck.set_gaussian_params(mus, np.repeat(np.eye(D)[None], K, 0), np.zeros(K), np.full(K, 1.0 / K), mu_lr, inv_lr, ld_lr, lrw)
    labels = (z + 1).astype(np.int32)
    ck.set_labels(labels)
    u = uniforms(2 * N, D)
    r = ck.create_subclusters_labels(K, uniforms=u, return_loglik=True).astype(np.float64)
    sub = ck.get_sub_labels()
    _, _, r64 = O.gauss_sub_labels(x, labels, mu_lr, inv_lr, ld_lr, lrw, u.astype(np.float64))
    row_err = P.gauss_ll(r, r64, D, ld_lr[z], 0.0, "fp32", f"sub tiles D={D} K={K}")
    P.sub_labels_vs_fp64(sub, r64, labels, lrw, u.reshape(N, 2).astype(np.float64), row_err, f"sub tiles draws D={D} K={K}")
    cnt, sm, S = ck.create_sufficient_statistics(np.arange(K))
    cnt_o, sm_o, S_o = O.suff_stats(x, labels, sub, K)
    np.testing.assert_array_equal(cnt, cnt_o)
    d = x - mus[z]
    eps = 38 * 2.0 ** -24
    for k in range(K):
        for side in (1, 2):
            m = (z == k) & (sub == side)
            slot = 3 * k + side
            a1, a2 = np.abs(d[m]).sum(0), np.abs(d[m]).T @ np.abs(d[m])
            # a second-moment record is restored from the centred sums: their error times |s| twice, and its own
            s = np.abs(mus[k])
            e1 = eps * a1 + 1e-12
            e2 = eps * a2 + np.outer(s, e1) + np.outer(e1, s) + 1e-9
            np.testing.assert_array_less(np.abs(np.asarray(sm).reshape(3 * K, D)[slot] - np.asarray(sm_o).reshape(3 * K, D)[slot]), e1 + 1e-12)
            np.testing.assert_array_less(np.abs(np.asarray(S).reshape(3 * K, D, D)[slot] - np.asarray(S_o).reshape(3 * K, D, D)[slot]), e2)
    ck.release()
