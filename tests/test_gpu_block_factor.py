"""The block factorisation behind the marginal likelihoods, ratios and parameter draws at the dimensions where
its panels (8 columns), row groups (32) and padded sizes change, against numpy in FP64.

Tolerances: a marginal likelihood is a sum of terms of size up to n D log(..); each is good to a few units of
2^-52, the log determinant to about cond * D * 2^-52 with cond <= 1e4 here, so 1e-9 of the sum of the terms'
magnitudes covers it.  The drawn factors are FP32: W, b and c carry 2^-24 relative each, so b = W^T m holds to
(D + 2) 2^-23 |W|^T |m|, and c = log |det W| + log w to about D 2^-23 cond."""
import numpy as np
import pytest
from scipy.special import gammaln

pytestmark = pytest.mark.gpu


def _lml(n, s, S, D):
    k0, v0 = 1.0, D + 3.0
    if n == 0:
        return 0.0, 1.0
    kp, vp = k0 + n, v0 + n
    psi = (v0 * np.eye(D) + S - np.outer(s, s) / kp) / vp
    ld = np.linalg.slogdet(psi)[1]
    j = np.arange(D)
    t = [-n * D / 2 * np.log(np.pi), (gammaln(vp / 2 - j / 2) - gammaln(v0 / 2 - j / 2)).sum(), v0 / 2 * D * np.log(v0),
         -vp / 2 * (D * np.log(vp) + ld), D / 2 * np.log(k0 / kp)]
    return sum(t), sum(abs(v) for v in t)


@pytest.mark.parametrize("D", [1, 2, 3, 4, 7, 8, 9, 15, 17, 31, 32, 33, 40, 50, 63, 64, 65, 96, 100, 127, 128])
def test_factor_edges(D):
    from dpmmsubclusters_gpu_b200 import CudaKernel, niw_hyperparams, prior_type
    rng = np.random.default_rng(D)
    N, K, alpha = 900, 4, 3.0
    z = rng.integers(0, K - 1, size=N)   # cluster K - 1 stays empty
    x = rng.normal(size=(K, D))[z] * 2 + rng.normal(size=(N, D))
    sub = rng.integers(1, 3, size=N).astype(np.int32)
    sub[z == 1] = 1                      # an empty sub-cluster
    k = CudaKernel(prior_type.Gaussian, k_max=8).init(N, x, 1, points_major=True)
    k.set_prior(niw_hyperparams(1.0, np.zeros(D), D + 3.0, np.eye(D)))
    k.set_labels((z + 1).astype(np.int32))
    k.set_sub_labels(sub)
    cnt, sm, S = k.create_sufficient_statistics(np.arange(K))
    lml, _ = k.split_hastings(K, alpha)
    want = [[_lml(cnt[c, s], sm[c, s], S[c, s], D) for s in range(3)] for c in range(K)]
    for c in range(K):
        for s in range(3):
            assert abs(lml[c, s] - want[c][s][0]) <= 1e-9 * want[c][s][1], (c, s)
    hr = k.merge_hastings(K, alpha)
    i, j = 0, 2
    both, mag = _lml(cnt[i, 0] + cnt[j, 0], sm[i, 0] + sm[j, 0], S[i, 0] + S[j, 0], D)
    ni, nj = float(cnt[i, 0]), float(cnt[j, 0])
    g = [-np.log(alpha), gammaln(alpha), -2 * gammaln(alpha / 2), gammaln(ni + nj), -gammaln(ni + nj + alpha),
         gammaln(ni + alpha / 2), -gammaln(ni), -gammaln(nj), gammaln(nj + alpha / 2), both, -want[i][0][0], -want[j][0][0]]
    assert abs(hr[i, j] - sum(g)) <= 1e-9 * (mag + want[i][0][1] + want[j][0][1])
    assert np.isnan(hr[0, K - 1]) and np.isnan(hr[1, 0])
    np.testing.assert_array_equal(k.merge_hastings_list(K, alpha, [[i, j]]), [hr[i, j]])
    if D > 64:
        return
    w = np.full(K, 1.0 / K)
    k.sample_gaussian_params(K, 11, 1, w, np.full((K, 2), 0.5))
    W, b, cst, m = (a.astype(np.float64) for a in k.gaussian_params(K))
    for q in range(3 * K):
        bound = (D + 2) * 2.0 ** -23 * (np.abs(W[q]).T @ np.abs(m[q])) + 1e-30
        assert (np.abs(b[q] - W[q].T @ m[q]) <= bound + 2.0 ** -23 * np.abs(b[q])).all(), q
        cond = np.linalg.cond(W[q])
        ld = np.linalg.slogdet(W[q])[1] + (np.log(w[q // 3]) if q % 3 == 0 else 0.0)
        assert abs(cst[q] - ld) <= 2.0 ** -23 * (D * cond + abs(cst[q]) + 1), q
    k.release()
