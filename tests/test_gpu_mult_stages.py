"""The staged multinomial sub-label + statistics kernel at the widths where its stages change: 32 categories (64
rows a stage) to 4096 (four rows), thread groups that do not divide the block, tiles and chunks with
remainders, against the FP64 oracle.  Counts and count sums are whole numbers and must be equal; a
log-likelihood is an FP32 sum of D products (at most 2^-24 D of the sum of their magnitudes), and a sub-label
may differ from the oracle's draw only within the margin that such an error can move."""
import numpy as np
import pytest

from conftest import uniforms
from dpmmsubclusters_gpu_b200 import CudaKernel, prior_type
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [1, 31, 33, 64, 100, 250, 1000, 1024, 1025, 2048, 2100, 3000, 4096])
@pytest.mark.parametrize("sizes", [[1, 127, 128, 129], [7, 300]])
def test_stages(D, sizes):
    rng = np.random.default_rng(D)
    K = len(sizes)
    z = rng.permutation(np.repeat(np.arange(K), sizes))
    N = z.size
    x = rng.poisson(3.0 if D < 200 else 0.4, size=(N, D)).astype(np.float64)
    theta = rng.dirichlet(np.ones(D), size=(K, 3))
    lt = np.log(theta * 0.9 + 0.1 / D)
    lrw = rng.dirichlet([2, 2], size=K)
    ck = CudaKernel(prior_type.Multinomial, k_max=8).init(N, x, 1, points_major=True)
    ck.set_multinomial_params(lt[:, 0], None, lt[:, 1:], lrw)
    ck.set_labels((z + 1).astype(np.int32))
    u = uniforms(2 * N, D)
    r = ck.create_subclusters_labels(K, uniforms=u, return_loglik=True).astype(np.float64)
    sub = ck.get_sub_labels()
    r64 = np.stack([(x * lt[z, 1 + s]).sum(1) for s in range(2)], 1)
    bound = 2.0 ** -24 * (D + 8) * np.stack([(x * np.abs(lt[z, 1 + s])).sum(1) for s in range(2)], 1) + 1e-6
    assert (np.abs(r - r64) <= bound).all()
    q = r64 + np.log(lrw[z])
    p = np.exp(q - q.max(1, keepdims=True))
    p /= p.sum(1, keepdims=True)
    uu = u.reshape(N, 2).astype(np.float64)
    col = (uu[:, 0] * 1.999999 + 1).astype(int)
    y = 2 * p[np.arange(N), col - 1]
    want = np.where((y < 1) & (y < uu[:, 1]), 3 - col, col)
    bad = sub != want
    assert (np.minimum(np.abs(y - uu[:, 1]), np.abs(y - 1))[bad] <= 2 * bound.sum(1)[bad] + 1e-6).all()
    for given in (False, True):          # the drawn sub-labels' statistics, then those of given ones
        if given:
            sub = rng.integers(1, 3, size=N).astype(np.int32)
            ck.set_sub_labels(sub)
        cnt, sm, _ = ck.create_sufficient_statistics(np.arange(K))
        for k in range(K):
            for s in (1, 2):
                rows = x[(z == k) & (sub == s)]
                assert cnt[k, s] == len(rows)
                np.testing.assert_array_equal(sm[k, s], rows.sum(0))
            np.testing.assert_array_equal(sm[k, 0], x[z == k].sum(0))
    ck.release()
