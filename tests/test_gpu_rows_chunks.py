"""The persistent sub-label kernel (csrc/dpmm_rows_tc.cu) where every CTA walks at least five chunks, so that both
operand buffers are filled again while they are drained and every ring of tile slots wraps several times: equal
bit for bit to the one-block-per-chunk fused pass.  And the fused pass switched on after the parameters were set,
twice: at Dp = 32 its operand is packed at the switch."""
import numpy as np
import pytest
import torch

from conftest import uniforms
from dpmmsubclusters_gpu_b200 import LL_TC_BF16X3, CudaKernel, prior_type
from dpmmsubclusters_gpu_b200.capi import check, lib

pytestmark = pytest.mark.gpu


def _params(rng, K, D):
    mus = rng.normal(size=(K, D)) * 3
    A = rng.normal(size=(K, 2, D, D)) * 0.3 / np.sqrt(D) + np.eye(D)
    inv_lr = A @ np.swapaxes(A, -1, -2)
    return (mus, np.repeat(np.eye(D)[None], K, 0), np.zeros(K), np.full(K, 1.0 / K), mus[:, None] + 0.5 * rng.normal(size=(K, 2, D)),
            inv_lr, -np.linalg.slogdet(inv_lr)[1], rng.dirichlet([2, 2], size=K))


@pytest.mark.parametrize("D", [20, 32, 64])
@pytest.mark.parametrize("K,lo,hi", [(1000, 1, 300), (800, 385, 500), (760, 128, 129)])
def test_five_chunks_per_block(D, K, lo, hi):
    rng = np.random.default_rng(D + K)
    sizes = rng.integers(lo, hi + 1, size=K)
    assert K >= 5 * torch.cuda.get_device_properties(0).multi_processor_count   # a cluster is at least one chunk
    z = rng.permutation(np.repeat(np.arange(K), sizes))
    N = z.size
    params = _params(rng, K, D)
    x = params[0][z] + rng.normal(size=(N, D))
    u = uniforms(2 * N, D)
    got = []
    for fused in (1, 0):
        ck = CudaKernel(prior_type.Gaussian, loglik_mode=LL_TC_BF16X3, k_max=1024).init(N, x, 3, points_major=True)
        check(lib().dpmm_set_fused_sub_stats(ck.ctx, fused))
        ck.set_gaussian_params(*params)
        ck.set_labels((z + 1).astype(np.int32))
        r = ck.create_subclusters_labels(K, uniforms=u, return_loglik=True)
        got.append((np.asarray(r), ck.get_sub_labels()))
        ck.release()
    np.testing.assert_array_equal(got[1][0], got[0][0])
    np.testing.assert_array_equal(got[1][1], got[0][1])


@pytest.mark.parametrize("D", [20, 64])
def test_fused_switched_on_after_the_parameters(D):
    rng = np.random.default_rng(D)
    K, N = 9, 6000
    z = rng.integers(0, K, size=N)
    p1, p2 = _params(rng, K, D), _params(rng, K, D)
    ck = CudaKernel(prior_type.Gaussian, loglik_mode=LL_TC_BF16X3, k_max=16).init(N, p1[0][z] + rng.normal(size=(N, D)), 3, points_major=True)
    ck.set_labels((z + 1).astype(np.int32))
    u = uniforms(2 * N, D)

    def run(fused):
        check(lib().dpmm_set_fused_sub_stats(ck.ctx, fused))
        r = ck.create_subclusters_labels(K, uniforms=u, return_loglik=True)
        return np.asarray(r), ck.get_sub_labels()
    for p in (p1, p2, p1):
        ck.set_gaussian_params(*p)     # the flag is off here
        a, b = run(0), run(1)
        np.testing.assert_array_equal(a[0], b[0])
        np.testing.assert_array_equal(a[1], b[1])
        check(lib().dpmm_set_fused_sub_stats(ck.ctx, 0))
    ck.release()
