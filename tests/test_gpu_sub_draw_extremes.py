"""Two-way sub-label draw (draw_sub_label, csrc/dpmm_device.cuh) where a log weight is infinite or NaN.  The
reference's softmax then has no finite sum, its comparisons are all false, and the label is the column of
the first uniform (cudaKernel.cu:352-372, 102-124); a weight of zero (log weight -inf) never draws its side."""
import numpy as np
import pytest

from conftest import uniforms
from dpmmsubclusters_gpu_b200 import LL_FP32, CudaKernel, prior_type
from dpmmsubclusters_gpu_b200.capi import check, lib

pytestmark = pytest.mark.gpu

WEIGHTS = [(np.inf, 0.5), (0.5, np.inf), (np.inf, np.inf), (np.nan, 0.5), (0.5, np.nan), (0.0, 0.5), (0.5, 0.0), (0.0, 0.0)]


@pytest.mark.parametrize("prior,D,mode,fused", [("g", 3, LL_FP32, 0), ("g", 16, LL_FP32, 0), ("g", 64, LL_FP32, 0), ("g", 100, None, 0),
                                                ("g", 32, None, 0), ("g", 64, None, 0), ("g", 32, None, 1), ("g", 64, None, 1),
                                                ("m", 20, None, 0)])
def test_infinite_log_weights(prior, D, mode, fused):
    rng = np.random.default_rng(D)
    K = len(WEIGHTS)
    N = 150 * K
    z = np.arange(N) % K
    lrw = np.array(WEIGHTS)
    if prior == "g":
        x = rng.normal(size=(N, D))
        ck = CudaKernel(prior_type.Gaussian, loglik_mode=mode, k_max=16).init(N, x, 1, points_major=True)
        check(lib().dpmm_set_fused_sub_stats(ck.ctx, fused))
        eye = np.eye(D)
        with np.errstate(divide="ignore"):
            ck.set_gaussian_params(np.zeros((K, D)), np.repeat(eye[None], K, 0), np.zeros(K), np.full(K, 1.0 / K),
                                   0.1 * rng.normal(size=(K, 2, D)), np.broadcast_to(eye, (K, 2, D, D)), np.zeros((K, 2)), lrw)
    else:
        x = rng.poisson(3.0, size=(N, D)).astype(np.float64)
        ck = CudaKernel(prior_type.Multinomial, k_max=16).init(N, x, 1, points_major=True)
        lt = np.log(rng.dirichlet(np.ones(D), size=(K, 3)))
        ck.set_multinomial_params(lt[:, 0], None, lt[:, 1:], lrw)
    u = uniforms(2 * N, 7).reshape(N, 2)
    ck.set_labels((z + 1).astype(np.int32))
    ck.create_subclusters_labels(K, uniforms=u)
    sub = ck.get_sub_labels()
    ck.release()
    col = (u[:, 0].astype(np.float64) * 1.999999 + 1).astype(int)
    want = np.where(z == 5, 2, np.where(z == 6, 1, col))
    np.testing.assert_array_equal(sub, want)
