"""Contexts on threads of their own (include/dpmm_capi.h: separate contexts may be used concurrently) whose K or
D ask the same kernels for different amounts of shared memory.  The limit of a kernel belongs to the device:
every call succeeds, and gives what it gives alone."""
import ctypes
import threading

import numpy as np
import pytest

from conftest import uniforms
from dpmmsubclusters_gpu_b200 import LL_FP32, LL_TC_BF16X3, CudaKernel, prior_type
from dpmmsubclusters_gpu_b200.capi import lib

pytestmark = pytest.mark.gpu

N, ROUNDS = 256, 2000


class _Context:
    def __init__(self, seed):
        self.u = uniforms(2 * N, seed)
        self.up = self.u.ctypes.data_as(ctypes.POINTER(ctypes.c_float))

    def result(self):
        assert self.call() == 0
        return [self.ck.get_labels(), self.ck.get_sub_labels()]


class _Gauss(_Context):
    def __init__(self, D, K, mode, spread=0.3):
        super().__init__(K)
        rng = np.random.default_rng(D + K)
        self.z = (np.arange(N) % K + 1).astype(np.int32)
        mus = spread * rng.normal(size=(K, D))
        x = mus[self.z - 1] + rng.normal(size=(N, D))
        self.ck, self.K = CudaKernel(prior_type.Gaussian, loglik_mode=mode, k_max=256).init(N, x, 1, points_major=True), K
        lib().dpmm_set_label_pruning(self.ck.ctx, 30.0 if spread > 1 else 0.0)
        eye = np.eye(D)
        self.ck.set_gaussian_params(mus, np.repeat(eye[None], K, 0), np.zeros(K), np.full(K, 1.0 / K))
        self.ck.set_labels(self.z)
        self.ck.set_sub_labels(np.ones(N, np.int32))

    def call(self):
        return lib().dpmm_create_clusters_labels(self.ck.ctx, self.K, 0, self.up, None)


class _Mult(_Context):
    def __init__(self, D, K):
        super().__init__(K)
        rng = np.random.default_rng(D + K)
        self.ck, self.K = CudaKernel(prior_type.Multinomial, k_max=128).init(
            N, rng.poisson(100.0 / D, size=(N, D)).astype(np.float64), 1, points_major=True), K
        lt = np.log(rng.dirichlet(np.ones(D), size=(K, 3)))
        self.ck.set_multinomial_params(lt[:, 0], None, lt[:, 1:], np.full((K, 2), 0.5))

    def call(self):
        return (lib().dpmm_create_clusters_labels(self.ck.ctx, self.K, 0, self.up, None) or
                lib().dpmm_create_subclusters_labels(self.ck.ctx, self.K, self.up, None))


@pytest.mark.parametrize("make", [
    pytest.param([lambda: _Gauss(64, 20, LL_TC_BF16X3), lambda: _Gauss(64, 120, LL_TC_BF16X3)], id="dense_d64"),
    pytest.param([lambda: _Gauss(32, 60, LL_TC_BF16X3), lambda: _Gauss(32, 90, LL_TC_BF16X3)], id="dense_d32"),
    pytest.param([lambda: _Gauss(7, 3, LL_FP32), lambda: _Gauss(7, 120, LL_FP32)], id="fp32_d7"),
    pytest.param([lambda: _Gauss(16, 20, LL_FP32, 9.0), lambda: _Gauss(16, 200, LL_FP32, 9.0)], id="pruned_d16"),
    pytest.param([lambda: _Mult(100, 70), lambda: _Mult(1000, 33), lambda: _Mult(500, 90)], id="multinomial"),
])
def test_contexts_on_threads(make):
    ctxs = [f() for f in make for _ in range(2)]
    want = [c.result() for c in ctxs]
    errors = []
    start = threading.Barrier(len(ctxs))

    def work(c):
        start.wait()
        for _ in range(ROUNDS):
            if c.call() != 0:
                errors.append(lib().dpmm_last_error())
    ts = [threading.Thread(target=work, args=(c,)) for c in ctxs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, (len(errors), errors[0])
    for c, w in zip(ctxs, want):
        for a, b in zip(c.result(), w):
            np.testing.assert_array_equal(a, b)
        c.ck.release()
