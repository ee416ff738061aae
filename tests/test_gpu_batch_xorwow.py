"""Batches whose data sets draw from per-point cuRAND XORWOW states (dpmm_batch_create accepts the generator of
each run): the launches that time the block sizes must leave the states alone, so that the chain is that of
the data set run by itself, also when the timing is repeated after the clusters have doubled."""
import ctypes
from ctypes import byref, c_double, c_int32, c_int64, c_void_p

import numpy as np
import pytest

from dpmmsubclusters_gpu_b200 import capi, niw_hyperparams, prior_type
from dpmmsubclusters_gpu_b200.api import ModelInfo, dp_parallel_sampling_class
from dpmmsubclusters_gpu_b200.capi import check, lib

pytestmark = pytest.mark.gpu


def test_xorwow_batch_equals_separate_runs():
    rng = np.random.default_rng(5)
    shapes = [(3000, 2, 6), (2500, 2, 3), (2000, 16, 5)]
    iters = 30
    runs = (capi.dpmm_run_desc * len(shapes))()
    pts = (ctypes.POINTER(c_double) * len(shapes))()
    keep, samplers = [], []
    n, d = np.array([s[0] for s in shapes], np.int64), np.array([s[1] for s in shapes], np.int32)
    for i, (N, D, K) in enumerate(shapes):
        z = rng.integers(0, K, size=N)
        x = (rng.uniform(-10, 10, size=(K, D))[z] + rng.normal(size=(N, D))).T.copy()
        hyp = niw_hyperparams(1.0, np.zeros(D), D + 3.0, np.eye(D))
        s = dp_parallel_sampling_class(N, x, 3 + i, prior_type.Gaussian, loglik_mode=capi.LL_FP32,
                                       rng_kind=capi.RNG_CURAND_XORWOW, k_max=32)
        runs[i], k = s.run_desc(hyp, 5.0, iters, 1, False, 5)
        keep += [k, s.points]
        pts[i] = s.points.ctypes.data_as(ctypes.POINTER(c_double))
        samplers.append((s, hyp))
    h = c_void_p()
    check(lib().dpmm_batch_create(len(shapes), runs, n.ctypes.data_as(ctypes.POINTER(c_int64)),
                                  d.ctypes.data_as(ctypes.POINTER(c_int32)), pts, byref(h)))
    try:
        check(lib().dpmm_batch_step(h, iters))
        for i, (s, hyp) in enumerate(samplers):
            m = c_void_p()
            check(lib().dpmm_batch_model_info(h, i, byref(m)))
            mb = ModelInfo._from_handle(m)
            lib().dpmm_model_info_free(m)
            ms = s.dp_parallel(hyp, 5.0, iters=iters, init_clusters=1, verbose=False, burnout=5)
            assert ms.cluster_count_history.max() >= 2
            np.testing.assert_array_equal(mb.cluster_count_history, ms.cluster_count_history)
            np.testing.assert_array_equal(mb.labels, ms.labels)
            np.testing.assert_array_equal(mb.weights, ms.weights)
    finally:
        lib().dpmm_batch_destroy(h)
