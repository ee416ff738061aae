"""The quotients of the FP64 factorisation (Divisor, csrc/dpmm_niw.cuh) against the division: bit for bit
where the quotient is zero, infinite, NaN or at least 2^-960 in magnitude, within two units of the last place
below that (four of the smallest subnormal where the quotient is one), and a ratio whose scale matrix overflows."""
import ctypes
import subprocess

import numpy as np
import pytest

from dpmmsubclusters_gpu_b200 import build as B

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "dpmm_niw.cuh"
__global__ void k_quotients(const double* a, const double* b, double* q, long long n)
{
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n) q[i] = dpmm::Divisor(b[i])(a[i]);
}
extern "C" int quotients(const double* a, const double* b, double* q, long long n)
{
    double* d = nullptr;
    if (cudaMalloc(&d, 24 * n) != cudaSuccess) return 1;
    cudaMemcpy(d, a, 8 * n, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, 8 * n, cudaMemcpyHostToDevice);
    k_quotients<<<(unsigned)((n + 255) / 256), 256>>>(d, d + n, d + 2 * n, n);
    const int e = (int)cudaMemcpy(q, d + 2 * n, 8 * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e;
}
"""


@pytest.fixture(scope="module")
def quotients(tmp_path_factory):
    d = tmp_path_factory.mktemp("divisor")
    (d / "q.cu").write_text(SOURCE)
    so = str(d / "q.so")
    subprocess.run([B.NVCC] + B.NVCC_FLAGS + ["-shared", "-o", so, str(d / "q.cu"), B.LIB, "-Xlinker", "-rpath," + B.HERE],
                   check=True, capture_output=True)
    fn = ctypes.CDLL(so).quotients
    fn.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_longlong]

    def run(a, b):
        a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
        q = np.empty_like(a)
        assert fn(a.ctypes.data, b.ctypes.data, q.ctypes.data, a.size) == 0
        return q
    return run


def _same(q, w, a, b):
    bad = ~((q.view(np.int64) == w.view(np.int64)) | (np.isnan(q) & np.isnan(w)))
    assert not bad.any(), [(x.hex(), y.hex(), u.hex(), v.hex()) for x, y, u, v in
                           list(zip(a[bad], b[bad], q[bad], w[bad]))[:5]]


@pytest.mark.parametrize("span", [0, 3, 60, 500, 1022])
def test_quotients_equal_the_division(quotients, span):
    rng = np.random.default_rng(span)
    n = 4_000_000
    mant = lambda: (1 + rng.random(n)) * rng.choice([-1.0, 1.0], size=n)
    a = np.ldexp(mant(), rng.integers(-span, span + 1, size=n))
    b = np.ldexp(mant(), rng.integers(-span, span + 1, size=n))
    hard = rng.integers(0, 1 << 20, size=n // 4)        # mantissas next to a power of two
    b[:n // 4] = np.ldexp(1 + hard * 2.0 ** -52, rng.integers(-span, span + 1, size=n // 4))
    with np.errstate(all="ignore"):
        w = a / b
    q = quotients(a, b)
    big = ~(np.abs(w) < 2.0 ** -960)
    _same(q[big], w[big], a[big], b[big])
    ulp = np.maximum(np.spacing(np.abs(w[~big])), 2 * 2.0 ** -1074)
    off = np.abs(q[~big] - w[~big]) > 2 * ulp
    assert not off.any(), [(x.hex(), y.hex(), u.hex(), v.hex()) for x, y, u, v in
                           list(zip(a[~big][off], b[~big][off], q[~big][off], w[~big][off]))[:5]]


def test_quotients_of_special_values(quotients):
    v = np.array([0.0, 5e-324, 2.2e-308, 2.3e-308, 1e-300, 0.3, 1.0, 3.0, 1e300, 8.9e307, 1.7976931348623157e308, np.inf])
    v = np.concatenate([v, -v, [np.nan]])
    a, b = (t.ravel() for t in np.meshgrid(v, v))
    with np.errstate(all="ignore"):
        w = a / b
    q = quotients(a, b)
    big = ~((np.abs(w) < 2.0 ** -960) & (w != 0) & (np.abs(a) != 0))
    _same(q[big], w[big], a[big], b[big])
    assert (np.abs(q[~big] - w[~big]) <= 4 * 2.0 ** -1074 + 2.0 ** -50 * np.abs(w[~big])).all()


@pytest.mark.parametrize("D", [1, 2, 40])
def test_merge_ratio_of_an_overflowing_scatter(D):
    # each cluster's scatter is finite, their sum overflows: log det psi' = inf, the merged marginal likelihood -inf
    import torch
    from dpmmsubclusters_gpu_b200.capi import check, lib
    K, sl = 2, 1 + D + D * D
    st = np.zeros((3 * K, sl))
    for k in range(K):
        st[3 * k, 0] = 10.0
        st[3 * k, 1 + D:] = (1e308 * np.eye(D)).ravel()
    prior = np.concatenate([np.zeros(D), np.eye(D).ravel()])
    d_st, d_pr = torch.from_numpy(st).cuda(), torch.from_numpy(prior).cuda()
    hr = torch.zeros(K * K, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    check(lib().dpmm_merge_hastings_static(0, D, K, 2.0, 1.0, D + 3.0, p(d_pr), p(d_st), p(hr), None))
    torch.cuda.synchronize()
    assert hr.cpu().numpy()[1] == -np.inf
