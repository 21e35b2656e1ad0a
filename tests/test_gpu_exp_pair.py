"""exp_and_m1, the pair exp(x) and exp(x) - 1 of the FP64 propagators, against 60-digit decimal values.

A kernel built from the header evaluates it on arguments over its whole range: |x| down to 1e-300, the
reduction's seams (half-odd multiples of ln 2, k = 0 to -1 at x = -ln(2)/2 among them) and its centres, both
sides of x = -700 where the library's exp takes over, results below the normal range, and the special values.
Bound: one ulp of the exact value, what the function states (half an ulp of the last rounding, the rest of
the sum, whose terms are at most 0.42 of the result's leading one, below half).
"""
import ctypes
import math
import subprocess
from decimal import Decimal, getcontext

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KERNEL = r"""
#include "pffrg_flow.cuh"
__global__ void pair(const double* x, double* e, double* m, int n) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) pffrg::exp_and_m1(x[k], e[k], m[k]);
}
extern "C" int exp_pair(const double* x, double* e, double* m, int n) {
    double* d = nullptr;
    cudaError_t rc = cudaMalloc(&d, sizeof(double) * 3 * n);
    if (rc) return (int)rc;
    rc = cudaMemcpy(d, x, sizeof(double) * n, cudaMemcpyHostToDevice);
    if (!rc) pair<<<(n + 127) / 128, 128>>>(d, d + n, d + 2 * n, n), rc = cudaGetLastError();
    if (!rc) rc = cudaMemcpy(e, d + n, sizeof(double) * n, cudaMemcpyDeviceToHost);
    if (!rc) rc = cudaMemcpy(m, d + 2 * n, sizeof(double) * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)rc;
}
"""


@pytest.fixture(scope="module")
def pair(pkg, tmp_path_factory):
    import pffrg_gb300.build as b

    d = tmp_path_factory.mktemp("exp_pair")
    (d / "pair.cu").write_text(KERNEL)
    subprocess.run([b.NVCC, *b.ARCH, *b.FLAGS, "-I", str(b.CSRC), "-shared", "-o", str(d / "pair.so"), str(d / "pair.cu"),
                    "-lcudart"], check=True)
    f = ctypes.CDLL(str(d / "pair.so")).exp_pair
    f.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int]

    def run(x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        e, m = np.empty_like(x), np.empty_like(x)
        assert f(x.ctypes.data, e.ctypes.data, m.ctypes.data, len(x)) == 0
        return e, m

    return run


def arguments():
    rng = np.random.default_rng(11)
    xs = [-np.exp(rng.uniform(math.log(1e-20), math.log(700.0), 3000)), -rng.uniform(0.0, 2.0, 2000),
          -rng.uniform(600.0, 760.0, 500), -(10.0 ** -np.arange(1.0, 300.0, 7.0))]
    for k in list(range(0, 24)) + [500, 1008, 1009, 1010]:
        for c in (k, k + 0.5):
            x = -c * math.log(2.0)
            for _ in range(3):
                xs.append([x])
                x = np.nextafter(x, -np.inf)
            xs.append([np.nextafter(-c * math.log(2.0), np.inf)])
    xs.append([np.nextafter(-700.0, 0.0), -700.0, np.nextafter(-700.0, -np.inf), -708.4, -745.1, -746.0, -1e5, -1e300])
    x = np.concatenate([np.asarray(v, dtype=np.float64) for v in xs])
    return x[x < 0]


def ulps(got, exact):
    """Distance from the exact value in ulps of it."""
    m, e = math.frexp(float(exact))
    ulp = Decimal(2) ** max(e - 53, -1074)
    return float(abs(Decimal(got) - exact) / ulp)


def test_exp_pair_within_an_ulp(pair):
    getcontext().prec = 60
    getcontext().Emin = -10**9
    x = arguments()
    e, m = pair(x)
    worst = [0.0, 0.0]
    for xi, ei, mi in zip(x.tolist(), e.tolist(), m.tolist()):
        d = Decimal(xi)
        if xi < -1e5:
            assert ei == 0.0 and mi == -1.0
            continue
        ref = d.exp()
        # where e^x - 1 would lose digits, four terms of its series hold them all
        m1 = d + d * d / 2 + d * d * d / 6 + d ** 4 / 24 if abs(xi) < 1e-12 else ref - 1
        worst = [max(worst[0], ulps(ei, ref)), max(worst[1], ulps(mi, m1))]
    print(f"{len(x)} arguments: exp {worst[0]:.3f}, exp - 1 {worst[1]:.3f} ulp")
    assert worst[0] <= 1.0 and worst[1] <= 1.0


def test_exp_pair_special_values(pair):
    e, m = pair([0.0, -0.0, -np.inf, np.nan])
    assert e[0] == e[1] == 1.0 and m[0] == m[1] == 0.0
    assert e[2] == 0.0 and m[2] == -1.0
    assert np.isnan(e[3]) and np.isnan(m[3])
