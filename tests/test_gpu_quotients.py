"""quot64 and root64 (vb_physics.cuh), the quotients and square roots without a
range branch that the float64 kernels use, against `/` and sqrt bit for bit: on
random operands and on operands built so that the exact result lies as close to
a midpoint between two numbers as any can (a rounding decided by the last bit)."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "vespa.jl_b200", "csrc")

PROGRAM = r'''
#include "vb_physics.cuh"
__global__ void k(const double *a, const double *b, double *q, double *r, long long n)
{
    for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n; i += gridDim.x * 256ll) {
        q[i] = vb::quot64(a[i], b[i], vb::rcp64(b[i]));
        r[i] = vb::root64(a[i]);
    }
}
extern "C" int quotients(const double *a, const double *b, double *q, double *r, long long n)
{
    double *d = nullptr;
    const size_t w = sizeof(double) * (size_t)n;
    cudaError_t e = cudaMalloc(&d, 4 * w);
    if (e == cudaSuccess) e = cudaMemcpy(d, a, w, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + n, b, w, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k<<<1184, 256>>>(d, d + n, d + 2 * n, d + 3 * n, n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(q, d + 2 * n, w, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(r, d + 3 * n, w, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
'''


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not available")
    d = tmp_path_factory.mktemp("quotients")
    (d / "q.cu").write_text(PROGRAM)
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false",
                    "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared", "-I", CSRC,
                    str(d / "q.cu"), "-o", str(d / "q.so")], check=True, capture_output=True, timeout=300)
    L = C.CDLL(str(d / "q.so"))
    dp = C.POINTER(C.c_double)
    L.quotients.argtypes = [dp, dp, dp, dp, C.c_longlong]

    def run(a, b):
        a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
        q, r = np.empty_like(a), np.empty_like(a)
        p = [x.ctypes.data_as(dp) for x in (a, b, q, r)]
        assert L.quotients(*p, len(a)) == 0
        return q, r
    return run


def near_midpoint_quotients(count, seed):
    """a = (B m + e) / 2^s exactly, for 53-bit odd B, 54-bit odd m and small odd e:
    a / B is the midpoint m / 2^s but for e / (B 2^s)."""
    rng = np.random.default_rng(seed)
    A, Bs = [], []
    for B in (int(x) * 2 + 1 for x in rng.integers(2 ** 51, 2 ** 52, count)):
        for e in (-3, -1, 1, 3):
            for s in (53, 54):
                m = -e * pow(B, -1, 2 ** s) % 2 ** s
                m += 2 ** 53 if m < 2 ** 53 and s == 53 else 0
                a = (B * m + e) >> s
                if 2 ** 53 <= m < 2 ** 54 and 2 ** 52 <= a < 2 ** 53:
                    assert (a << s) == B * m + e
                    A.append(float(a))
                    Bs.append(float(B))
    return np.array(A), np.array(Bs)


def near_midpoint_roots(count):
    """x = m^2 - c for 54-bit odd m, small c and x a 53-bit number times 2^t: its
    root is the midpoint m but for c / 2 m."""
    X = []
    for c in range(1 - 8 * (count // 2), 8 * (count // 2), 8):
        s = 1
        for t in range(3, 56):  # lift s^2 = c (mod 2^t) a bit at a time
            if (s * s - c) % 2 ** (t + 1):
                s += 2 ** (t - 1)
        for t in (54, 55):
            for m in {(g * s + h) % 2 ** t for g in (1, -1) for h in (0, 2 ** (t - 1))}:
                if 2 ** 53 <= m < 2 ** 54 and (m * m - c) % 2 ** t == 0 and 2 ** 52 <= (m * m - c) >> t < 2 ** 53:
                    X.append(float((m * m - c) >> t) * 2.0 ** t)
    return np.array(X)


def test_near_midpoints_round_as_the_operators_do(device):
    a, b = near_midpoint_quotients(20000, seed=1)
    assert len(a) > 20000
    for scale in (1.0, 2.0 ** -100, 2.0 ** 90):
        q, _ = device(a * scale, b)
        assert np.array_equal(q, a * scale / b)
        q, _ = device(-a, b * scale)
        assert np.array_equal(q, -a / (b * scale))
    x = near_midpoint_roots(20000)
    assert len(x) > 10000
    for scale in (1.0, 2.0 ** -100, 2.0 ** 90):
        _, r = device(x * scale, np.ones_like(x))
        assert np.array_equal(r, np.sqrt(x * scale))


def test_random_operands_round_as_the_operators_do(device):
    rng = np.random.default_rng(7)
    n = 1 << 22
    for span in (1, 100):
        a, b = (rng.uniform(1, 2, n) * np.exp2(rng.integers(-span, span, n)) for _ in range(2))
        q, r = device(a, b)
        assert np.array_equal(q, a / b)
        assert np.array_equal(r, np.sqrt(a))
    a[: n // 2] = 0.0
    q, _ = device(a, b)
    assert np.array_equal(q, a / b)
