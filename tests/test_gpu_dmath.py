"""The short double-precision quotient and root of the polyhedron kernel (fxe_dmath.cuh) against the
correctly rounded operations, over operands of every kind: bit for bit, with nothing to tolerate."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from flexaidds_gb300 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "fxe_dmath.cuh"
__global__ void short_ops(const double* a, const double* b, double* q, double* s, float* t, double* w, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    bool slow;
    double v = fxe::div_short(a[i], b[i], &slow);
    q[i] = slow ? fxe::plain_div(a[i], b[i]) : v;
    v = fxe::sqrt_short(a[i], &slow);
    s[i] = slow ? fxe::plain_sqrt(a[i]) : v;
    t[i] = fxe::d2f_trunc(a[i]);
    w[i] = fxe::f2d((float)b[i]);
}
__global__ void comparisons(const double* a, const double* b, int* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        out[i] = fxe::gt0(a[i]) | fxe::lt0(a[i]) << 1 | fxe::is0(a[i]) << 2 | fxe::lt_nn(a[i], b[i]) << 3 |
                 fxe::le_nn(a[i], b[i]) << 4;
}
extern "C" int compare(const double* a, const double* b, int* out, int n) {
    double* d = nullptr;
    const size_t z = sizeof(double) * n;
    if (cudaMalloc(&d, 3 * z) != cudaSuccess) return 1;
    cudaMemcpy(d, a, z, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, z, cudaMemcpyHostToDevice);
    comparisons<<<(n + 255) / 256, 256>>>(d, d + n, (int*)(d + 2 * n), n);
    cudaMemcpy(out, d + 2 * n, sizeof(int) * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return cudaGetLastError() != cudaSuccess;
}
extern "C" int run(const double* a, const double* b, double* q, double* s, float* t, double* w, int n) {
    double* d = nullptr;
    const size_t z = sizeof(double) * n;
    if (cudaMalloc(&d, 6 * z) != cudaSuccess) return 1;
    cudaMemcpy(d, a, z, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, z, cudaMemcpyHostToDevice);
    short_ops<<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * n, d + 3 * n, (float*)(d + 4 * n), d + 5 * n, n);
    cudaMemcpy(q, d + 2 * n, z, cudaMemcpyDeviceToHost);
    cudaMemcpy(s, d + 3 * n, z, cudaMemcpyDeviceToHost);
    cudaMemcpy(t, d + 4 * n, z / 2, cudaMemcpyDeviceToHost);
    cudaMemcpy(w, d + 5 * n, z, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return cudaGetLastError() != cudaSuccess;
}
"""


@pytest.fixture(scope="module")
def ops(tmp_path_factory):
    d = tmp_path_factory.mktemp("dmath")
    (d / "ops.cu").write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "--fmad=false", "-Xcompiler", "-fPIC", "-shared",
                    "-cudart", "static", "-I", build.CSRC, "-o", str(d / "ops.so"), str(d / "ops.cu")], check=True)
    lib = C.CDLL(os.path.join(str(d), "ops.so"))

    def run(a, b):
        q, s, w, t = (np.empty(len(a)) for _ in range(3)), None, None, np.empty(len(a), np.float32)
        q, s, w = q
        p = [x.ctypes.data_as(C.c_void_p) for x in (a, b, q, s, t, w)]
        assert lib.run(*p, C.c_int(len(a))) == 0
        return q, s, t, w
    run.lib = lib
    return run


def _operands(kind, n, rng):
    if kind == "ordinary":
        return rng.normal(0.0, 10.0, n), rng.normal(0.0, 10.0, n)
    if kind == "wide":         # the edges of the short forms' exponent range
        e = rng.integers(-360, 361, (2, n))
        return tuple(np.ldexp(rng.uniform(1.0, 2.0, n) * rng.choice([-1.0, 1.0], n), k) for k in e)
    if kind == "bits":         # every exponent, denormals, infinities and NaN among them
        return tuple(rng.integers(0, 1 << 64, n, dtype=np.uint64).view(np.float64) for _ in range(2))
    if kind == "midway":       # quotients and roots next to the midpoint of two doubles
        b = rng.integers(1 << 52, 1 << 53, n).astype(np.float64)
        q = rng.integers(1 << 52, 1 << 53, n).astype(np.float64)
        a = q * b
        return np.nextafter(a, np.where(rng.random(n) < 0.5, 0.0, np.inf)), b
    special = np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 5e-324, 2.0 ** -1022, 1.7e308,
                        np.nextafter(2.0, 1.0), np.nextafter(4.0, 1.0), 2.0 ** 350, 2.0 ** -350, 1.0 + 2.0 ** -52])
    return tuple(np.ascontiguousarray(x.ravel()) for x in np.meshgrid(special, special))


@pytest.mark.parametrize("kind", ["ordinary", "wide", "bits", "midway", "special"])
def test_short_operations_are_correctly_rounded(ops, kind):
    a, b = _operands(kind, 1 << 20, np.random.default_rng(17))
    q, s, t, w = ops(a, b)
    with np.errstate(all="ignore"):
        for got, want in ((q, a / b), (s, np.sqrt(a)), (w, b.astype(np.float32).astype(np.float64))):
            same = (got.view(np.uint64) == want.view(np.uint64)) | (np.isnan(got) & np.isnan(want))
            assert same.all(), (kind, a[~same][:3], b[~same][:3])
        # truncated toward zero, below the normal range to zero, past the range to infinity
        f = np.abs(t.astype(np.float64))
        normal = (np.abs(a) >= 2.0 ** -126) & (np.abs(a) < 2.0 ** 128)
        assert np.all(f[normal] <= np.abs(a[normal])) and np.all(np.abs(a[normal]) - f[normal] < np.abs(a[normal]) * 2.0 ** -22)
        assert np.all(t[np.abs(a) < 2.0 ** -126] == 0.0) and np.all(np.isinf(t[np.abs(a) >= 2.0 ** 128]))


def _square_root_mod(u, n):
    """r with r * r = u (mod 2^n), u = 1 (mod 8), a bit at a time."""
    r = 1
    for i in range(3, n):
        if (r * r - u) % (1 << (i + 1)):
            r += 1 << (i - 1)
    return r % (1 << n)


def _roots_beside_midpoints(n):
    """x whose root lies as close to the midpoint of two doubles as a root can: k is a midpoint's 54-bit
    significand, k^2 = u (mod 2^54) with a small u, and x = (k^2 - u) / 2^54 is a significand of 53 bits."""
    out, m = [], 1 << 54
    for u in range(1 - 8 * n, 8 * n, 8):
        r = _square_root_mod(u, 54)
        for k in {r, -r % m, (r + m // 2) % m, (m // 2 - r) % m}:
            x = (k * k - u) >> 54
            if k >= m // 2 and x < m and (x < m // 2 or x % 2 == 0):
                out.append(x)
    return np.array(out, np.float64)


def _quotients_beside_midpoints(divisors):
    """(a, b) whose quotient lies as close to a midpoint as one can: a 2^54 = c (mod b), c small and odd."""
    a, b = [], []
    for B in divisors:
        inv = pow(2, -54, B)
        for c in (-7, -5, -3, -1, 1, 3, 5, 7):
            for A in (c * inv % B, 2 * c * inv % B + B):
                if 1 << 52 <= A < 1 << 53:
                    a.append(A)
                    b.append(B)
    return np.array(a, np.float64), np.array(b, np.float64)


def test_roots_beside_midpoints(ops):
    x = _roots_beside_midpoints(6000)
    assert len(x) > 10000
    rng = np.random.default_rng(3)
    x = np.ldexp(x, 2 * rng.integers(-150, 150, len(x)))
    s = ops(x, np.ones(len(x)))[1]
    wrong = s != np.sqrt(x)
    assert not wrong.any(), (int(wrong.sum()), x[wrong][:3])


def test_quotients_beside_midpoints(ops):
    """Divisors of every kind, and those just below a power of two: their reciprocal lies beside a midpoint
    itself ((2^53 - k) (2^53 + k) = 2^106 - k^2), where its rounding is uncertain."""
    rng = np.random.default_rng(4)
    any_b = [int(v) | 1 for v in rng.integers(1 << 52, 1 << 53, 20000)]
    near = [(1 << 53) - k for k in range(1, 20001, 2)] + [(1 << 52) + k for k in range(1, 2001, 2)]
    a, b = _quotients_beside_midpoints(any_b + near)
    assert len(a) > 100000
    ea, eb = rng.integers(-250, 250, (2, len(a)))
    a = np.ldexp(a * rng.choice([-1.0, 1.0], len(a)), ea)
    b = np.ldexp(b * rng.choice([-1.0, 1.0], len(b)), eb)
    q = ops(a, b)[0]
    wrong = q != a / b
    assert not wrong.any(), (int(wrong.sum()), a[wrong][:3], b[wrong][:3])


def test_comparisons_on_bit_patterns(ops):
    """Signs of any value; order of values whose sign bit is clear, with NaN of both signs among them."""
    rng = np.random.default_rng(6)
    special = np.array([0.0, 5e-324, 2.0 ** -1022, 1.0, 1.0 + 2.0 ** -52, 1.7e308, np.inf, np.nan, -np.nan])
    a, b = (np.ascontiguousarray(x.ravel()) for x in np.meshgrid(special, special))
    x = np.abs(rng.normal(0.0, 1.0, 1000))
    a, b = np.concatenate([a, x]), np.concatenate([b, np.where(rng.random(1000) < 0.3, x, x[::-1])])
    out = np.zeros(len(a), np.int32)
    args = [v.ctypes.data_as(C.c_void_p) for v in (a, b, out)]
    assert ops.lib.compare(*args, C.c_int(len(a))) == 0
    np.testing.assert_array_equal(out >> 3, (a < b) | (a <= b).astype(int) << 1)
    s = np.concatenate([special, -special, rng.normal(0.0, 1.0, 1000)])
    out = np.zeros(len(s), np.int32)
    args = [v.ctypes.data_as(C.c_void_p) for v in (s, s, out)]
    assert ops.lib.compare(*args, C.c_int(len(s))) == 0
    np.testing.assert_array_equal(out & 7, (s > 0.0) | (s < 0.0).astype(int) << 1 | (s == 0.0).astype(int) << 2)
