"""Quotients and square roots of cumc_round.cuh against the IEEE operators,
bit for bit: random operands over the stated ranges and the operands whose
quotient or root lies nearest to a rounding midpoint. On the CPU the
approximate seeds carry the largest error the header allows; on the GPU they
are the hardware's, whose error is checked against that bound too."""
import ctypes
import math
import os
import random
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "cumpic_b200", "csrc", "cumc_round.cuh")
SEED_ERR = 2.0 ** -19

CPU_SRC = """
#include "%s"
extern "C" void run(long n, const double* a, const double* b, const double* e, double* q, double* r) {
    for (long i = 0; i < n; ++i) {
        const double y = (1.0 / b[i]) * (1.0 + e[i]), s = (1.0 / std::sqrt(b[i])) * (1.0 + e[i]);
        q[i] = cumc::quot(a[i], b[i], cumc::recip_refine(b[i], y));
        r[i] = cumc::root_refine(b[i], s);
    }
}
""" % HEADER

GPU_SRC = """
#include "%s"
#include <cuda_runtime.h>
using namespace cumc;
__global__ void k(long n, const double* a, const double* b, double* q, double* r, double* ey, double* es) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    q[i] = quot_signed(a[i], b[i], recip_of(b[i]));
    r[i] = root_pos(b[i]);
    ey[i] = fma(-b[i], recip_seed(b[i]), 1.0);
    const double s = rsqrt_seed(b[i]);
    es[i] = fma(-(b[i] * s), s, 1.0);
}
__global__ void kf(long n, const float* x, float* q, float* r) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    q[i] = recip_f(x[i]);
    r[i] = root_f(x[i]);
}
extern "C" int runf(long n, const float* x, float* out) {
    float *dx, *d;
    const size_t bytes = n * sizeof(float);
    if (cudaMalloc(&dx, bytes) || cudaMalloc(&d, 2 * bytes)) return 1;
    cudaMemcpy(dx, x, bytes, cudaMemcpyHostToDevice);
    kf<<<(unsigned)((n + 255) / 256), 256>>>(n, dx, d, d + n);
    const int rc = cudaMemcpy(out, d, 2 * bytes, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(dx), cudaFree(d);
    return rc;
}
extern "C" int run(long n, const double* a, const double* b, double* out) {
    double *da, *db, *d;
    const size_t bytes = n * sizeof(double);
    if (cudaMalloc(&da, bytes) || cudaMalloc(&db, bytes) || cudaMalloc(&d, 4 * bytes)) return 1;
    cudaMemcpy(da, a, bytes, cudaMemcpyHostToDevice);
    cudaMemcpy(db, b, bytes, cudaMemcpyHostToDevice);
    k<<<(unsigned)((n + 255) / 256), 256>>>(n, da, db, d, d + n, d + 2 * n, d + 3 * n);
    const int rc = cudaMemcpy(out, d, 4 * bytes, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(da), cudaFree(db), cudaFree(d);
    return rc;
}
""" % HEADER


def hard_quotients(count, rng):
    """(a, b) with a/b within a few units of 2^-53/b of a rounding midpoint"""
    out = []
    while len(out) < count:
        b = rng.choice([rng.randrange(2 ** 52, 2 ** 53), 2 ** 53 - rng.randrange(1, 2 ** 12),
                        2 ** 52 + rng.randrange(1, 2 ** 12)]) | 1
        n = rng.choice([-3, -1, 1, 3])
        for bits in (53, 54):  # quotient in [1, 2), in [1/2, 1)
            m = 2 ** bits
            s = (-n * pow(b, -1, m)) % m
            s = s + 2 ** 53 if bits == 53 else s
            if not 2 ** 53 < s < 2 ** 54:
                continue
            a = (n + s * b) >> bits
            if 2 ** 52 <= a < 2 ** 53 and (n + s * b) % m == 0:
                out.append((float(a), float(b)))
    return out


def hard_roots():
    """x whose root is nearest to a midpoint: 4x - m^2 = N for small N (7 mod 8), m odd of 54 bits"""
    out = []
    for n in (-1, 7, -9, 15, -17, 23, -25, 31):
        roots = [1]
        for k in range(3, 56):  # square roots of -n modulo 2^k, one bit at a time
            roots = [r + d for r in set(roots) for d in (0, 1 << (k - 1), 1 << (k - 2)) if (r + d) ** 2 % (1 << k) == -n % (1 << k)]
            roots = list({r % (1 << k) for r in roots})[:64]
        for r in roots:
            for m in (r, r + 2 ** 54, r + 2 ** 55, (2 ** 54 - r) % 2 ** 54):
                if not 2 ** 53 < m < 2 ** 54 or (m * m + n) % 4:
                    continue
                x = (m * m + n) // 4
                if int(float(x)) == x:
                    out.append(float(x))
    assert len(out) >= 4
    return out


def special():
    """the significands whose rounding hangs on the seed (N = -1 for roots, the
    divisor with every bit set) and their neighbours, over the exponents"""
    return [math.ldexp(m, e) for e in range(-250, 250)
            for m in (2.0 ** 53 - 1, 2.0 ** 52 + 1, 2.0 ** 53 - 3, 2.0 ** 53 - 5, 2.0 ** 52 + 3)]


def operands(n, seeds_fixed):
    rng, r = random.Random(7), np.random.default_rng(7)
    a = r.standard_normal(n) * 2.0 ** r.integers(-300, 300, n)
    b = (1.0 + r.random(n)) * 2.0 ** r.integers(-300, 300, n)
    b[: n // 4] = 1.0 - r.integers(3, 64, n // 4) * 2.0 ** -53  # just below a power of two
    a[n // 4: n // 2] = b[n // 4: n // 2] * (1.0 + r.integers(-8, 8, n // 4) * 2.0 ** -52)
    h = np.array(hard_quotients(4000, rng))
    x = np.array(hard_roots())
    small = np.array([1.0, 2.0, 3.0, 5.0, 0.1, 1.0 / 3.0])
    a = np.concatenate([a, h[:, 0], -h[:, 0], np.ones_like(x), np.repeat(small, 6)])
    b = np.concatenate([b, h[:, 1], h[:, 1], x, np.tile(small, 6)])
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    if not seeds_fixed:
        # for any allowed seed every quotient is right, and every root but those at N = -1
        f = np.frexp(b)[0]
        keep = (f != 1.0 - 2.0 ** -53) & (f != 0.5 + 2.0 ** -53)
        return a, b, keep
    x = np.array(special())
    a = np.concatenate([a] + [np.full_like(x, v) for v in (1.0, 3.0, -1.0)] + [np.roll(x, 1)])
    return a, np.concatenate([b, x, x, x, x]), None


def _dp(x):
    return x.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def _same(x, y):
    return np.array_equal(x.view(np.int64), y.view(np.int64))


def test_quotients_and_roots_cpu(tmp_path):
    src, so = tmp_path / "r.cpp", tmp_path / "r.so"
    src.write_text(CPU_SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-x", "c++", "-o", str(so),
                    str(src)], check=True)
    lib = ctypes.CDLL(str(so))
    a, b, keep = operands(200_000, False)
    for err in (-SEED_ERR, 0.0, SEED_ERR / 3, SEED_ERR):
        e = np.full_like(a, err)
        q, r = np.empty_like(a), np.empty_like(a)
        lib.run(ctypes.c_long(len(a)), _dp(a), _dp(b), _dp(e), _dp(q), _dp(r))
        assert _same(q, a / b), err
        assert _same(r[keep], np.sqrt(b)[keep]), err


@pytest.fixture(scope="module")
def gpu_lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("round")
    src, so = d / "r.cu", d / "r.so"
    src.write_text(GPU_SRC)
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--fmad=false",
                    "-shared", "-Xcompiler", "-fPIC", "-o", str(so), str(src)], check=True)
    return ctypes.CDLL(str(so))


@pytest.mark.gpu
@pytest.mark.parametrize("exponent", [-100, -61, -38, -1, 0, 1, 44, 60, 99])
def test_fp32_reciprocals_and_roots_gpu(gpu_lib, exponent):
    """every significand at one exponent (with its neighbour: both parities)"""
    x = (np.arange(2 ** 23, dtype=np.uint32) + np.uint32((exponent + 127) << 23)).view(np.float32)
    out = np.empty((2, len(x)), dtype=np.float32)
    fp = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_float))  # noqa: E731
    assert gpu_lib.runf(ctypes.c_long(len(x)), fp(x), fp(out)) == 0
    assert np.array_equal(out[0].view(np.int32), (np.float32(1.0) / x).view(np.int32))
    assert np.array_equal(out[1].view(np.int32), np.sqrt(x).view(np.int32))


@pytest.mark.gpu
def test_quotients_and_roots_gpu(gpu_lib):
    lib = gpu_lib
    a, b, _ = operands(4_000_000, True)
    a = np.concatenate([a, [0.0, -0.0, 0.0, -0.0]])  # zeros keep their sign
    b = np.concatenate([b, [1.0, 3.0, 0.7, 2.0 ** -200]])
    out = np.empty((4, len(a)))
    assert lib.run(ctypes.c_long(len(a)), _dp(a), _dp(b), _dp(out)) == 0
    assert _same(out[0], a / b)
    assert _same(out[1], np.sqrt(b))
    assert np.abs(out[2]).max() <= SEED_ERR
    assert np.abs(out[3]).max() <= 2 * SEED_ERR
