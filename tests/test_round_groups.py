"""quot_group of cumc_round.cuh against the division operator over every range
of its operands, on the host and on the GPU: infinite, NaN and overflowing
numerators, quotients that leave the normal numbers, and divisors it hands on;
and what a stage reports when an energy overflows."""
import ctypes
import itertools
import math
import os
import subprocess

import numpy as np
import pytest

from cumpic_b200 import _native as N
from cumpic_b200 import problems as P

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cumpic_b200", "csrc",
                      "cumc_round.cuh")
CPU_SRC = """
#include "%s"
extern "C" void run(long n, const double* a, const double* b, double* q) {
    for (long i = 0; i + 3 <= n; i += 3) {
        const double num[3] = {a[i], a[i + 1], a[i + 2]};
        double r[3];
        cumc::quot_group(num, b[i], r);
        for (int m = 0; m < 3; ++m) q[i + m] = r[m];
    }
}
""" % HEADER
GPU_SRC = """
#include "%s"
#include <cuda_runtime.h>
__global__ void k(long n, const double* a, const double* b, double* q) {
    const long i = 3 * (blockIdx.x * (long)blockDim.x + threadIdx.x);
    if (i + 3 > n) return;
    const double num[3] = {a[i], a[i + 1], a[i + 2]};
    double r[3];
    cumc::quot_group(num, b[i], r);
    for (int m = 0; m < 3; ++m) q[i + m] = r[m];
}
extern "C" int run(long n, const double* a, const double* b, double* q) {
    double* d;
    const size_t bytes = n * sizeof(double);
    if (cudaMalloc(&d, 3 * bytes)) return 1;
    cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, bytes, cudaMemcpyHostToDevice);
    k<<<(unsigned)((n / 3 + 255) / 256), 256>>>(n, d, d + n, d + 2 * n);
    const int rc = cudaMemcpy(q, d + 2 * n, bytes, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(d);
    return rc;
}
""" % HEADER


def operands():
    """groups of three numerators by one divisor (b holds it three times)"""
    rng = np.random.default_rng(11)
    num = [0.0, 5e-324, 1e-310, 2.0 ** -1022, 2.0 ** -901, 2.0 ** -900, 2.0 ** -899, 2.0 ** -801, 2.0 ** -800, 1e-200,
           1.0, 2.0 ** 799, 2.0 ** 800, 1e300, 1.7e308, np.inf, np.nan]
    div = [s * m * 2.0 ** e for s in (1, -1) for m in (1.0, 1.5, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 4.0 / 3.0)
           for e in (-1000, -201, -200, -199, -10, 0, 10, 198, 199, 200, 1000)] + [0.0, np.inf, np.nan]
    groups = []
    for a, b in itertools.product(num, div):
        x = rng.choice(num, 2) * rng.choice([-1.0, 1.0], 2)
        groups.append((a, b, x[0], 1.0))
        groups.append((-a, b, 1.0, x[1]))
    # quotients halfway between two subnormal numbers: a/b = (odd) 2^-1075
    for e, k in itertools.product(range(-899, -880), (1, 3, 5, 7, 2 ** 20 + 1)):
        groups.append((math.ldexp(3.0 * k, e), math.ldexp(3.0, e + 1075), 1.0, 1.0))
    g = np.array(groups)
    a = np.ascontiguousarray(g[:, [0, 2, 3]].reshape(-1))
    return a, np.ascontiguousarray(np.repeat(g[:, 1], 3))


def check(run):
    a, b = operands()
    q = np.empty_like(a)
    assert not run(ctypes.c_long(len(a)), *(x.ctypes.data_as(ctypes.c_void_p) for x in (a, b, q)))
    with np.errstate(all="ignore"):
        want = a / b
    bad = ~((q.view(np.int64) == want.view(np.int64)) | (np.isnan(q) & np.isnan(want)))
    assert not bad.any(), (bad.sum(), [(x, y, u, v) for x, y, u, v in zip(a[bad], b[bad], q[bad], want[bad])][:5])


def test_quot_group_cpu(tmp_path):
    src, so = tmp_path / "g.cpp", tmp_path / "g.so"
    src.write_text(CPU_SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(so), str(src)],
                   check=True)
    run = ctypes.CDLL(str(so)).run
    run.restype = None
    check(run)


@pytest.mark.gpu
def test_quot_group_gpu(tmp_path):
    src, so = tmp_path / "g.cu", tmp_path / "g.so"
    src.write_text(GPU_SRC)
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--fmad=false",
                    "-shared", "-Xcompiler", "-fPIC", "-o", str(so), str(src)], check=True)
    check(ctypes.CDLL(str(so)).run)


@pytest.mark.gpu
@pytest.mark.parametrize("nx", [12, 13], ids=["pairs", "single_cells"])
def test_overflowing_energy_is_reported(nx):
    """A fluid at rest whose pressure alternates from row to row: the momenta
    stay zero by symmetry while the energy's rate times a huge dt is infinite.
    The pressure of the rows that gain energy is then infinite, and the step
    must report it."""
    from cumpic_b200.solver import CUMC3D
    p = P.orszag_tang(nx, ny=6, nz=4)
    p.prim[..., P.IVX:P.IVZ + 1] = 0.0
    p.prim[..., P.IBX:P.IBZ + 1] = 0.0
    p.prim[..., P.IRHO] = 1.0
    p.prim[..., P.ITAU] = 1e60 * (1.0 + 0.5 * (np.arange(12) % 2))[None, :, None]
    p.eps[...] = p.prim[..., P.ITAU] / (p.ggas - 1.0)
    g = CUMC3D(p)
    g.upload()
    g.initial_update()
    g.finddt()
    g.rungekutta(1e220)
    with pytest.raises(N.CumcError) as e:
        g.finddt()
    assert e.value.code == N.CUMC_ERR_NONFINITE
