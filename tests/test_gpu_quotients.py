"""The quotients that share a reciprocal (md_device.cuh) against CUDA's IEEE divisions, compiled
from that header: every FP32 significand and, in FP64, divisors whose reciprocals are the
hardest to round (all ones left to the division, as low_ones() has it), random ones and the edges
of divides_fast(); and the pair forces at squared separations whose significand is all ones,
against the oracle."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle as O
from conftest import ROOT

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "%s"
using namespace mdb;

// the reciprocal, and dividends 1, 3 and a random one, for every significand at exponent e
__global__ void f32(int e, unsigned seed, unsigned long long* bad) {
    const unsigned s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= 1u << 23) return;
    const float b = __uint_as_float(unsigned(127 + e) << 23 | s), y = reciprocal(b);
    if (y != __frcp_rn(b)) atomicAdd(bad, 1ull);
    const float a[3] = {1.0f, 3.0f, __uint_as_float(127u << 23 | ((s * 2654435761u ^ seed) >> 9))};
    for (int k = 0; k < 3; ++k)
        if (quotient(a[k], b, y) != __fdiv_rn(a[k], b)) atomicAdd(bad, 1ull);
}

__global__ void f64(int n, const double* a, const double* b, unsigned long long* bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double q = divides_fast(b[i]) && !low_ones(b[i]) ? quotient(a[i], b[i], reciprocal(b[i]))
                                                           : __ddiv_rn(a[i], b[i]);
    if (q != __ddiv_rn(a[i], b[i])) atomicAdd(bad, 1ull);
}

extern "C" long long run_f32(int e, unsigned seed) {
    unsigned long long *d, h = 0;
    cudaMalloc(&d, 8);
    cudaMemset(d, 0, 8);
    f32<<<(1 << 23) / 256, 256>>>(e, seed, d);
    if (cudaMemcpy(&h, d, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    cudaFree(d);
    return (long long)h;
}

extern "C" long long run_f64(int n, const double* a, const double* b) {
    double* in;
    unsigned long long *d, h = 0;
    cudaMalloc(&in, 16ull * n);
    cudaMalloc(&d, 8);
    cudaMemset(d, 0, 8);
    cudaMemcpy(in, a, 8ull * n, cudaMemcpyHostToDevice);
    cudaMemcpy(in + n, b, 8ull * n, cudaMemcpyHostToDevice);
    f64<<<(n + 255) / 256, 256>>>(n, in, in + n, d);
    if (cudaMemcpy(&h, d, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    cudaFree(in);
    cudaFree(d);
    return (long long)h;
}
"""


@pytest.fixture(scope="module")
def quotients(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    d = tmp_path_factory.mktemp("quotients")
    src, lib = d / "q.cu", d / "q.so"
    src.write_text(SOURCE % os.path.join(ROOT, "moleculardynamics_b200", "csrc", "md_device.cuh"))
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-shared",
                    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", str(src), "-o", str(lib)], check=True)
    q = ctypes.CDLL(str(lib))
    q.run_f32.restype = q.run_f64.restype = ctypes.c_longlong

    def f64(a, b):
        a, b = (np.ascontiguousarray(np.broadcast_to(x, np.broadcast(a, b).shape).ravel(), dtype=np.float64)
                for x in (a, b))
        ptr = [ctypes.c_void_p(x.ctypes.data) for x in (a, b)]
        return q.run_f64(len(a), *ptr)
    return q.run_f32, f64


@pytest.mark.parametrize("exponent", [-59, -1, 0, 1, 30])
def test_every_fp32_significand(md, quotients, exponent):
    assert quotients[0](exponent, 12345) == 0


def test_fp64_divisors_just_below_a_power_of_two(md, quotients):
    """1 / (1 - x 2^-53) for small odd x lies just above the midpoint of two doubles."""
    x = np.arange(1, 4096, 2) * 2.0 ** -53
    for a in (1.0, 2.0, 3.0, 0.1, 24.0 * 7.0):
        for e in (-99, -1, 0, 1, 2, 3, 398):
            assert quotients[1](a, (1.0 - x) * 2.0 ** e) == 0


def test_fp64_random_and_edges(md, quotients):
    rng = np.random.default_rng(7)
    a, b = rng.uniform(1.0, 2.0, (2, 1 << 21)) * 2.0 ** rng.integers(-60, 60, (2, 1 << 21))
    assert quotients[1](a, b) == 0
    lo, hi = 2.0 ** -100, 2.0 ** 400
    b = np.array([lo, np.nextafter(lo, 0), np.nextafter(lo, 1), hi, np.nextafter(hi, 0), 5e-324,
                  1.7e308, 1e-310])
    assert quotients[1](rng.uniform(1.0, 2.0, (64, 1)), b) == 0


@pytest.mark.parametrize("tiles", [False, True])
@pytest.mark.parametrize("r2", [2.0 - 2.0 ** -52, 4.0 - 2.0 ** -51, 1.0 - 2.0 ** -53])
def test_pairs_at_all_ones(md, r2, tiles):
    """A pair whose squared separation, as the reference rounds it, has every significand bit
    set (dividend sigma^2 = 1): forces, energy and virial are the oracle's bit for bit."""
    rng = np.random.default_rng(11)
    while True:  # a displacement with that r^2
        d = np.append(rng.uniform(0.2, 0.4, 2) * np.sqrt(r2), 0.0)
        d[2] = np.sqrt(r2 - d[0] * d[0] - d[1] * d[1])
        if (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2] == r2:
            break
    box = np.array([12.0, 12.0, 12.0])
    pos = np.stack([np.zeros(3), d])
    s = md.System.from_arrays(pos, box, mass=np.ones(2))
    md.VelocityVerlet(0.001).step(s, lambda sys: None)  # wrapped: what tiles need
    v = md.VerletList(box, 2.5, 0.3)
    v.build(s)
    v.set_halo(tiles)
    e, w = md.LennardJones(1.0, 1.0, 2.5).compute_forces(s, v)
    f_ref, e_ref, w_ref = O.lj_compute(pos, box, rc=2.5, trunc=0)
    assert np.array_equal(s.forces, f_ref) and e == e_ref and w == w_ref
