"""reciprocal and quotient of physics.cuh against the correctly rounded
division. A harness of its own (nvcc, a few seconds): the functions run inside
the flux and Newton kernels and have no entry point."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from uqcreator_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "physics.cuh"
__global__ void k( int n, const double* a, const double* d, double* r, double* q ) {
    for( int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x ) {
        r[i] = uqc::reciprocal( d[i] );
        q[i] = uqc::quotient( a[i], d[i] );
    }
}
extern "C" int division( int n, const double* a, const double* d, double* r, double* q ) {
    double* x = nullptr;
    const size_t b = size_t( n ) * sizeof( double );
    if( cudaMalloc( &x, 4 * b ) != cudaSuccess ) return 1;
    cudaMemcpy( x, a, b, cudaMemcpyHostToDevice );
    cudaMemcpy( x + n, d, b, cudaMemcpyHostToDevice );
    k<<<592, 256>>>( n, x, x + n, x + 2 * size_t( n ), x + 3 * size_t( n ) );
    cudaMemcpy( r, x + 2 * size_t( n ), b, cudaMemcpyDeviceToHost );
    cudaMemcpy( q, x + 3 * size_t( n ), b, cudaMemcpyDeviceToHost );
    return cudaFree( x ) != cudaSuccess;
}
"""


@pytest.fixture(scope="module")
def division(tmp_path_factory):
    d = tmp_path_factory.mktemp("division")
    (d / "division.cu").write_text(SOURCE)
    subprocess.run([build.NVCC, *build.ARCH, "-std=c++17", "-O3", "-Xcompiler", "-fPIC", "-shared", "-I" + str(build.CSRC),
                    "-I" + str(build.ROOT / "include"), str(d / "division.cu"), "-o", str(d / "division.so")], check=True)
    f = C.CDLL(str(d / "division.so")).division

    def run(a, d):
        p = [np.ascontiguousarray(x, dtype=np.float64) for x in (a, d)] + [np.empty(len(d)) for _ in range(2)]
        assert f(len(d), *(x.ctypes.data_as(C.POINTER(C.c_double)) for x in p)) == 0
        return p[2], p[3]

    return run


def _draw(seed, n, exponents):
    r = np.random.default_rng(seed)
    return r.choice([-1.0, 1.0], n) * np.ldexp(r.uniform(1, 2, n), r.integers(-exponents, exponents, n))


# the fluxes' and ansatz's divisors (densities, speeds, 1 + E), and the pivots' determinants
@pytest.mark.parametrize("exponents", [3, 200, 1000])
def test_within_an_ulp_of_division(division, exponents):
    """The estimate's error e (2^-20 at most) leaves e^3 < 2^-59 after the
    iteration, and the last operation rounds once: at most one unit in the last
    place, 2^-52 of the value, from the rounded quotient. A quotient whose
    residual stays normal likewise."""
    n = 1 << 22
    a, d = _draw(1, n, min(exponents, 200)), _draw(2, n, exponents)
    r, q = division(a, d)
    np.testing.assert_array_less(np.abs(r - 1.0 / d), 1.01 * 2.0 ** -52 * np.abs(1.0 / d))
    if exponents <= 200:
        np.testing.assert_array_less(np.abs(q - a / d), 1.01 * 2.0 ** -52 * np.abs(a / d))


def test_edges(division):
    """Exact for powers of two; zero and infinite divisors, which no finite state
    has, give NaN."""
    d = np.ldexp(1.0, np.arange(-900, 901))
    r, q = division(np.full(len(d), 3.0), d)
    np.testing.assert_array_equal(r, 1.0 / d)
    np.testing.assert_array_equal(q, 3.0 / d)
    r, q = division(np.ones(5), np.array([0.0, -0.0, np.inf, -np.inf, np.nan]))
    assert np.isnan(r).all() and np.isnan(q).all()
