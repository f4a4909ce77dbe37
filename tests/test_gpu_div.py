"""The kernels' quotients by fixed divisors: the functions themselves, and where they must hold.

div_by and mg_div (cfd_common.cuh, cfd_step.cuh) are compiled into a small kernel and compared bit for
bit with the device's own division: over random operands, and for div_by also where a quotient by
reciprocal goes wrong unless it is looked after (zeros of either sign, infinite operands,
overflow). An O-grid whose Re or Pr is infinite divides by infinity next to its walls: its steps
must match the oracle's like any other case's.
"""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

from cfd_solver_b200.grid import ogrid

pytestmark = pytest.mark.gpu

CSRC = Path(__file__).resolve().parents[1] / "cfd_solver_b200" / "csrc"
SOURCE = r"""
#include "cfd_step.cuh"
using namespace cfd;
__global__ void k64(const double* n, const double* d, const double* y, double* q, double* ref, int m) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= m) return;
    q[e] = div_by(n[e], DivBy{d[e], y[e]});
    ref[e] = n[e] / d[e];
}
__global__ void k32(const float* n, const float* d, float* q, float* ref, int m) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= m) return;
    q[e] = mg_div(n[e], d[e], __frcp_rn(d[e]));
    ref[e] = n[e] / d[e];
}
template <class T>
static int on_device(int m, const T* const* in, int nin, T* q, T* ref, bool f64) {
    T* b[5] = {};
    const size_t bytes = sizeof(T) * (size_t)m;
    for (auto& p : b)
        if (cudaMalloc((void**)&p, bytes) != cudaSuccess) return 1;
    for (int k = 0; k < nin; k++) cudaMemcpy(b[k], in[k], bytes, cudaMemcpyHostToDevice);
    if (f64) k64<<<(m + 255) / 256, 256>>>((double*)b[0], (double*)b[1], (double*)b[2], (double*)b[3], (double*)b[4], m);
    else k32<<<(m + 255) / 256, 256>>>((float*)b[0], (float*)b[1], (float*)b[3], (float*)b[4], m);
    cudaMemcpy(q, b[3], bytes, cudaMemcpyDeviceToHost);
    cudaMemcpy(ref, b[4], bytes, cudaMemcpyDeviceToHost);
    for (auto p : b) cudaFree(p);
    return cudaGetLastError() != cudaSuccess;
}
extern "C" int div64(int m, const double* n, const double* d, const double* y, double* q, double* ref) {
    const double* in[3] = {n, d, y};
    return on_device<double>(m, in, 3, q, ref, true);
}
extern "C" int div32(int m, const float* n, const float* d, float* q, float* ref) {
    const float* in[2] = {n, d};
    return on_device<float>(m, in, 2, q, ref, false);
}
"""


@pytest.fixture(scope="module")
def quotients(tmp_path_factory):
    t = tmp_path_factory.mktemp("div")
    (t / "div.cu").write_text(SOURCE)
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-I", str(CSRC), "-o", str(t / "div.so"), str(t / "div.cu")], check=True)
    return ctypes.CDLL(str(t / "div.so"))


def _ptr(*arrays):
    return [a.ctypes.data_as(ctypes.c_void_p) for a in arrays]


def _div64(lib, n, d):
    n, d = np.broadcast_arrays(n, d)
    n, d = np.ascontiguousarray(n, np.float64), np.ascontiguousarray(d, np.float64)
    with np.errstate(all="ignore"):
        y = np.minimum(1.0 / d, np.finfo(np.float64).max)  # as the host forms it
    q, ref = np.empty_like(n), np.empty_like(n)
    assert lib.div64(n.size, *_ptr(n, d, y, q, ref)) == 0
    return q, ref


def _same(q, ref):
    both = np.isnan(q) & np.isnan(ref)
    assert np.array_equal(q[~both].view(f"i{q.itemsize}"), ref[~both].view(f"i{q.itemsize}"))


def _random(rng, m, bits, emax, dtype):
    """Random significands (some at the edges) with exponents in [-emax, emax]."""
    s = 1.0 + rng.integers(0, 1 << bits, m) * 2.0 ** -bits
    edge = rng.integers(0, 8, m)
    s = np.where(edge == 0, 1.0, np.where(edge == 1, 2.0 - 2.0 ** -bits, s))
    return (s * 2.0 ** rng.integers(-emax, emax + 1, m) * rng.choice([-1.0, 1.0], m)).astype(dtype)


def test_div_by_rounds_like_the_division(quotients):
    rng = np.random.default_rng(7)
    # exponents to +-480: quotients and their residuals stay normal
    n, d = _random(rng, 1 << 21, 52, 480, np.float64), np.abs(_random(rng, 1 << 21, 52, 480, np.float64))
    _same(*_div64(quotients, n, d))


@pytest.mark.parametrize("d", [0.25, 1.0 / 3.0, 71.0, 1e-8, 1e200, np.inf])
def test_div_by_at_the_ends(quotients, d):
    big = np.finfo(np.float64).max
    n = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1.0, -1.0, big, -big, 0.5 * big, 1e-5, 3.0], np.float64)
    _same(*_div64(quotients, n, d))


def test_zero_over_a_divisor_whose_reciprocal_overflows(quotients):
    q, ref = _div64(quotients, np.array([0.0, -0.0]), 1e-309)
    _same(q, ref)


def test_mg_div_rounds_like_the_division(quotients):
    rng = np.random.default_rng(8)
    # quotients of 2^-96 .. 2^96, inside the stated 1e-30 .. 1e38, of operands whose residuals are normal
    n, d = _random(rng, 1 << 21, 23, 48, np.float32), _random(rng, 1 << 21, 23, 48, np.float32)
    q, ref = np.empty_like(n), np.empty_like(n)
    assert quotients.div32(n.size, *_ptr(n, d, q, ref)) == 0
    _same(q, ref)


@pytest.mark.parametrize("host", [False, True])
@pytest.mark.parametrize("phys", [dict(Re=np.inf), dict(Re=100.0, Pr=np.inf), dict(Re=1e200, Pr=1e200)])
def test_infinite_re_or_pr_matches_the_oracle(phys, host):
    """Tight inner tolerances on both sides, so the bar is that of the step tests (1e-8)."""
    from cfd_solver_b200.solver import Batch, case_params
    from oracle import oracle
    g = ogrid(33, 25, skew=0.1)
    phys = dict(dict(Ri=1.0, dt=1e-3), **phys)
    with Batch([g], [case_params(g, **phys, tol_mom=1e-13, atol_mom=1e-13, maxit_mom=400, tol_p=1e-12, atol_p=1e-12,
                                 maxit_p=400)]) as b:
        b.profile(host)
        b.step(3)
        st = b.stats(0)
        gpu = {k: b.plane(0, k) for k in ("u", "v", "T", "p")}
    assert st["status"] == 0
    ref = oracle.OracleCase(g, **phys, tol_gs=1e-13, maxit_gs=400, tol_sip=1e-12, maxit_sip=4000)
    ref.step(3)
    for k, a in gpu.items():
        r = ref.field(k)
        assert np.linalg.norm(a - r) <= 1e-8 * np.linalg.norm(r), k
