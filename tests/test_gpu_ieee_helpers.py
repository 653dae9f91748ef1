"""Roots, reciprocals, quotients and powers of the FP64 gathers against the IEEE operations
they stand for, bit for bit: a fluid at rest cancels pressure terms to a 1e-9 th of themselves,
so they have to round as the reference's operations do.

A small unit that includes the gathers' header is built and run on random operands of the
stated ranges and on edges: the ends of the ranges, mantissas of all ones, of all zeros and
next to them, in every binade.  numpy's sqrt and division are correctly rounded; powers are
compared with the restatement of Julia's, on the device.
"""
import ctypes as C
import importlib
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

UNIT = r"""
#include "sph_coop.cuh"
using namespace sph;
__global__ void k_helpers(int n, const double* a, const double* b, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double inv;
    out[i] = sqrt_rn(fabs(a[i]), inv);
    out[n + i] = inv;
    out[2 * n + i] = rcp_rn(a[i]);
    out[3 * n + i] = div_rn(a[i], b[i], 1.0 / b[i]);
}
__global__ void k_powers(int n, const double* a, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x = a[i];
    const double fixed[4] = {powi_fixed<4>(x), powi_fixed<5>(x), powi_fixed<6>(x), powi_fixed<7>(x)};
    for (int k = 0; k < 4; ++k) {
        out[2 * k * n + i] = fixed[k];
        out[(2 * k + 1) * n + i] = jl_powi(x, 4 + k);
    }
}
__global__ void k_ranges(int n, const double* a, int* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (sqrt_rn_range(a[i]) ? 1 : 0) | (rcp_rn_range(a[i]) ? 2 : 0);
}
// r, W, dW/dr and grad W of a pair: the gathers' (out[0..5]), the plain restatement (out[6..11])
template <int KK>
__global__ void k_pairs(int n, const double* a, SceneDev S, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double rv[3] = {a[3 * i], a[3 * i + 1], a[3 * i + 2]};
    const double d2 = norm_sq<3>(rv);
    double r, W, dW, g[3];
    pair_kernel<3, KK>(rv, d2, S, r, W, dW, g);
    const double got[6] = {r, W, dW, g[0], g[1], g[2]};
    r = sqrt(d2);
    kernel_wdw<KK>(r, S, W, dW);
    grad_vec<3>(dW, r, rv, g);
    const double want[6] = {r, W, dW, g[0], g[1], g[2]};
    for (int k = 0; k < 6; ++k) {
        out[k * n + i] = got[k];
        out[(6 + k) * n + i] = want[k];
    }
}
__global__ void k_widen(int n, const float* a, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = widen(a[i]);
}
static int run(int n, const double* a, const double* b, void* out, size_t bytes, int which) {
    double *da = nullptr, *db = nullptr;
    void* dout = nullptr;
    cudaMalloc((void**)&da, n * 8);
    cudaMalloc((void**)&db, n * 8);
    cudaMalloc(&dout, bytes);
    if (!da || !db || !dout) return -1;
    cudaMemcpy(da, a, n * 8, cudaMemcpyHostToDevice);
    if (b) cudaMemcpy(db, b, n * 8, cudaMemcpyHostToDevice);
    const int grid = (n + 255) / 256;
    if (which == 0) k_helpers<<<grid, 256>>>(n, da, db, (double*)dout);
    if (which == 1) k_powers<<<grid, 256>>>(n, da, (double*)dout);
    if (which == 2) k_ranges<<<grid, 256>>>(n, da, (int*)dout);
    cudaMemcpy(out, dout, bytes, cudaMemcpyDeviceToHost);
    if (which == 7) {  // a holds 2 n floats
        k_widen<<<(2 * n + 255) / 256, 256>>>(2 * n, (const float*)da, (double*)dout);
        cudaMemcpy(out, dout, bytes, cudaMemcpyDeviceToHost);
    } else if (which >= 3) {
        SceneDev S{};
        S.h = 0.037;
        S.inv_h = 1.0 / S.h;
        S.kw_a = 123.456;
        S.kg_a = -78.9 / S.h;
        auto kernel = which == 3   ? k_pairs<SPH_KERNEL_CUBIC_SPLINE>
                      : which == 4 ? k_pairs<SPH_KERNEL_GAUSSIAN>
                      : which == 5 ? k_pairs<SPH_KERNEL_WENDLAND_C2>
                                   : k_pairs<SPH_KERNEL_WENDLAND_C4>;
        kernel<<<grid / 3 + 1, 256>>>(n / 3, da, S, (double*)dout);
        cudaMemcpy(out, dout, bytes, cudaMemcpyDeviceToHost);
    }
    cudaFree(da);
    cudaFree(db);
    cudaFree(dout);
    return (int)cudaGetLastError();
}
extern "C" int helpers(int n, const double* a, const double* b, double* out) { return run(n, a, b, out, 32ull * n, 0); }
extern "C" int powers(int n, const double* a, double* out) { return run(n, a, nullptr, out, 64ull * n, 1); }
extern "C" int ranges(int n, const double* a, int* out) { return run(n, a, nullptr, out, 4ull * n, 2); }

extern "C" int pairs(int n, const double* a, double* out, int kernel) {
    return run(3 * n, a, nullptr, out, 96ull * n, 3 + kernel);
}
extern "C" int widened(int n, const float* a, double* out) {  // n even
    return run(n / 2, (const double*)a, nullptr, out, 8ull * n, 7);
}
"""

N = 1 << 22


@pytest.fixture(scope="module")
def unit(pkg, tmp_path_factory):
    recipe = importlib.import_module(pkg.__name__ + ".build")
    tmp = tmp_path_factory.mktemp("helpers")
    (tmp / "unit.cu").write_text(UNIT)
    so = tmp / "libunit.so"
    subprocess.run([recipe.nvcc(), *recipe.ARCH, *recipe.COMMON, *recipe.UNIT_FLAGS["sph_fp64.cu"], "-I",
                    str(recipe.CSRC), "-shared", str(tmp / "unit.cu"), "-o", str(so)], check=True, capture_output=True)
    return C.CDLL(str(so))


def ptr(a):
    return C.c_void_p(a.ctypes.data)


def with_exponents(rng, mantissa, lo, hi):
    e = rng.integers(lo, hi, len(mantissa))
    return np.ldexp(1.0 + mantissa.astype(np.float64) / 2.0**52, e)


def operands(rng, lo, hi):
    """Random mantissas, and 0, 1, 2^52 - 1, ... and their neighbours, exponents in [lo, hi)."""
    few = np.concatenate([np.arange(64), 2**52 - 1 - np.arange(64), 2**51 - 32 + np.arange(64)])
    edge = np.repeat(few, hi - lo)
    e = np.tile(np.arange(lo, hi), len(few))
    edges = np.ldexp(1.0 + edge.astype(np.float64) / 2.0**52, e)
    return np.concatenate([edges, with_exponents(rng, rng.integers(0, 2**52, N), lo, hi)])


def helpers(unit, a, b):
    out = np.empty((4, len(a)))
    assert unit.helpers(len(a), ptr(a), ptr(b), ptr(out)) == 0
    return out


def same(got, want, *of):
    bad = np.flatnonzero(got.view(np.int64) != want.view(np.int64))
    assert not len(bad), (len(bad), *(o[bad[0]].hex() for o in of), got[bad[0]].hex(), want[bad[0]].hex())


def test_roots_and_their_reciprocals(unit):
    rng = np.random.default_rng(1)
    a = operands(rng, -900, 900)
    # squares of mantissas of all ones and next to them: the root's reciprocal at its worst place
    r = np.ldexp(2.0 - np.arange(1, 65) * 2.0**-52, 0)
    sq = np.concatenate([np.ldexp(r * r * (1.0 + k * 2.0**-52), e) for e in range(-450, 450, 7) for k in (-1, 0, 1)])
    a = np.concatenate([a, sq])
    out = helpers(unit, a, np.ones_like(a))
    root = np.sqrt(a)
    same(out[0], root, a)
    same(out[1], 1.0 / root, a)


def test_reciprocals(unit):
    rng = np.random.default_rng(2)
    a = operands(rng, -900, 900)
    a *= np.where(rng.random(len(a)) < 0.5, -1.0, 1.0)
    same(helpers(unit, a, np.ones_like(a))[2], 1.0 / a, a)


def test_quotients(unit):
    rng = np.random.default_rng(3)
    b = operands(rng, -300, 300)
    a = operands(rng, -300, 300)[rng.permutation(len(b))]
    a *= np.where(rng.random(len(a)) < 0.5, -1.0, 1.0)
    same(helpers(unit, a, b)[3], a / b, a, b)


def test_powers(unit):
    rng = np.random.default_rng(4)
    x = operands(rng, -100, 100)
    out = np.empty((4, 2, len(x)))
    assert unit.powers(len(x), ptr(x), ptr(out)) == 0
    for k in range(4):
        same(out[k, 0], out[k, 1], x)


@pytest.mark.parametrize("kernel", range(4), ids=["CubicSpline", "Gaussian", "WendlandC2", "WendlandC4"])
def test_pairs(unit, kernel):
    # vectors of every direction up to 3.1 h, some along an axis, some coincident or nearly so
    rng = np.random.default_rng(5)
    v = rng.normal(size=(1 << 20, 3))
    v *= (rng.uniform(0.0, 3.1, len(v)) * 0.037 / np.linalg.norm(v, axis=1))[:, None]
    v[: 1 << 16, 1:] = 0.0
    v[-4096:] *= 10.0 ** -rng.uniform(0, 320, 4096)[:, None]
    v[-16:] = 0.0
    v = np.ascontiguousarray(v)
    out = np.empty((2, 6, len(v)))
    assert unit.pairs(len(v), ptr(v), ptr(out), kernel) == 0
    for k in range(6):
        same(out[0, k] + 0.0, out[1, k] + 0.0, v[:, 0], v[:, 1], v[:, 2])  # a zero of either sign


def test_widened_floats(unit):
    # every exponent with mantissas at both ends and in the middle, both signs, subnormals,
    # zeros, infinities, and random bits
    mantissa = np.concatenate([np.arange(256), 2**23 - 1 - np.arange(256), 2**22 - 128 + np.arange(256)])
    bits = (np.arange(512, dtype=np.int64)[:, None] << 23 | mantissa).ravel().astype(np.uint32)
    bits = np.concatenate([bits, np.random.default_rng(6).integers(0, 2**32, N, dtype=np.uint32)])
    x = bits.view(np.float32)
    out = np.empty(len(x))
    assert len(x) % 2 == 0 and unit.widened(len(x), ptr(x), ptr(out)) == 0
    nan = np.isnan(x)
    assert np.all(np.isnan(out[nan]))
    same(out[~nan], x[~nan].astype(np.float64), x[~nan].astype(np.float64))


def test_ranges_take_only_what_the_helpers_are_exact_on(unit):
    x = np.array([0.0, 5e-324, 2.0**-1022, 2.0**-901, 2.0**-900, 2.0**-301, 2.0**-300, 1.0, 2.0**299, 2.0**300, 2.0**301,
                  2.0**899, 2.0**901, 1.7e308, np.inf, np.nan, -1.0, -2.0**301, -0.0, -np.inf, np.float64("-nan")])
    got = np.empty(len(x), np.int32)
    assert unit.ranges(len(x), ptr(x), ptr(got)) == 0
    for v, g in zip(x, got):
        if g & 1:
            assert 2.0**-900 <= v <= 2.0**900, v
        if g & 2:
            assert 2.0**-300 <= abs(v) < 2.0**301, v
    ordinary = (x >= 2.0**-300) & (x <= 2.0**299)
    assert np.all(got[ordinary] == 3)
