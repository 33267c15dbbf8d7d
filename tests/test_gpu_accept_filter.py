"""The accept decision u < exp(-max(dS, 0)) is taken in binary32, m < -log u,
outside a band around equality and evaluated inside it (csrc/su3_exp.cuh
neg_log_unit, accept_log).  Here its two halves are compiled into a kernel of
their own, with and without fused multiply-adds as the engine's units are.

neg_log_unit against binary64 log over words spread over the exponent and at
the edges of its range: within 2e-5 (1.53e-5 for the 32 bits it takes of the
word, 3.3e-6 for the conversion and __logf), less than the 2.5e-5 of the band
minus the 7e-7 of m's rounding; NaN below 2^-16.  accept_log against the plain
decision with dS at, just inside and just outside the band, and at zeros,
infinities and NaN: equal everywhere.  Words are chosen by inverting the
stream's mixing function, so that the decision inside the band draws the same
word again."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GOLDEN = 0x9E3779B97F4A7C15
MASK = (1 << 64) - 1

SOURCE = r"""
#include "su3_exp.cuh"
using namespace ym;
__global__ void k_filter(const uint64_t *keys, const double *ds, long n, uint64_t *words, float *logu, int *fast,
                         int *plain) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t w = splitmix_at(keys[i], 1);     // hit 0's accept word
    words[i] = w;
    logu[i] = neg_log_unit(w);
    fast[i] = accept_log(ds[i], logu[i], keys[i], 0);
    plain[i] = unit_from(w) < exp(-fmax(ds[i], 0.0));
}
extern "C" int run(const uint64_t *keys, const double *ds, long n, uint64_t *words, float *logu, int *fast,
                   int *plain) {
    uint64_t *dk, *dw;
    double *dd;
    float *dl;
    int *df, *dp;
    if (n < 1 || cudaMalloc(&dk, n * 8) || cudaMalloc(&dd, n * 8) || cudaMalloc(&dw, n * 8) ||
        cudaMalloc(&dl, n * 4) || cudaMalloc(&df, n * 4) || cudaMalloc(&dp, n * 4))
        return 1;
    cudaMemcpy(dk, keys, n * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(dd, ds, n * 8, cudaMemcpyHostToDevice);
    k_filter<<<(unsigned)((n + 127) / 128), 128>>>(dk, dd, n, dw, dl, df, dp);
    if (cudaGetLastError()) return 2;
    cudaMemcpy(words, dw, n * 8, cudaMemcpyDeviceToHost);
    cudaMemcpy(logu, dl, n * 4, cudaMemcpyDeviceToHost);
    cudaMemcpy(fast, df, n * 4, cudaMemcpyDeviceToHost);
    cudaMemcpy(plain, dp, n * 4, cudaMemcpyDeviceToHost);
    const int err = cudaDeviceSynchronize();
    cudaFree(dk); cudaFree(dd); cudaFree(dw); cudaFree(dl); cudaFree(df); cudaFree(dp);
    return err;
}
"""


def _unshift(z, s):
    """x of z = x ^ (x >> s)."""
    x = z
    for _ in range(64 // s):
        x = z ^ (x >> np.uint64(s))
    return x


def _keys_of(words):
    """The keys whose second stream word each is (splitmix64's mixing inverted)."""
    with np.errstate(over="ignore"):
        z = _unshift(words, 31)
        z = _unshift(z * np.uint64(pow(0x94D049BB133111EB, -1, 1 << 64)), 27)
        z = _unshift(z * np.uint64(pow(0xBF58476D1CE4E5B9, -1, 1 << 64)), 30)
        return z - np.uint64(2 * GOLDEN & MASK)


def _words():
    rng = np.random.default_rng(4)
    spread = (2.0 ** rng.uniform(30.0, 64.0, 400000)).astype(np.float64)
    words = [np.minimum(spread, 2.0 ** 63).astype(np.uint64) |
             rng.integers(0, 2 ** 11, spread.size, dtype=np.uint64),
             rng.integers(0, 2 ** 64, 400000, dtype=np.uint64)]
    edges = []
    for hi in (0, 1, 2, 65534, 65535, 65536, 65537, 2 ** 24 - 1, 2 ** 24, 2 ** 24 + 1, 2 ** 31 - 1, 2 ** 31,
               2 ** 31 + 1, 2 ** 32 - 257, 2 ** 32 - 129, 2 ** 32 - 2, 2 ** 32 - 1):
        for lo in (0, 1, 2 ** 11, 2 ** 31, 2 ** 32 - 1):
            edges.append(hi << 32 | lo)
    words.append(np.array(edges, np.uint64))
    return np.concatenate(words)


@pytest.fixture(scope="module", params=["exact", "fused"])
def run(request, tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    where = tmp_path_factory.mktemp("filter")
    src, lib = str(where / "filter.cu"), str(where / "filter.so")
    with open(src, "w") as fh:
        fh.write(SOURCE)
    flags = ["-fmad=false"] if request.param == "exact" else []
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", *flags, "-shared",
                    "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "yang-mills_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"), src, "-o", lib, "-lcudart"], check=True)
    fn = C.CDLL(lib).run
    fn.argtypes = [C.c_void_p, C.c_void_p, C.c_long] + [C.c_void_p] * 4

    def call(words, ds):
        n = words.size
        keys, ds = _keys_of(words), np.ascontiguousarray(ds, np.float64)
        got, logu = np.zeros(n, np.uint64), np.zeros(n, np.float32)
        fast, plain = np.zeros(n, np.int32), np.zeros(n, np.int32)
        assert fn(keys.ctypes.data, ds.ctypes.data, n, got.ctypes.data, logu.ctypes.data, fast.ctypes.data,
                  plain.ctypes.data) == 0
        assert np.array_equal(got, words)
        return logu, fast, plain
    return call


def _minus_log(words):
    u = (words >> np.uint64(11)).astype(np.float64) * 2.0 ** -53
    with np.errstate(divide="ignore"):
        return -np.log(u)


def test_logarithm_within_its_bound(run):
    words = _words()
    logu, _, _ = run(words, np.zeros(words.size))
    small = (words >> np.uint64(32)) < 65536
    assert small.any() and np.isnan(logu[small]).all()
    err = np.abs(logu[~small].astype(np.float64) - _minus_log(words[~small]))
    assert err.max() <= 2.0e-5


def test_decisions_are_the_plain_ones(run):
    words = _words()
    m = _minus_log(words)
    m = np.where(np.isfinite(m), m, 40.0)
    band = 2.5e-5
    cases = [m * (1.0 + f) for f in (0.0, 2.0 ** -52, -2.0 ** -52, 1e-12, -1e-12)]
    cases += [m + f * band for f in (0.5, -0.5, 0.9, -0.9, 1.0, -1.0, 1.1, -1.1, 2.0, -2.0, 100.0, -100.0)]
    cases += [np.full(words.size, v) for v in (0.0, -0.0, -1.0, 5e-324, 1e300, np.inf, -np.inf, np.nan)]
    seen = set()
    for ds in cases:
        _, fast, plain = run(words, ds)
        assert np.array_equal(fast, plain)
        seen.update(np.unique(plain).tolist())
    assert seen == {0, 1}
