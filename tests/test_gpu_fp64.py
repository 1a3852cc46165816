"""The sweeps' FP64 square root and division by a known constant (fp64.cuh)
against the IEEE ones, bit for bit: arguments whose result lies next to the
middle of two numbers, built from their congruences, next to powers of two, at
the ends of the root's range, and random ones.  And the tile schedule's FP64
fields against the slab schedule's, which takes sqrt()."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from test_gpu_tiles import SLABS, TILES, _cells, _solve, _src

pytestmark = pytest.mark.gpu

CODE = r"""
#include "fp64.cuh"
__global__ void k(const double *a, const double *c, long long n, int random, unsigned long long *bad)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        double x = 0.0, d = 0.0;
        if (random) {
            unsigned long long z = (i + 1) * 0x9e3779b97f4a7c15ull, v[2];
            for (int j = 0; j < 2; ++j) {
                z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
                z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
                z ^= z >> 31;
                v[j] = (z >> 12) | (unsigned long long)(1023 - 64 + (z & 127)) << 52;
            }
            x = __longlong_as_double(v[0]);
            d = __longlong_as_double(v[1]);
        } else {
            x = a[i];
            if (c) d = c[i];
        }
        const double r = sqrt(x), s = fk64::sqrt64(x);
        if ((random || !c) && fk64::sqrt64_ok(x) && !(r == s || (r != r && s != s))) atomicAdd(bad, 1ull);
        if ((random || c) && fk64::div64(x, d, 1.0 / d) != x / d) atomicAdd(bad + 1, 1ull);
    }
}
extern "C" int check(const double *a, const double *c, long long n, int random, unsigned long long *bad)
{
    k<<<1184, 256>>>(a, c, n, random, bad);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def check(fk, tmp_path_factory):
    import torch
    d = tmp_path_factory.mktemp("fp64")
    csrc = os.path.join(os.path.dirname(os.path.dirname(fk.LIB_PATH)), "csrc")
    (d / "k.cu").write_text(CODE)
    nvcc = os.path.join(os.environ.get("CUDA", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-fmad=false", "-shared", "-Xcompiler", "-fPIC",
                    "-I", csrc, str(d / "k.cu"), "-o", str(d / "k.so")], check=True, timeout=300)
    lib = ctypes.CDLL(str(d / "k.so"))

    def run(x, c=None, n=0):
        bad = torch.zeros(2, dtype=torch.int64, device="cuda")
        t = [torch.from_numpy(np.ascontiguousarray(v)).cuda() if v is not None else None for v in (x, c)]
        torch.cuda.synchronize()
        p = [ctypes.c_void_p(v.data_ptr() if v is not None else None) for v in t]
        e = lib.check(p[0], p[1], ctypes.c_longlong(n or len(x)), ctypes.c_int(x is None), ctypes.c_void_p(bad.data_ptr()))
        assert e == 0
        return bad.tolist()
    return run


def _hard_roots(most=40000):
    """x = X 2^k whose root is (M + D / (2 M) ...) / 2 with M odd: X 2^k - M^2 = D small."""
    out = []
    for k in (54, 55):
        for d in range(-most, most + 1):
            a = -d % (1 << k)
            if a % 8 != 1:
                continue
            m = 1
            for j in range(3, k):
                if (m * m - a) >> j & 1:
                    m += 1 << (j - 1)
            for r in (m, -m, m + (1 << (k - 1)), -m + (1 << (k - 1))):
                r %= 1 << k
                x, rest = divmod(r * r + d, 1 << k)
                assert rest == 0
                if 1 << 53 <= r < 1 << 54 and 1 << 52 <= x < 1 << 53:
                    out.append(float(x << (k - 54)))
    return np.array(out)


def test_root_equals_ieee(check):
    x = _hard_roots()
    assert len(x) > 10000
    for j in (-950, -500, -2, 0, 2, 300, 850):
        assert check(np.ldexp(x, j)) == [0, 0], j
    p = np.ldexp(1.0, np.arange(-920, 921))
    near = [p]
    lo = hi = p
    for _ in range(8):
        lo, hi = np.nextafter(lo, 0.0), np.nextafter(hi, np.inf)
        near += [lo, hi]
    ends = [np.nextafter(1e-280, 1.0), np.nextafter(1e280, 0.0), -1e-300, -1.0, -1e300]
    assert check(np.concatenate(near + [ends])) == [0, 0]


def test_division_equals_ieee(check):
    rng = np.random.default_rng(1)
    a, c = [], []
    for i in range(20000):
        d = [int(rng.integers(1 << 51, 1 << 52)) * 2 + 1, (1 << 53) - 1 - 2 * int(rng.integers(0, 500)),
             (1 << 52) + 1 + 2 * int(rng.integers(0, 500))][i % 3]
        for k in (53, 54):
            inv = pow(d, -1, 1 << k)
            for r in (-5, -3, -1, 1, 3, 5):      # M d - r = X 2^k: X 2^k / d next to M, odd
                m = inv * r % (1 << k)
                for m in (m, m + (1 << k)):
                    x = (m * d - r) >> k
                    if 1 << 53 <= m < 1 << 54 and 1 << 52 <= x < 1 << 53:
                        a.append(float(x))
                        c.append(float(d))
    assert len(a) > 20000
    assert check(np.array(a), np.array(c)) == [0, 0]
    assert check(np.ldexp(a, -30), np.ldexp(c, 12)) == [0, 0]


def test_random_arguments(check):
    assert check(None, n=1 << 30) == [0, 0]


@pytest.mark.parametrize("n", [(3, 3, 3), (23, 33, 25), (61, 20, 31), (41, 53, 47), (70, 60, 64)])
@pytest.mark.parametrize("where", ["inside", "corner", "end"])
def test_fp64_tiles_equal_slabs(fk, n, where):
    vel, src = _cells(n, sum(n) + 1), _src(n, where)
    for nsweep, eps in ((2, min(3.0, min(n) - 1)), (1, 0.0)):
        a = _solve(fk, n, vel, src, TILES, 8, nsweep, eps)
        assert np.array_equal(a, _solve(fk, n, vel, src, SLABS, 8, nsweep, eps)), (nsweep, eps)
