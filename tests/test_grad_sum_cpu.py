"""The sum of the weight gradients' partial sums (fr_sum.cuh, compiled for the host) against
the exact sum: no further off than FP64 sums of the terms c, c + 8, ... combined pairwise,
rounded once to FP32. Each of those adds rounds by at most 2^-53 of a partial sum, which is
at most sum |x|, and there are at most ceil(n / 8) + 2 one after another."""

import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FLT_MAX = float(np.finfo(np.float32).max)
INF = math.inf

SOURCE = '#include "fr_sum.cuh"\nextern "C" float sum_terms(const float* v, int n) { return frx::sum_terms(v, 1, n); }\n'


@pytest.fixture(scope="module")
def sum_terms(tmp_path_factory):
    d = tmp_path_factory.mktemp("sum")
    (d / "sum.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    f"-I{ROOT}/forkerrenderer_gb300/csrc", str(d / "sum.cpp"), "-o", str(d / "sum.so")], check=True)
    f = C.CDLL(str(d / "sum.so")).sum_terms
    f.restype, f.argtypes = C.c_float, [C.c_void_p, C.c_int]
    return lambda v: f(np.ascontiguousarray(v, np.float32).ctypes.data, len(v))


def _check(sum_terms, v):
    v = np.asarray(v, np.float32)
    got, wide = sum_terms(v), v.astype(np.float64)
    if not np.isfinite(v).all():
        with np.errstate(invalid="ignore"):
            want = float(wide.sum())
        assert got == want or (math.isnan(got) and math.isnan(want)), (v, got, want)
        return
    exact = math.fsum(wide)
    if abs(exact) > FLT_MAX * (1 + 2.0 ** -24):
        assert got == math.copysign(INF, exact), (v, got, exact)
        return
    bound = (math.ceil(len(v) / 8) + 2) * 2.0 ** -53 * math.fsum(np.abs(wide))
    assert abs(got - exact) <= bound + 2.0 ** -24 * (abs(exact) + bound) + 2.0 ** -150, (v, got, exact)


@pytest.mark.parametrize("n", [1, 4, 31, 32, 33, 128, 152])
def test_infinities_and_sums_beyond_the_range_of_fp32(sum_terms, n):
    """Infinite and NaN terms, and running sums that overflow although the whole does not:
    what FP64 gives, wherever the terms stand."""
    heads = [[INF], [-INF], [INF, -INF], [math.nan], [INF, 1, -3], [3e38, 3e38, -3.2e38], [-3e38, -3e38, 3.2e38, 1],
             [3e38, 3e38], [-3e38, -3e38], [FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX, 5], [FLT_MAX, -FLT_MAX, 1e30]]
    for head in heads:
        for at in (0, 1, n - len(head)):
            for gap in (1, 4):  # in neighbouring sums, in one
                v = np.full(n, 0.25, np.float32)
                for i, x in enumerate(head):
                    if 0 <= at + i * gap < n:
                        v[at + i * gap] = x
                _check(sum_terms, v)


@pytest.mark.parametrize("n", [2, 33, 128, 152])
@pytest.mark.parametrize("spread", [0, 8, 20, 60])
def test_terms_that_cancel(sum_terms, n, spread):
    """Random terms over 2^spread whose last one cancels nearly all of the rest, sums of
    signed pairs in a shuffled order, and long runs of one sign: no further off than FP64."""
    rng = np.random.default_rng(100 * n + spread)
    for _ in range(300):
        v = (rng.standard_normal(n) * 2.0 ** rng.uniform(-spread, 0, n)).astype(np.float32)
        _check(sum_terms, v)
        _check(sum_terms, np.abs(v))
        w = v.copy()
        w[-1] = -math.fsum(v[:-1].astype(np.float64))
        _check(sum_terms, w)
        k = n // 2
        w = v.copy()
        w[k:2 * k] = -w[:k] * np.float32(1 + 2.0 ** -23)
        _check(sum_terms, rng.permutation(w))
