"""The running sums of the Float64 reductions (FxAcc of mgb_fxsum.h), compiled
for the host with g++: groups of one or four values, against exact rational
sums and against FxSum, which aligns and adds one value at a time."""
import ctypes
import math
import random
import shutil
import subprocess

import pytest

from tests.test_fxsum import exact, window
from tests.test_x96 import CSRC, same

SHIM = r'''
#include "mgb_fxsum.h"
using namespace mgb;
extern "C" double acc_sum(const double *x, int n, int parts) {
    FxSum total = fx_zero();
    for (int p = 0; p < parts; ++p) {
        FxAcc a = fx_acc_zero();
        int i = (int)((long long)n * p / parts);
        const int end = (int)((long long)n * (p + 1) / parts);
        for (; i + 4 <= end; i += 4) {
            const double v[4] = {x[i], x[i + 1], x[i + 2], x[i + 3]};
            fx_acc_push(a, v);
        }
        for (; i < end; ++i) {
            const double v[1] = {x[i]};
            fx_acc_push(a, v);
        }
        fx_merge(total, fx_acc_sum(a));
    }
    return fx_value(total);
}
'''


@pytest.fixture(scope="module")
def acc(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("acc")
    src, so = d / "shim.cpp", d / "libacc.so"
    src.write_text(SHIM)
    subprocess.run([gxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.acc_sum.restype = ctypes.c_double
    lib.acc_sum.argtypes = [ctypes.POINTER(ctypes.c_double), ctypes.c_int, ctypes.c_int]
    return lambda xs, parts=1: lib.acc_sum((ctypes.c_double * max(len(xs), 1))(*xs), len(xs), parts)


def test_exact_within_the_window(acc):
    rng = random.Random(1)
    for trial in range(400):
        base = rng.randint(-1000, 960)
        xs = window(rng, rng.randint(1, 300), base, base + rng.randint(0, 9))
        want = exact(xs)
        for parts in (1, 3, 32):
            got = acc(xs, parts)
            assert same(got, want) or (want == 0.0 and got == 0.0), (trial, parts, got, want)


def test_wide_ranges_within_the_documented_bound(acc):
    """2^-62 of the largest term per term (the largest terms may cancel, so
    this is no bound in units of the sum), and the final rounding."""
    rng = random.Random(2)
    for trial in range(300):
        xs = window(rng, rng.randint(1, 200), -1070, 1000)
        rng.shuffle(xs)
        want = exact(xs)
        got = acc(xs, rng.choice([1, 4, 32]))
        assert abs(got - want) <= len(xs) * 2.0**-62 * max(map(abs, xs)) + math.ulp(want), (trial, got, want)


def test_rising_exponents_zeros_and_subnormals(acc):
    tiny = 5e-324
    assert same(acc([]), 0.0) and same(acc([0.0, -0.0, 0.0]), 0.0)
    assert same(acc([tiny] * 7), 7 * tiny)
    assert same(acc([2.0**-1022, -tiny]), 2.0**-1022 - tiny)
    assert same(acc([-tiny, 2.0**-1022, 0.0, tiny, -2.0**-1022]), 0.0)
    xs = [(-1.0) ** i * 2.0**i for i in range(60)]  # every group raises the exponent: sums of 60 exact bits
    assert abs(acc(xs) - exact(xs)) <= len(xs) * 2.0**-62 * 2.0**59 + math.ulp(exact(xs))
    xs = [-1.0] * 1000 + [1.0] * 999 + [2.0**9]
    assert same(acc(xs, 5), exact(xs))
    assert acc([1.7e308, 1.7e308]) == math.inf and same(acc([1.7e308, 1.7e308, -1.7e308]), 1.7e308)


def test_infinities_and_nans(acc):
    for xs, want in (([1.0, math.inf, 2.0, 3.0, 4.0], math.inf), ([-math.inf, 3.0], -math.inf)):
        assert acc(xs) == want and acc(xs, 2) == want
    for xs in ([math.inf, 1.0, -math.inf], [math.nan, 1.0, 2.0, 3.0], [1.0] * 7 + [math.nan]):
        assert math.isnan(acc(xs)) and math.isnan(acc(xs, 3))
