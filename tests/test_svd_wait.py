"""The limits of the cooperative SVD's waits (muscle.jl_gb300/csrc/mgb_svd_wait.h,
compiled for the host): every matrix that mgb_svd takes has several rounds' time
for a neighbour, and a sweep's end waits for the farthest CTA, while the time
after which a lost CTA is reported stays bounded."""
import ctypes
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "muscle.jl_gb300", "csrc")
SHIM = r'''
#include "mgb_svd_wait.h"
extern "C" long long wait_round(long long f, long long m, long long n, long long s) { return mgb::svd_wait_round(f, m, n, s); }
extern "C" long long wait_sweep(long long f, long long m, long long n, long long s, long long c) {
    return mgb::svd_wait_sweep(f, m, n, s, c);
}
'''
FLOOR = 2 * 10**9
SMS = 152


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("svdw")
    (d / "s.cpp").write_text(SHIM)
    subprocess.run([gxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, str(d / "s.cpp"), "-o", str(d / "s.so")],
                   check=True)
    lib = ctypes.CDLL(str(d / "s.so"))
    for f, n in ((lib.wait_round, 4), (lib.wait_sweep, 5)):
        f.restype, f.argtypes = ctypes.c_longlong, [ctypes.c_longlong] * n
    return lib


def test_limits_cover_every_matrix(lib):
    for N in (1, 2, 3, 7, 32, 128, 129, 255, 304, 305, 1000, 1024):
        pairs = (N + 1) // 2
        spc = -(-pairs // SMS)
        ctas = -(-pairs // spc)
        for M in sorted({N, 1024, 4096, 1 << 18, (1 << 28) // N}):
            if M < N or M * N > 1 << 28:
                continue
            # measured cycles per element of a pair
            busy = 14.4 * spc * (M + N)
            r, s = lib.wait_round(FLOOR, M, N, spc), lib.wait_sweep(FLOOR, M, N, spc, ctas)
            assert r >= FLOOR and r >= 8 * busy
            assert s >= r and s >= ctas * busy  # neighbours differ by a round at most
            assert s <= FLOOR + 400 * 16 * spc * (M + N)


def test_the_kernel_waits_by_them():
    src = open(os.path.join(CSRC, "mgb_svd.cu")).read()
    assert "svd_wait_round(kWaitTimeoutCycles" in src and "svd_wait_sweep(kWaitTimeoutCycles" in src
    assert "clock64() - t0 > limit" in src
