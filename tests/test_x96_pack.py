"""The two-step conversion of the epilogue's 96-bit integers (x96_normalise or
x64_normalise, then x96_pack, in muscle.jl_gb300/csrc/mgb_x96.h), compiled for
the host: bit for bit the general routine's result (which is checked against
exact rational rounding elsewhere) for every exponent that x96_plain_exponent
takes, up to its ends; and those ends are the last at which no result is
subnormal or overflows."""
import ctypes
import os
import random
import shutil
import struct
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "muscle.jl_gb300", "csrc")

SHIM = r'''
#include "mgb_x96.h"
using namespace mgb;
extern "C" double general(unsigned w0, unsigned w1, unsigned w2, int e) { return x96_ldexp_rn_general(w0, w1, w2, e); }
extern "C" double pack96(unsigned w0, unsigned w1, unsigned w2, int e) {
    return x96_bits_to_double(x96_pack(x96_normalise(w0, w1, w2), e));
}
extern "C" double pack64(unsigned w0, unsigned w1, unsigned w2, int e) {
    return x96_bits_to_double(x96_pack(x64_normalise(w0, w1), e));
}
extern "C" int is64(unsigned w1, unsigned w2) { return x96_is_64(w1, w2); }
extern "C" int plain(int e) { return x96_plain_exponent(e); }
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("x96p")
    (d / "s.cpp").write_text(SHIM)
    subprocess.run([gxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, str(d / "s.cpp"), "-o", str(d / "s.so")],
                   check=True)
    lib = ctypes.CDLL(str(d / "s.so"))
    for n in ("general", "pack96", "pack64"):
        getattr(lib, n).restype = ctypes.c_double
        getattr(lib, n).argtypes = [ctypes.c_uint32] * 3 + [ctypes.c_int]
    return lib


def words(x):
    u = x & ((1 << 96) - 1)
    return u & 0xFFFFFFFF, (u >> 32) & 0xFFFFFFFF, (u >> 64) & 0xFFFFFFFF


def bits(d):
    return struct.pack("<d", d)


def values():
    rng = random.Random(7)
    v = {0}
    for p in range(96):
        for d in (-1, 0, 1):
            v.add((1 << p) + d)
        for s in (52, 53, 54, 63, 64):  # ties at the last kept bit, and one unit beside them
            if p > s:
                for d in (-1, 0, 1):
                    v.add((1 << p) + (1 << (p - s)) + d)
                    v.add((1 << p) + (3 << (p - s)) + d)
        for _ in range(6):
            v.add(rng.getrandbits(p + 1))
    return sorted(x for x in v if x < 1 << 95)


@pytest.mark.parametrize("e", [-1022, -1021, -500, -56, 0, 500, 926, 927])
def test_pack_is_the_general_conversion(lib, e):
    assert lib.plain(e)
    for a in values():
        for x in (a, -a):
            w = words(x)
            want = bits(lib.general(*w, e))
            assert bits(lib.pack96(*w, e)) == want, (x, e)
            fits = -(1 << 63) <= x < 1 << 63
            assert bool(lib.is64(w[1], w[2])) == fits, x
            if fits:
                assert bits(lib.pack64(*w, e)) == want, (x, e)


def test_plain_exponents_end_where_results_leave_the_normal_range(lib):
    assert not lib.plain(-1023) and not lib.plain(928) and not lib.plain(1 << 20) and not lib.plain(-(1 << 20))
    assert lib.general(*words(1), -1022) >= 2.0 ** -1022 > lib.general(*words(1), -1023)
    top = (1 << 95) - 1
    assert lib.general(*words(top), 927) == 2.0 ** 1022 and lib.general(*words(top), 928) == 2.0 ** 1023
