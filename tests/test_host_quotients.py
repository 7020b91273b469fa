"""The branch-free quotients of the FP64 column solves (rcp2, quot and the range
tests in vphys_device.cuh) against the IEEE quotient a / b, bit for bit, on
the CPU: the header is compiled as host C++ with the hardware's reciprocal
seed replaced by 1/b cut to 20 bits (the seed's documented precision), so the
two Newton steps and Markstein's correction run as on the GPU.

Random operands, and the hardest ones: for an odd 53-bit B and a midpoint q
(odd, 54 bits) with B q = r (mod 2^54), A = (B q - r) / 2^54 gives a quotient
A / B that misses the midpoint between two doubles by r units of the last place
of the product; r = +-1 is the closest any quotient comes.  B covers both ends of
the binade, next to the significands that den_ok refuses.  No difference is
allowed, so there is no tolerance."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
HERE = Path(__file__).resolve().parent / "host_kernels"

SOURCE = r'''
#include "prelude.h"
using namespace vphys;
typedef unsigned long long u64;
typedef unsigned __int128 u128;
static u64 mix(u64 &s) { s += 0x9e3779b97f4a7c15ull; u64 z = s; z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull; z = (z ^ (z >> 27)) * 0x94d049bb133111ebull; return z ^ (z >> 31); }
// 0: not taken by the fast form, 1: equal, 2: different
static int one(double a, double b)
{
    if (!(num_ok(a) && den_ok(b))) return 0;
    const double q = quot(a, b, rcp2(b)), w = a / b;
    return q == w ? 1 : 2;
}
extern "C" void host_random(u64 seed, long long n, int emin, int erange, long long *out)
{
    u64 s = seed;
    for (long long i = 0; i < n; ++i) {
        const u64 r = mix(s), t = mix(s);
        const double a = __longlong_as_double((long long)((r & 0x800fffffffffffffull) | ((u64)(1023 + emin + (int)((r >> 52) % 2048) % erange) << 52)));
        const double b = __longlong_as_double((long long)((t & 0x800fffffffffffffull) | ((u64)(1023 + emin + (int)((t >> 52) % 2048) % erange) << 52)));
        out[one(a, b)]++;
    }
}
// B odd, its high bits from `top` (0: the whole binade, 1: just above a power of two, 2: just below the refused ones)
extern "C" void host_midpoints(u64 seed, long long n, int top, long long *out)
{
    u64 s = seed;
    const u64 M = (1ull << 54) - 1;
    for (long long i = 0; i < n; ++i) {
        u64 B = (mix(s) & ((1ull << 52) - 1)) | (1ull << 52) | 1;
        if (top == 1) B = (1ull << 52) | (B & 0xfffff) | 1;
        if (top == 2) B = (1ull << 52) | (0xffffeull << 32) | 0xffffffffull ^ ((B & 0xff) << 1);
        u64 inv = B;   // B^-1 mod 2^64 by Newton
        for (int k = 0; k < 6; ++k) inv *= 2 - B * inv;
        const long long r = ((long long)(mix(s) % 8) - 4) * 2 + 1;   // odd, -7 .. 7
        const u64 q = (inv * (u64)r) & M;
        if (q < (1ull << 53)) continue;   // not a 54-bit midpoint
        const u128 prod = (u128)B * q;
        const u128 A = (prod - (u128)(__int128)r) >> 54;
        if (A >= ((u128)1 << 53) || A == 0) continue;
        const int e = (int)(mix(s) % 200) - 100;
        out[one(std::ldexp((double)(u64)A, e), (r & 2) ? (double)B : -(double)B)]++;
    }
}
extern "C" int host_refused(void)
{
    const double inf = INFINITY, tiny = 0x1p-1060, nan = NAN;
    return num_ok(inf) + num_ok(nan) + num_ok(tiny) + num_ok(-tiny) + num_ok(0x1p-600) + den_ok(0.0) + den_ok(inf) +
           den_ok(nan) + den_ok(tiny) + den_ok(0x1p600) + den_ok(__longlong_as_double(0x3fffffffffffffffll)) +
           !num_ok(0.0) + !num_ok(-0.0) + !num_ok(-3.0) + !den_ok(-1.0) + !den_ok(1.0) + !den_ok(1.0e-30);
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    tmp = tmp_path_factory.mktemp("quot")
    (tmp / "q.cpp").write_text(SOURCE)
    so = tmp / "q.so"
    cmd = ["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-fPIC", "-shared", "-w", f"-I{HERE}",
           f"-I{ROOT / 'roundabout_b200' / 'csrc'}", "-o", str(so), str(tmp / "q.cpp")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    L = ctypes.CDLL(str(so))
    L.host_random.argtypes = [ctypes.c_ulonglong, ctypes.c_longlong, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    L.host_midpoints.argtypes = [ctypes.c_ulonglong, ctypes.c_longlong, ctypes.c_int, ctypes.c_void_p]
    return L


@pytest.mark.parametrize("emin,erange", [(0, 1), (-40, 80), (-511, 1022)])
def test_random_quotients(lib, emin, erange):
    out = (ctypes.c_longlong * 3)()
    lib.host_random(1234 + emin, 2_000_000, emin, erange, out)
    assert out[2] == 0 and out[1] > 1_900_000, list(out)


@pytest.mark.parametrize("top", [0, 1, 2])
def test_quotients_next_to_a_midpoint(lib, top):
    out = (ctypes.c_longlong * 3)()
    lib.host_midpoints(77 + top, 1_000_000, top, out)
    assert out[2] == 0 and out[1] > 100_000, list(out)


def test_operands_the_fast_form_refuses(lib):
    assert lib.host_refused() == 0
