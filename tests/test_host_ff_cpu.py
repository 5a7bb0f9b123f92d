"""The host field arithmetic (host_ff.hpp), compiled by itself: products with a factor at or above the
modulus, and what a caller's words become before they enter a product whose first factor has to be
below it.  Checked against Python integers."""
import ctypes
import os
import random
import subprocess

import pytest

import bn254_ref as o
from conftest import PKG

R = 1 << 256
SRC = r"""
#include "host_ff.hpp"
using namespace bgh;
static Fe ld(const uint64_t* a) { return {{a[0], a[1], a[2], a[3]}}; }
static void st(uint64_t* r, const Fe& a) { for (int i = 0; i < 4; i++) r[i] = a.v[i]; }
extern "C" {
void t_mul(int fq, const uint64_t* a, const uint64_t* b, uint64_t* r) { st(r, fe_mul(fq ? FQ : FR, ld(a), ld(b))); }
void t_to_mont(int fq, const uint64_t* a, uint64_t* r) { st(r, fe_to_mont(fq ? FQ : FR, ld(a))); }
void t_from_mont(int fq, const uint64_t* a, uint64_t* r) { st(r, fe_from_mont(fq ? FQ : FR, ld(a))); }
void t_inv(int fq, const uint64_t* a, uint64_t* r) { st(r, fe_inv(fq ? FQ : FR, ld(a))); }
void t_steps(int64_t delta, uint64_t f, uint64_t g, int64_t* out) { out[4] = dsteps::steps62(delta, f, g, out); }
void t_blinding(const uint32_t* rs16, uint64_t* out) { blinding_scalars(rs16, out, out + 4, out + 8); }
void t_point(const uint32_t* w32, uint64_t* out) {
  const Aff<Fq2Ops> a = aff_from_input32<Fq2Ops>(w32);
  st(out, a.x.c0); st(out + 4, a.x.c1); st(out + 8, a.y.c0); st(out + 12, a.y.c1);
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("host_ff")
    (d / "t.cpp").write_text(SRC)
    so = str(d / "t.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(PKG, "csrc"), "-o", so,
                    str(d / "t.cpp")], check=True)
    return ctypes.CDLL(so)


def w64(x, n=4):
    return (ctypes.c_uint64 * n)(*[(x >> (64 * i)) & (2**64 - 1) for i in range(n)])


def value(w):
    return sum(int(v) << (64 * i) for i, v in enumerate(w))


def call(lib, name, *args):
    out = (ctypes.c_uint64 * 4)()
    getattr(lib, name)(*args, out)
    return value(out)


def edges(p, rng):
    """representatives at and above the modulus, up to the largest 256-bit word"""
    return [0, 1, p - 1, p, p + 1, 2 * p - 1, 4 * p, 5 * p - 1, R - p - 1, R - p, R - p + 1, R - 2, R - 1] + \
        [rng.randrange(p, R) for _ in range(300)]


@pytest.mark.parametrize("fq", [0, 1])
def test_conversions_take_any_words(lib, fq):
    p = o.P_FQ if fq else o.P_FR
    rng = random.Random(70 + fq)
    ri = pow(R, -1, p)
    for a in edges(p, rng):
        assert call(lib, "t_to_mont", fq, w64(a)) == a * R % p
        assert call(lib, "t_from_mont", fq, w64(a)) == a * ri % p
        b = rng.randrange(p)
        assert call(lib, "t_mul", fq, w64(b), w64(a)) == a * b * ri % p


def test_blinding_scalars_at_and_above_the_modulus(lib):
    p = o.P_FR
    rng = random.Random(72)
    ri = pow(R, -1, p)
    words = edges(p, rng)
    for rm in words:
        sm = rng.choice(words)
        rs = (ctypes.c_uint32 * 32)(*[(v >> (16 * i)) & 0xffff for v in (rm, sm) for i in range(16)])
        out = (ctypes.c_uint64 * 12)()
        lib.t_blinding(rs, out)
        r, s = rm * ri % p, sm * ri % p
        assert [value(out[4 * i:4 * i + 4]) for i in range(3)] == [r, s, r * s % p]


def test_input_points_are_reduced(lib):
    p = o.P_FQ
    rng = random.Random(73)
    words = edges(p, rng)
    for _ in range(200):
        v = [rng.choice(words) for _ in range(4)]
        w = (ctypes.c_uint32 * 32)(*[(x >> (32 * i)) & 0xffffffff for x in v for i in range(8)])
        out = (ctypes.c_uint64 * 16)()
        lib.t_point(w, out)
        assert [value(out[4 * i:4 * i + 4]) for i in range(4)] == [x % p for x in v]


def divstep(delta, f, g):
    """Bernstein and Yang's division step (CHES 2019, section 8)"""
    if delta > 0 and g & 1:
        return 1 - delta, g, (g - f) // 2
    return 1 + delta, f, (g + (g & 1) * f) // 2


def test_division_steps_follow_the_recurrence(lib):
    """62 steps on the low words: the matrix takes the whole numbers where the recurrence does"""
    rng = random.Random(74)
    for i in range(400):
        f, g = rng.getrandbits(254) | 1, rng.getrandbits(254) << rng.choice([0, 1, 7, 61, 70])
        f, g = (f, g) if i % 3 else (-f, g)
        delta = rng.randint(-40, 40)
        out = (ctypes.c_int64 * 5)()
        mask = (1 << 64) - 1
        lib.t_steps(ctypes.c_int64(delta), ctypes.c_uint64(f & mask), ctypes.c_uint64(g & mask), out)
        d, F, G = delta, f, g
        for _ in range(62):
            d, F, G = divstep(d, F, G)
        u, v, q, r = out[:4]
        assert (u * f + v * g, q * f + r * g, out[4]) == (F << 62, G << 62, d)


@pytest.mark.parametrize("fq", [0, 1])
def test_inverse(lib, fq):
    p = o.P_FQ if fq else o.P_FR
    rng = random.Random(75 + fq)
    ri = pow(R, -1, p)
    vals = [1, 2, 3, p - 1, p - 2, R % p, R * R % p] + [1 << k for k in range(0, 254, 5)] + \
        [p - (1 << k) for k in range(1, 250, 11)] + [rng.randrange(1, p) for _ in range(3000)]
    assert call(lib, "t_inv", fq, w64(0)) == 0
    for a in vals:
        assert call(lib, "t_inv", fq, w64(a)) == pow(a * ri, -1, p) * R % p
