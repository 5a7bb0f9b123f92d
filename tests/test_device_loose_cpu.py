"""The device arithmetic on values that are not fully reduced -- mul_loose, sub_loose, the NTT's
butterflies --, the additions with inlined products and the pair rounds' case logic, emulated on the
host (tests/device_emul.py) at the ends of the ranges that their bounds name."""
import ctypes
import random

import pytest

import bn254_ref as o
import device_emul
from test_device_arith_cpu import CurveIO, dev  # noqa: F401  (the emulation fixture)

PQ, PR = o.P_FQ, o.P_FR
R = 1 << 256


def ends(p, k, rng, n=40):
    """values below k p: the ends of every multiple of p, and random ones of each"""
    out = []
    for i in range(k):
        out += [i * p, i * p + 1, (i + 1) * p - 2, (i + 1) * p - 1] + [rng.randrange(i * p, (i + 1) * p) for _ in range(n)]
    return [v for v in out if v < R]


@pytest.mark.parametrize("pfx,p", [("fq", PQ), ("fr", PR)])
def test_mul_loose(dev, pfx, p):  # noqa: F811
    rng, W, ri = random.Random(30), dev.words, pow(R, -1, p)
    for b in ends(p, 5, rng) + [R - 1, R - 2, R - p]:
        for a in [0, 1, p - 1, rng.randrange(p)]:
            got = dev.call(pfx + "_mul_loose", [W(a), W(b)], 8)
            assert got % p == a * b * ri % p
            assert got <= p + a * b // R
            if b < 5 * p:
                assert got < 2 * p
            # and the fully reduced product of the same
            assert dev.call(pfx + "_mul", [W(a), W(b)], 8) % p == a * b * ri % p


def test_sub_loose(dev):  # noqa: F811
    rng, W = random.Random(31), dev.words
    vals = ends(PQ, 1, rng)
    for a in vals:
        for b in [0, 1, PQ - 1, a, rng.choice(vals)]:
            got = dev.call("fq_sub_loose", [W(a), W(b)], 8)
            assert got == a - b + PQ


def test_ntt_helpers(dev):  # noqa: F811
    rng, W, r = random.Random(32), dev.words, PR
    for a in ends(r, 4, rng):
        assert dev.call("fr_reduce2", [W(a)], 8) == (a - 2 * r if a >= 2 * r else a)
    for a in ends(r, 6, rng) + [R - 1, R - 2, R >> 1]:  # a caller's word: any of 256 bits
        got = dev.call("fr_below2", [W(a)], 8)
        assert got % r == a % r and got < 2 * r
    two = ends(r, 2, rng)
    for a in two:
        assert dev.call("fr_reduce1", [W(a)], 8) == a % r
        b = rng.choice(two)
        assert dev.call("fr_add_raw", [W(a), W(b)], 8) == a + b
        for b in [0, 2 * r - 1, b]:
            assert dev.call("fr_sub_plus2", [W(a), W(b)], 8) == a - b + 2 * r


@pytest.mark.parametrize("name,bound", [("butterfly_dif", 2), ("butterfly_dit", 4)])
@pytest.mark.parametrize("unit", [0, 1])
def test_butterflies(dev, name, bound, unit):  # noqa: F811
    """(x0 + x1, (x0 - x1) w) and (x0 + x1 w, x0 - x1 w) modulo r, and back within the bound"""
    rng, r = random.Random(33 + unit), PR
    ri = pow(R, -1, r)
    vals = ends(r, bound, rng, 20)
    for x0 in vals:
        for x1 in [0, r, bound * r - 1, rng.choice(vals), rng.choice(vals)]:
            w = rng.choice([1, r - 1, rng.randrange(r)])
            f = 1 if unit else w * ri
            a, b = (ctypes.c_uint32 * 8)(*dev.words(x0)), (ctypes.c_uint32 * 8)(*dev.words(x1))
            getattr(dev.lib, name)(a, b, dev.words(w), unit)
            a, b = dev.value(a), dev.value(b)
            want = ((x0 + x1) % r, (x0 - x1) * f % r) if bound == 2 else ((x0 + x1 * f) % r, (x0 - x1 * f) % r)
            assert (a % r, b % r) == want
            assert a < bound * r and b < bound * r


@pytest.mark.parametrize("g2", [False, True], ids=["g1", "g2"])
def test_inlined_additions(dev, g2):  # noqa: F811
    curve = o.G2 if g2 else o.G1
    io, pfx, rng = CurveIO(dev, curve, g2), "g2" if g2 else "g1", random.Random(34 + g2)
    pts = [curve.mul(curve.gen, rng.randrange(1, PR)) for _ in range(6 if g2 else 20)]
    for i, P in enumerate(pts):
        Q = pts[(i + 1) % len(pts)]
        for A, B in [(P, Q), (P, P), (P, curve.neg(P)), (None, Q), (P, None), (None, None)]:
            got = dev.call(pfx + "_add_inline", [io.xyzz(A, io.rand_lam(rng)), io.xyzz(B, io.rand_lam(rng))], 4 * io.fw)
            assert io.from_xyzz(got) == curve.add(A, B)


def test_division_steps_follow_the_recurrence(dev):  # noqa: F811
    """30 steps on the low words: the matrix takes the whole numbers where Bernstein and Yang's
    recurrence does"""
    from test_host_ff_cpu import divstep
    rng = random.Random(35)
    for i in range(400):
        f, g = rng.getrandbits(254) | 1, rng.getrandbits(254) << rng.choice([0, 1, 7, 29, 40])
        f, g = (f, g) if i % 3 else (-f, g)
        delta = rng.randint(-40, 40)
        m = (ctypes.c_int32 * 4)()
        got = dev.lib.dsteps30(delta, ctypes.c_uint32(f & 0xffffffff), ctypes.c_uint32(g & 0xffffffff), m)
        d, F, G = delta, f, g
        for _ in range(30):
            d, F, G = divstep(d, F, G)
        u, v, q, r = m
        assert (u * f + v * g, q * f + r * g, got) == (F << 30, G << 30, d)


def test_pair_cases_of_x_zero(dev):  # noqa: F811
    """a point of x = 0 beside a missing one has a zero denominator without an addition due; two of
    equal x and opposite y have no sum, equal ones the tangent"""
    W, rng = dev.words, random.Random(36)
    y = rng.randrange(1, PQ)
    mont = lambda v: v * R % PQ
    z, p, n = (0, 0), (0, mont(y)), (0, mont(PQ - y))

    def add(a, b):
        kind, out = ctypes.c_uint32(), (ctypes.c_uint32 * 16)()
        cat = lambda t: W(t[0] | t[1] << 256, 16)
        dev.lib.g1_pair_add(cat(a), cat(b), ctypes.byref(kind), out)
        v = dev.value(out)
        return kind.value, (v & (R - 1), v >> 256)
    assert add(p, z) == (3, p) and add(z, p) == (4, p) and add(z, z) == (4, z)
    assert add(p, n) == (2, z)
    # x = 0: the tangent's slope is 0, so 2 P = (0, -y)
    assert add(p, p) == (1, n)


@pytest.mark.parametrize("header,old,new,check", [
    ("ec.cuh", "none = none || (!mp && !mq);", "none = none;", test_pair_cases_of_x_zero),
    ("ntt_butterfly.cuh", "const Fr a = reduce2(x0);", "const Fr a = x0;", None),
])
def test_a_planted_mistake_is_seen(tmp_path, header, old, new, check):
    """the tests above run the kernels' own functions"""
    from test_device_arith_cpu import _mutated_build

    def edit(src):
        t = (src / header).read_text()
        assert t.count(old) == 1
        (src / header).write_text(t.replace(old, new))
    d = _mutated_build(tmp_path, edit)
    with pytest.raises(AssertionError):
        if check:
            check(d)
        else:
            test_butterflies(d, "butterfly_dit", 4, 0)
