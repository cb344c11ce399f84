"""The residue-number-system products of the final sum (csrc/rns.cuh), run
lane by lane on the host (tests/native/rns_check.cpp) against big integers: the
moduli, products of reduced values and of sums at the stated bounds, the
doubling chain's value and word bounds, and the conversions in and out."""
import ctypes
import math
import os
import random
import subprocess

import numpy as np
import pytest

from conftest import NATIVE, PKG

P = 0x30644E72E131A029B85045B68181585D97816A916871CA8D3C208C16D87CFD47
W = 1 << 32


@pytest.fixture(scope="module")
def lib():
    out = os.path.join(NATIVE, "_build")
    os.makedirs(out, exist_ok=True)
    so, src = os.path.join(out, "librns_check.so"), os.path.join(NATIVE, "rns_check.cpp")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I" + os.path.join(PKG, "csrc"),
                    "-o", so, src], check=True)
    return ctypes.CDLL(so)


class Rns:
    def __init__(self, lib):
        self.lib = lib
        self.n = lib.rns_residues()
        a, b = np.zeros(self.n, np.int32), np.zeros(self.n, np.int32)
        lib.rns_moduli(a.ctypes.data_as(ctypes.c_void_p), b.ctypes.data_as(ctypes.c_void_p))
        self.a, self.b = [int(v) for v in a], [int(v) for v in b]
        self.A, self.B = math.prod(self.a), math.prod(self.b)

    def call(self, name, *args):
        getattr(self.lib, name)(*[v.ctypes.data_as(ctypes.c_void_p) for v in args])

    def enter(self, v):
        words = np.array([(v >> (32 * k)) & 0xFFFFFFFF for k in range(8)], np.uint32)
        out = np.zeros(2 * self.n, np.int32)
        self.call("rns_from_words", words, out)
        return out

    def product(self, x, y):
        out = np.zeros(2 * self.n, np.int32)
        self.call("rns_product", np.ascontiguousarray(x, np.int32), np.ascontiguousarray(y, np.int32), out)
        return out

    def words(self, x, y):
        out = np.zeros(8, np.uint32)
        self.call("rns_product_words", np.ascontiguousarray(x, np.int32), np.ascontiguousarray(y, np.int32), out)
        return sum(int(w) << (32 * k) for k, w in enumerate(out))

    def value(self, x):
        """The integer nearest to zero with these stored residues; both bases agree."""
        got = []
        for mods, M, part in ((self.a, self.A, x[:self.n]), (self.b, self.B, x[self.n:])):
            v = sum(int(r) * pow(W, -1, m) % m * pow(M // m, -1, m) % m * (M // m) for r, m in zip(part, mods)) % M
            got.append(v - M if v > M // 2 else v)
        assert got[0] == got[1]
        return got[0]


@pytest.fixture(scope="module")
def rns(lib):
    return Rns(lib)


def test_moduli(rns):
    mods = rns.a + rns.b
    assert len(set(mods)) == len(mods) and all(m < 1 << 27 for m in mods)
    for i, m in enumerate(mods):
        assert all(m % q for q in range(2, math.isqrt(m) + 1)), f"{m} is not prime"
        assert all(math.gcd(m, q) == 1 for q in mods[:i])


def corner_values():
    rng = random.Random(5)
    return [0, 1, 2, P - 1, P, P + 1, 2 * P - 1] + [rng.randrange(2 * P) for _ in range(40)]


def test_products(rns):
    """r = x y / A modulo p, |r| < 6.5 p + |x y| / A, words within 1.25 * 2^26."""
    inv = pow(rns.A, -1, P)
    vals = corner_values()
    for x, y in zip(vals, reversed(vals)):
        r = rns.product(rns.enter(x), rns.enter(y))
        v = rns.value(r)
        assert (v - x * y * inv) % P == 0
        assert abs(v) < 6.5 * P + x * y / rns.A
        assert max(abs(int(w)) for w in r) < 1.25 * 2 ** 26


def test_products_of_sums(rns):
    """Operands of up to 20 summed outputs, the most the doubling uses."""
    rng = random.Random(6)
    outs = [rns.product(rns.enter(rng.randrange(P)), rns.enter(rng.randrange(P))) for _ in range(8)]
    inv = pow(rns.A, -1, P)
    for x, y in zip(outs, outs[1:]):
        for i, j in ((20, 20), (-20, 13), (3, -20), (20, 1)):
            r = rns.product(i * x, j * y)
            assert (rns.value(r) - rns.value(i * x) * rns.value(j * y) * inv) % P == 0
            assert max(abs(int(w)) for w in r) < 1.25 * 2 ** 26


def test_zero_stays_zero(rns):
    zero, x = rns.enter(0), rns.enter(12345)
    assert not rns.product(zero, x).any()


def test_words_out(rns):
    """p + (x y + q p) / A with q nearest to zero: the right residue class, in (0, 2p)."""
    enter, leave = np.zeros(2 * rns.n, np.int32), np.zeros(2 * rns.n, np.int32)
    rns.call("rns_constants", enter, leave)
    inv = pow(rns.A, -1, P)
    for x in corner_values():
        inside = rns.product(rns.enter(x), enter)  # x 2^256 mod p -> x A
        assert (rns.value(inside) - (x * pow(1 << 256, -1, P)) * rns.A) % P == 0
        for k in (1, -7, 20):
            v = rns.words(k * inside, leave)
            assert 0 < v < 2 * P and (v - k * x) % P == 0
    assert (rns.words(rns.enter(7), rns.enter(9)) - 63 * inv) % P == 0


def test_doubling_chain(rns):
    """The doubling of the final sum, 260 times over: the right point, values
    and words within the bounds its comment states."""
    rng = random.Random(8)
    x, y, z = (rng.randrange(P) for _ in range(3))
    X, Y, Z = (rns.enter(v * rns.A % P) for v in (x, y, z))
    most_word, most_value = 0, 0
    for _ in range(260):
        A, B, YZ = rns.product(X, X), rns.product(Y, Y), rns.product(Y, Z)
        E = 3 * A
        F, S, C = rns.product(E, E), rns.product(X, B), rns.product(B, B)
        D = 4 * S
        X3 = F - 8 * S
        operands = [E, D - X3]
        Y3 = rns.product(E, D - X3) - 8 * C
        X, Y, Z = X3, Y3, 2 * YZ
        e = 3 * x * x
        nx = (e * e - 8 * x * y * y) % P
        x, y, z = nx, (e * (4 * x * y * y - nx) - 8 * y ** 4) % P, 2 * y * z % P
        for w in operands + [X, Y, Z]:
            most_word = max(most_word, int(np.abs(w.astype(np.int64)).max()))
            most_value = max(most_value, abs(rns.value(w)))
    inv = pow(rns.A, -1, P)
    assert [rns.value(v) * inv % P for v in (X, Y, Z)] == [x, y, z]
    assert most_word < 13 * 1.25 * 2 ** 26 and most_value < 85 * P


def test_multiples_of_p(rns):
    """A product's output is recognised as k p, |k| <= 6, and only then."""
    rng = random.Random(9)
    one = rns.enter(1)
    is_multiple = lambda x: (rns.lib.rns_multiples(np.ascontiguousarray(x, np.int32).ctypes.data_as(ctypes.c_void_p)) & 0x007F007F) != 0
    for trial in range(200):
        x = rng.randrange(P)
        zero = rns.product(rns.enter(P) if trial % 2 else rns.enter(0), rns.enter(x))  # (p or 0) x: some multiple of p
        assert rns.value(zero) % P == 0 and is_multiple(zero)
        other = rns.product(rns.enter(x), one)
        assert is_multiple(other) == (x == 0)
    stored_p = rns.enter(P)
    for k in range(-6, 7):  # every multiple, with words reduced as a product's are
        words = []
        for part, mods in ((stored_p[:rns.n], rns.a), (stored_p[rns.n:], rns.b)):
            words += [((int(w) * k + m // 2) % m) - m // 2 for w, m in zip(part, mods)]
        assert is_multiple(np.array(words))
        near = list(words)
        near[3] += 1 if near[3] <= 0 else -1
        assert not is_multiple(np.array(near))


def test_additions(rns):
    """The final sum's addition on doubled and added operands, 60 times over."""
    rng = random.Random(10)
    inv = pow(rns.A, -1, P)
    p, q = ([rng.randrange(1, P) for _ in range(3)] for _ in range(2))
    Pt, Qt = ([rns.enter(v * rns.A % P) for v in pt] for pt in (p, q))
    for step in range(60):
        (x1, y1, z1), (x2, y2, z2) = Pt, Qt
        zz1, zz2, z12 = rns.product(z1, z1), rns.product(z2, z2), rns.product(z1, z2)
        U1, U2, z2c = rns.product(x1, zz2), rns.product(x2, zz1), rns.product(z2, zz2)
        H = U2 - U1
        S1, z1c, HH = rns.product(y1, z2c), rns.product(z1, zz1), rns.product(H, H)
        S2, HHH, V = rns.product(y2, z1c), rns.product(H, HH), rns.product(U1, HH)
        R = S2 - S1
        RR, T, Z = rns.product(R, R), rns.product(S1, HHH), rns.product(z12, H)
        X = RR - HHH - 2 * V
        Y = rns.product(R, V - X) - T
        (a, b, c), (d, e, f) = p, q
        h, r = (d * c * c - a * f * f) % P, (e * c ** 3 - b * f ** 3) % P
        v = a * f * f * h * h % P
        x = (r * r - h ** 3 - 2 * v) % P
        want = [x, (r * (v - x) - b * f ** 3 * h ** 3) % P, c * f * h % P]
        assert [rns.value(w) * inv % P for w in (X, Y, Z)] == want
        assert max(int(np.abs(w.astype(np.int64)).max()) for w in (H, R, X, V - X, Y)) < 13 * 1.25 * 2 ** 26
        p, q, Pt, Qt = q, want, Qt, [X, Y, Z]
