"""The final sum's device code (csrc/msm_final.cuh) run on the host with the
warp, block and cluster intrinsics emulated (tests/native/final_check.cpp), with
array bounds checked: whole sums against the oracle's Horner pass, and what
every lane of a warp holds after each of its operations."""
import os
import subprocess

import numpy as np
import pytest

import msm_helpers as H
from conftest import NATIVE, PKG, REPO

P, MONT = H.P, H.MONT
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
RESIDUES, GROUPS = 10, 3
OPERATIONS = ("load p", "load q", "put and get", "doubled", "added")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    out = os.path.join(NATIVE, "_build")
    os.makedirs(out, exist_ok=True)
    exe = os.path.join(out, "final_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fsanitize=bounds,null,alignment", "-fno-sanitize-recover=all", "-U_FORTIFY_SOURCE",
                    "-I" + os.path.join(PKG, "csrc"), "-I" + os.path.join(REPO, "include"), "-I" + os.path.join(NATIVE, "emulation"),
                    "-I" + CUDA_INCLUDE, "-o", exe, os.path.join(NATIVE, "final_check.cpp")], check=True)
    directory = tmp_path_factory.mktemp("final")

    def run(mode, words, *options):
        source, target = directory / "in", directory / "out"
        np.ascontiguousarray(words, np.uint32).tofile(source)
        done = subprocess.run([exe, mode, source, target, *options], capture_output=True, text=True, timeout=300)
        assert done.returncode == 0, done.stderr
        return np.fromfile(target, np.uint32)
    return run


def jacobian(pt, z=1):
    """Montgomery-form Jacobian words of an affine point (None: infinity)."""
    if pt is None:
        return np.concatenate([H.limbs(0), H.limbs(MONT % P), H.limbs(0)])
    x, y = pt
    return np.concatenate([H.limbs(x * z * z % P * MONT % P), H.limbs(y * z ** 3 % P * MONT % P), H.limbs(z * MONT % P)])


def neg(pt):
    return (pt[0], (P - pt[1]) % P)


def results_of(points, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    zs = [int.from_bytes(rng.bytes(32), "little") % P or 1 for _ in range(254)]
    return np.stack([jacobian(points.get(i), zs[i]) for i in range(254)]).astype(np.uint32)


def points(out):
    return [(bool(w[16]), H.to_int(w[:8]), H.to_int(w[8:16])) for w in out.reshape(-1, 20)]


def cases():
    table = H.load_g_bases()  # (i + 1) G
    rng = np.random.Generator(np.random.PCG64(3))
    some = lambda: table[int(rng.integers(0, 256))]
    yield "every bit", {i: some() for i in range(254)}
    yield "most bits", {i: neg(some()) if i % 5 == 0 else some() for i in range(254) if rng.random() < 0.8}
    yield "a batched instance", {i: some() for i in range(20)}
    yield "none", {}
    for bits in ([0], [253], [127, 128], [15, 16, 31, 48, 80, 96, 112, 144, 176, 208, 240]):
        yield f"bits {bits}", {i: some() for i in bits}


@pytest.mark.parametrize("order", ["ascending", "descending"])
def test_sums(check, oracle, order):
    named = list(cases())
    if order == "descending":  # lanes, warps and blocks resumed in the other order
        named = named[1:3]
    results = [results_of(pts, k) for k, (_, pts) in enumerate(named)]
    got = points(check("sum", np.concatenate(results), *(["descending"] if order == "descending" else [])))
    for (name, _), r, point in zip(named, results, got):
        assert point == oracle.horner(r), name


def test_equal_and_opposite_partners(check, oracle):
    """2^bit G against +-(G at that bit): a level's two operands are equal or
    opposite; at bit 1 and 2 four lanes per point, from 4 a warp per point."""
    G = H.load_g_bases()[0]
    results = []
    for bit in (1, 2, 4, 8, 16, 64):
        inf, *big = oracle.affine_mul(G[0], G[1], 1 << bit)
        assert not inf
        for partner in (G, neg(G)):
            results.append(results_of({0: tuple(big), bit: partner}, bit))
    for r, point in zip(results, points(check("sum", np.concatenate(results)))):
        assert point == oracle.horner(r)


def test_lanes_of_a_warp(check):
    """Lanes 30 and 31 hold what lanes 20 and 21 hold after every operation (no
    lane reads past a point's ten residues), the three groups agree on X and Y
    and the two that carry Z on Z, and the addition refuses equal and opposite
    points."""
    table = H.load_g_bases()
    rng = np.random.Generator(np.random.PCG64(8))
    z = lambda: int.from_bytes(rng.bytes(32), "little") % P or 1
    pairs = [(table[3], table[8], True), (table[200], table[9], True), (table[5], table[5], False), (table[5], neg(table[5]), False)]
    out = check("lanes", np.concatenate([np.concatenate([jacobian(p, z()), jacobian(q, z())]) for p, q, _ in pairs]))
    size = (len(OPERATIONS) * 6 + 1) * 32
    for k, (_, _, holds) in enumerate(pairs):
        words = out[k * size:(k + 1) * size]
        assert (words[-32:] == holds).all()
        for name, lanes in zip(OPERATIONS, words[:-32].reshape(len(OPERATIONS), 32, 6)):
            if name == "added" and not holds:
                continue
            assert (lanes[30:] == lanes[2 * RESIDUES:2 * RESIDUES + 2]).all(), name
            groups = lanes[:GROUPS * RESIDUES].reshape(GROUPS, RESIDUES, 6)
            assert (groups[:, :, :4] == groups[0, :, :4]).all(), name
            assert (groups[1, :, 4:] == groups[2, :, 4:]).all(), name


def test_inverse_of_a_group(check):
    """inverse_group4 on edge values and random ones, groups of one warp ending
    after different numbers of rounds: a a^-1 = 1 modulo p, 0 -> 0."""
    rng = np.random.Generator(np.random.PCG64(12))
    values = [0, 1, 2, 3, P - 1, P - 2, P // 2, (P + 1) // 2, 1 << 128, (1 << 253) - 1, 0xFFFFFFFF, 1 << 32, 1 << 30, (1 << 30) - 1, P - (1 << 30), 0]
    values += [int.from_bytes(rng.bytes(32), "little") % P for _ in range(400)]
    out = check("inverse", np.concatenate([H.limbs(v) for v in values])).reshape(-1, 8)
    for v, r in zip(values, out):
        assert H.to_int(r) == (pow(v, -1, P) if v else 0), hex(v)


def test_split_constants(check, oracle):
    """beta and lambda are the endomorphism's: phi(G) = (beta x, y) = lambda G; and
    every split power is 2^(16 g) with both halves below 2^126, the bits summed."""
    lam = 0xB3C4D79D41A917585BFC41088D8DAAA78B17EA66B99C90DD
    out = check("constants", np.zeros(0))
    beta = H.to_int(out[-8:]) * pow(MONT, -1, P) % P
    assert beta != 1 and pow(beta, 3, P) == 1 and (lam * lam + lam + 1) % H.R == 0
    for x, y in H.load_g_bases()[:3]:
        assert oracle.affine_mul(x, y, lam) == (False, beta * x % P, y)
    rows = out[:-8].reshape(8, 10)
    for g, row in zip(range(8, 16), rows):
        a, b = H.to_int(row[:4]), H.to_int(row[4:8])
        assert a < 1 << 126 and b < 1 << 126
        assert ((-a if row[8] else a) + (-b if row[9] else b) * lam - (1 << (16 * g))) % H.R == 0
