"""The residue GEMM at the edge of its exactness: every FP32 accumulator holds integers, whatever
the operands, because a chunk of 384 products of balanced residues stays below 2^24.  Nothing
checks that at run time, so operand rows are made here whose residues for one modulus are all
as large as they get."""
import os
import re
import shutil
import struct
import subprocess
from math import prod

import numpy as np
import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "gain-mpi_gb300", "csrc")
MODULI = [int(x) for x in re.search(r"kModuli\[kMaxMod\] = \{([^}]*)\}", open(os.path.join(CSRC, "residue.h")).read())
          .group(1).split(",")]


def edge_rows(nmod, bits, K, side, rng):
    """Rows of integers T (exact in FP64, of the row scale that makes the plane's integer X = T 2^s)
    whose residues modulo m_i are all +-(m_i - 1) / 2, one row per modulus and sign.  side 1: as
    operand B, whose residues carry the factor (M / m_i)^-1."""
    tbits = min(bits, 53)
    s = bits - tbits
    rows = []
    for m in MODULI[:nmod]:
        if s and m % 2 == 0:
            continue                      # 2^s has no inverse
        for sign in (1, -1):
            r = sign * ((m - 1) // 2)
            if side:
                r = r * (prod(MODULI[:nmod]) // m)
            r = r * pow(pow(2, s, m), -1, m) % m
            t = rng.integers((1 << (tbits - 1)) // m + 1, (1 << tbits) // m - 1, K) * m + r
            assert t.max() < 1 << tbits and t.min() >= 1 << (tbits - 1)
            rows.append(t)
    return np.array(rows, dtype=np.int64)


def nmod_of(bits, K):
    """The fewest moduli whose product exceeds 2 K 2^(2 bits)."""
    return next(n for n in range(1, len(MODULI) + 1) if prod(MODULI[:n]) > (2 * K) << (2 * bits))


@pytest.mark.parametrize("bits", [48, 56])
def test_edge_rows_fill_the_accumulator(bits):
    """The rows do what they are made for: the largest chunk sum of a modulus is within 2 % of 2^24."""
    n = nmod_of(bits, 384)
    rng = np.random.default_rng(bits)
    A, B = edge_rows(n, bits, 384, 0, rng), edge_rows(n, bits, 384, 1, rng)
    s = bits - min(bits, 53)
    most = 0
    for m in MODULI[:n]:
        f = pow(prod(MODULI[:n]) // m, -1, m)
        ra = np.array([(int(t) << s) % m for t in A.ravel()]).reshape(A.shape)
        rb = np.array([(int(t) << s) * f % m for t in B.ravel()]).reshape(B.shape)
        ra, rb = np.where(2 * ra > m, ra - m, ra), np.where(2 * rb > m, rb - m, rb)
        most = max(most, int(np.abs(ra @ rb.T).max()) + m // 2)
    assert 0.98 * 2 ** 24 < most < 2 ** 24


@pytest.fixture(scope="module")
def driver(built_lib, tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = str(tmp_path_factory.mktemp("drv") / "residue_driver")
    lib = os.path.join(ROOT, "gain-mpi_gb300", "lib")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-I", CSRC, os.path.join(ROOT, "tests", "cpp", "residue_driver.cpp"),
                    "-o", out, "-L", lib, "-lgainls", "-Xlinker", "-rpath", "-Xlinker", lib], check=True)
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("pair", [0, 1])
@pytest.mark.parametrize("bits,K", [(48, 384), (48, 400), (48, 1152), (56, 384), (56, 1152)])
def test_products_of_edge_rows_are_exact(driver, tmp_path, bits, K, pair):
    """One, two and three chunks, the second partly zeros: every product of two edge rows against the
    exact integer sum.  A single wrong residue moves an output by about M / m_i, the whole range;
    what is allowed is the rounding of the result and the reconstruction's own bound."""
    kpad = -(-K // 64) * 64
    n = nmod_of(bits, kpad)
    rng = np.random.default_rng(K + bits)
    A, B = edge_rows(n, bits, K, 0, rng), edge_rows(n, bits, K, 1, rng)
    at = np.arange(256) % len(A)
    with open(tmp_path / "in", "wb") as f:
        f.write(struct.pack("<4i", 256, K, bits, pair))
        f.write(A[at].astype(np.float64).tobytes())
        f.write(B[at].astype(np.float64).tobytes())
    subprocess.run([driver, str(tmp_path / "in"), str(tmp_path / "out")], check=True, timeout=120)
    raw = (tmp_path / "out").read_bytes()
    assert struct.unpack("<2i", raw[:8]) == (n, 0)
    got = np.frombuffer(raw[8:], np.float64).reshape(256, 256)
    s = bits - min(bits, 53)
    # reconstruction: M 2^-80 sum m_i in units of X Y, here of T T'
    fix = prod(MODULI[:n]) * 2.0 ** -80 * sum(MODULI[:n]) * 1.02 * 2.0 ** (-2 * s)
    for i, a in enumerate(A):
        for j, b in enumerate(B):
            exact = sum(int(x) * int(y) for x, y in zip(a, b))
            out = got[np.ix_(at == i, at == j)]
            assert np.all(out == out[0, 0])
            assert abs(int(out[0, 0]) - exact) <= exact * 2.0 ** -53 * 1.01 + fix, (i, j)
