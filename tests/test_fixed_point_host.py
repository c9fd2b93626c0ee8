"""The fixed-point headers of the element kernels, compiled for the host, against 128-bit arithmetic
(tests/cpp/*_fixed_point.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ULP = 2.0 ** -53


def run(name, tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no C++ compiler")
    probe = subprocess.run(["g++", "-std=gnu++17", "-fsyntax-only", "-x", "c++", "-"], input="__float128 x = 0;",
                           text=True, capture_output=True)
    if probe.returncode:
        pytest.skip("no 128-bit floating point in this compiler")
    exe = str(tmp_path / name)
    subprocess.check_call(["g++", "-O2", "-std=gnu++17", "-ffp-contract=off", "-I",
                           os.path.join(ROOT, "proxpde_gb300", "csrc"), os.path.join(ROOT, "tests", "cpp", name + ".cpp"),
                           "-o", exe])
    return [line.split() for line in subprocess.check_output([exe], text=True, timeout=300).splitlines()]


def test_tetrahedra(tmp_path):
    lines = run("tet_fixed_point", tmp_path)
    assert len(lines) == 2 + 6 * 4
    for name, eps, taken, refused, det, gram, det64, gram64 in lines:
        taken, refused, det, gram, det64, gram64 = int(taken), int(refused), *map(float, (det, gram, det64, gram64))
        # ordinary elements are taken
        if name in ("kuhn", "scaled") or eps == "1":
            assert refused <= 0.02 * (taken + refused), name
        if not taken:
            continue
        # |det J|: the cofactors' truncation (3 x 2^-60) and the normalised sum's, at most 2^5 smaller than its
        # terms (2^-53 in all), the rounded edges of an inexact element (3 x 2^-61 over 2^-8: 1.5 ulp), the
        # conversion (1).  Gram: two cofactors (truncation, rounded edges over 2^-8: 1.5 ulp each), the products'
        # and the quotient's units (1 ulp each), the determinant's 3.5, the conversion
        assert det <= 3.5 * ULP, (name, eps)
        assert gram <= 9.5 * ULP, (name, eps)
        # and no further off than the plain FP64 formulas, up to the last rounding
        assert det <= det64 + 2 * ULP and gram <= gram64 + 2 * ULP, (name, eps)


def test_hexahedra(tmp_path):
    lines = run("hex_fixed_point", tmp_path)
    assert len(lines) == 1 + 6 * 5
    for name, eps, taken, refused, k, m, k64, m64 in lines:
        taken, refused, k, m, k64, m64 = int(taken), int(refused), *map(float, (k, m, k64, m64))
        assert refused <= 0.02 * (taken + refused), (name, eps)
        # nowhere further off than the FP64 form with the Gram determinant, up to the last rounding
        assert not k > k64 + ULP and not m > m64 + ULP, (name, eps)
        # in ordinary elements within a few roundings: a dozen steps of 2^-60 of the largest value each, which is
        # at most 2^5 times an entry's bound, and the conversion
        if name in ("cube", "small"):
            assert k <= 4 * ULP and m <= 3 * ULP, (name, eps)
