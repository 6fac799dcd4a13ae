"""The residue form's arithmetic (momms_gb300/csrc/crt_elem.cuh), compiled for the host, against
Python integers: residues of scaled elements for every slice count and modulus, and the
reconstruction of the product's integer and its one rounding."""
import math
import os
import random
import re
import struct
import subprocess
from fractions import Fraction

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "momms_gb300", "csrc")
SRC = os.path.join(ROOT, "tests", "cpp", "test_crt_elem.cpp")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("crt") / "crt_elem")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, SRC, "-o", out], check=True, capture_output=True, text=True)
    return out


def _moduli():
    text = open(os.path.join(CSRC, "crt_elem.cuh")).read()
    return [int(x) for x in re.search(r"kModuli\[kMaxModuli\] = \{([^}]*)\}", text).group(1).split(",")]


def _run(exe, lines):
    r = subprocess.run([exe], input="\n".join(lines) + "\n", capture_output=True, text=True, check=True)
    return r.stdout.split("\n")


def _bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def test_moduli_pairwise_coprime_and_fit():
    p = _moduli()
    assert len(p) == 36 and max(p) == 256
    assert all(math.gcd(a, b) == 1 for i, a in enumerate(p) for b in p[:i])
    # the most slices over the longest k fit
    assert math.prod(p) > 2 * 32704 * 2 ** (16 * 15) * 1.03


@pytest.mark.parametrize("ns", range(5, 16))
def test_residues(exe, ns):
    rng = random.Random(ns)
    values = [0.0, 0.5, 1 - 2.0**-53, -(1 - 2.0**-53), 2.0**-40, -(2.0**-60), 2.0**-1074, 2.0 ** (-8 * ns - 1)]
    for _ in range(400):
        mant = rng.choice([rng.getrandbits(53), 2**53 - 1, rng.getrandbits(53) | (2**14 - 1) << rng.randrange(0, 40)])
        values.append(rng.choice([-1, 1]) * math.ldexp(min(mant, 2**53 - 1), -53 - rng.choice([0, 0, 1, 7, 30, 61])))
    out = _run(exe, [f"0 {ns} 0 {_bits(v)}" for v in values])
    for v, line in zip(values, out):
        x = math.floor(abs(Fraction(v)) * 2 ** (8 * ns) + Fraction(1, 2))
        x = -x if v < 0 else x
        got = [int(t) for t in line.split()]
        for r, p in zip(got, _moduli()):
            assert abs(r) <= 128 and (r - x) % p == 0, (v, p, r)


@pytest.mark.parametrize("ns", range(5, 16))
def test_reconstruction(exe, ns):
    rng = random.Random(100 + ns)
    p = _moduli()
    lines, want = [], []
    for _ in range(300):
        k = rng.choice([128, 1000, 8192, 32704])
        n = next(i for i in range(1, 37) if sum(math.log2(x) for x in p[:i]) >= 16 * ns + math.log2(k) + 1 + 0.03)
        most = k * 2 ** (16 * ns)
        R = rng.choice([0, 1, -1, most, -most, rng.randint(-most, most), rng.getrandbits(rng.randrange(1, 16 * ns)),
                        -(rng.getrandbits(60) << rng.randrange(0, 16 * ns - 60))])
        if rng.random() < 0.3 and abs(R) > 2**60:  # a tie at the rounding position
            t = abs(R).bit_length() - 53
            R = (abs(R) >> t << t | 1 << (t - 1)) * (1 if R > 0 else -1)
        scale = rng.choice([-16 * ns, -16 * ns - 1000, -1074])
        # a byte holds the symmetric residue plus 128, modulo 256
        r = [((x + 128) if 2 * x <= q else (x - q + 128)) % 256 for q in p[:n] for x in [R % q]]
        lines.append(f"1 {ns} {n} {scale} " + " ".join(map(str, r)))
        want.append(_bits(float(Fraction(R) * Fraction(2) ** scale)))
    assert [int(x) for x in _run(exe, lines)[: len(want)]] == want
