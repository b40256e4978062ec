"""The two-term reciprocal that replaces the FP64 sweeps' division
(csrc/bfb_recip.h): every divisor it accepts gives IEEE division's quotient,
and its search for the numerators that could round wrongly is complete (on
short mantissas, where all numerators can be tried)."""
from __future__ import annotations

import subprocess
from fractions import Fraction
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    exe = tmp_path_factory.mktemp("recip") / "recip_check"
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O2", "-Wall", "-ffp-contract=off",
                    f"-I{ROOT / 'biofvm-b_b200' / 'csrc'}", "-o", str(exe), str(ROOT / "tests" / "recip_check.cpp")],
                   check=True)
    return exe


def test_accepted_divisors_divide_exactly(driver):
    r = subprocess.run([str(driver), "3000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    accepted, refused, bad = map(int, r.stdout.split())
    assert bad == 0
    assert accepted + refused == 3000 and refused <= 30


@pytest.mark.parametrize("Y", [513, 769, 1023, 514, 516, 1000, 1022])
def test_search_for_hard_numerators_is_complete(Y):
    """The header's congruence with 10-bit mantissas in place of 53-bit ones:
    its solutions are exactly the numerators within the window of a midpoint."""
    p, window = 10, 4
    want = set()
    for X in range(2 ** (p - 1), 2**p):
        k = p if X >= Y else p + 1
        q = Fraction(X * 2**k, Y)
        M = q.numerator // q.denominator
        for odd in (M | 1, (M | 1) - 2, (M | 1) + 2):
            if abs(X * 2**k - odd * Y) <= window:
                want.add(X)
    got = set()
    s, Yo = 0, Y
    while Yo % 2 == 0:
        Yo //= 2
        s += 1
    for k in (p, p + 1):
        inv = pow(pow(2, k, Yo), -1, Yo) if Yo > 1 else 0
        for r in range(-window, window + 1):
            if r == 0 or r % (1 << s):
                continue
            x = r * inv % Yo
            got |= {X for X in range(x, 2**p, Yo) if X >= 2 ** (p - 1) and (k == p) == (X >= Y)}
    assert want <= got
