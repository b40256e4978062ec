"""The two-term reciprocal (csrc/bfb_recip.h) where it could go wrong: every
divisor meets the numerators whose quotients lie next to the midpoint of two
doubles, listed here from the congruence X 2^k = r (mod b) with Python's
integers, and the header's own search is compared with all numerators of short
mantissas."""
from __future__ import annotations

import math
import random
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    exe = tmp_path_factory.mktemp("recip") / "recip_hard"
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O2", "-Wall", "-ffp-contract=off",
                    f"-I{ROOT / 'biofvm-b_b200' / 'csrc'}", "-o", str(exe), str(ROOT / "tests" / "recip_hard.cpp")],
                   check=True)
    return exe


def hard_numerators(Y, window=16):
    """53-bit X with X 2^k = r (mod Y), 0 < |r| <= window, k = 53 for X >= Y and 54 below."""
    s = (Y & -Y).bit_length() - 1
    Yo, out = Y >> s, []
    for k in (53, 54):
        inv = pow(2, -k, Yo) if Yo > 1 else 0
        for r in range(-window, window + 1):
            if r and r % (1 << s) == 0:
                x = r * inv % Yo
                first = x + -(-((1 << 52) - x) // Yo) * Yo if x < 1 << 52 else x
                out += [X for X in range(first, 1 << 53, Yo) if (k == 53) == (X >= Y)]
    return out


def test_divisors_on_their_hardest_numerators(driver):
    """3000 divisors of the Thomas factors' range: accepted ones divide exactly, refused ones have
    no low term that does. Among them are divisors for which the nearest low term fails, and
    refused ones, so a proof that is skipped or a low term that is a little off is noticed."""
    rng = random.Random(7)
    lines = []
    for _ in range(3000):
        b = 1.0 + math.exp(math.log(1e-4) + rng.random() * math.log(1e8)) * (1.0 + rng.random())
        X = hard_numerators(int(math.frexp(b)[0] * 2**53))
        lines.append(f"{b.hex()} {len(X)} " + " ".join(map(str, X)))
    r = subprocess.run([str(driver), "divide"], input="\n".join(lines), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    rows = [tuple(map(int, ln.split())) for ln in r.stdout.splitlines()]
    assert len(rows) == 3000
    accepted = [q for q in rows if q[0]]
    refused = [q for q in rows if not q[0]]
    assert all(wrong == 0 for _, wrong, _, _ in accepted)
    assert refused and all(least > 0 for _, _, _, least in refused)
    assert any(nearest > 0 for _, _, nearest, _ in accepted)
    assert len(refused) <= 30


@pytest.mark.parametrize("P", [10, 12])
def test_search_visits_exactly_the_hard_numerators(driver, P):
    """All P-bit mantissas and residues to 4: the header's search against every numerator."""
    r = subprocess.run([str(driver), "search", str(P)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    rows = {int(f[0]): set(map(int, f[1:])) for f in (ln.split() for ln in r.stdout.splitlines())}
    assert set(rows) == set(range(1 << (P - 1), 1 << P))
    for Y, got in rows.items():
        want = set()
        for X in range(1 << (P - 1), 1 << P):
            rem = X * 2 ** (P if X >= Y else P + 1) % Y
            if 0 < min(rem, Y - rem) <= 4:
                want.add(X)
        assert got == want, Y


def test_equal_axes_are_proven_once(driver):
    """An axis tries only the divisors that the axis before has not: none on an equal one, a last
    row (3 substrates) on a shorter one, the rows beyond on a longer one; the results are those
    of a proof on its own."""
    r = subprocess.run([str(driver), "axes", "40", "40", "25", "90"], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    rows = [tuple(map(int, ln.split())) for ln in r.stdout.splitlines()]
    assert all(same for _, _, same in rows)
    assert [shared for _, shared, _ in rows] == [3 * 39, 0, 3, 3 * (89 - 23)]
