"""A CPU model of the split DGEMM's reconstruction (the `reconstruct` kernel in
csrc/ozaki.cu): the residues of an integer |C'| <= M/8 go by pairs of moduli into
t_p = c r + c' r', and C' = sum_p t_p W_p - q M with W_p = M / (m m') and M split at
2^T1 and 2^T2.  Checked with exact rational arithmetic for each FP64 operation: t_p
fits 24 bits, the sums of the upper two parts are exact, q is the exact quotient, and
C' comes back within one rounding of itself plus 2^-80 of the range M/8."""
import math
import random
from fractions import Fraction

import pytest

MODULI = [256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193]


def rnd(x):
    return float(x)  # Fraction.__float__ rounds correctly


def fma(a, b, c):
    return rnd(Fraction(a) * Fraction(b) + Fraction(c))


def plan(nmod):
    mods = MODULI[:nmod]
    M = math.prod(mods)
    pairs = [(mods[l], mods[l + 1] if l + 1 < nmod else 1) for l in range(0, nmod, 2)]
    T1 = max(0, max((M // (m * n)).bit_length() for m, n in pairs) - 26)
    T2 = max(0, T1 - 26)

    def coef(m, other, mod):
        v = other * pow(M // m, -1, m) % mod
        return v - mod if 2 * v > mod else v

    def parts(v):
        return float(v >> T1), float((v >> T2) & ((1 << (T1 - T2)) - 1)), rnd(v & ((1 << T2) - 1))

    return dict(M=M, mods=mods, T1=T1, T2=T2, Mp=parts(M),
                c=[(coef(m, n, m * n), coef(n, m, m * n) if n > 1 else 0) for m, n in pairs],
                W=[parts(M // (m * n)) for m, n in pairs], pairs=pairs,
                t_x=rnd(Fraction(2 ** T1, 1) / Fraction(rnd(M))))


@pytest.mark.parametrize("nmod", range(2, 17))
def test_pairs_return_the_integer(nmod):
    p = plan(nmod)
    M = p["M"]
    rng = random.Random(nmod)
    top = M // 8
    cs = [0, 1, -1, top, -top, top - 1, 1 - top, M // 256, -(M // 255)]
    cs += [rng.randint(-top, top) for _ in range(150)]
    cs += [rng.choice([-1, 1]) * rng.getrandbits(rng.randint(1, max(1, M.bit_length() - 4)))
           for _ in range(150)]
    for C in cs:
        r = [(C + m // 2) % m - m // 2 for m in p["mods"]] + [0]
        t = [a * r[2 * i] + b * r[2 * i + 1] for i, (a, b) in enumerate(p["c"])]
        assert all(abs(a) < 1 << 15 and abs(b) < 1 << 15 for a, b in p["c"])
        assert all(abs(v) < 1 << 23 for v in t)
        full = sum(v * (M // (m * n)) for v, (m, n) in zip(t, p["pairs"]))
        assert (full - C) % M == 0
        X = []
        for k in range(3):
            x, exact = 0.0, 0
            for v, w in zip(t, p["W"]):
                x = fma(v, w[k], x)
                exact += v * int(w[k])
            if k < 2:
                assert int(x) == exact and abs(exact) <= 1 << 52
            X.append(x)
        q = round(Fraction(rnd(Fraction(X[0]) * Fraction(p["t_x"]))))
        assert q == (full - C) // M
        h = [fma(-q, mp, x) for mp, x in zip(p["Mp"], X)]
        assert int(h[0]) == int(X[0]) - q * int(p["Mp"][0])
        assert int(h[1]) == int(X[1]) - q * int(p["Mp"][1])
        k = float(round(Fraction(h[1]) / 2 ** (p["T1"] - p["T2"])))
        h[0], h[1] = h[0] + k, fma(-k, 2.0 ** (p["T1"] - p["T2"]), h[1])
        got = fma(h[0], 2.0 ** p["T1"], fma(h[1], 2.0 ** p["T2"], h[2]))
        err = abs(Fraction(got) - C)
        assert err <= Fraction(abs(C)) / 2 ** 53 + Fraction(M, 8) / 2 ** 80
        if M.bit_length() < 100 and abs(C) < 1 << 52:
            assert got == C
