"""CPU model of the INT8 GEMM's epilogue: the symmetric residue of an exact INT32
sum a (|a| <= 2^30) modulo each of the moduli, from q = (a mul + 2^37) >> 38 with
mul = rint(2^38 / m), is the one of exact integer arithmetic."""
import numpy as np

MODULI = [256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193]


def test_epilogue_quotient_is_exact():
    rng = np.random.default_rng(5)
    top = 1 << 30
    for m in MODULI:
        mul = ((2 << 38) // m + 1) // 2
        assert abs(mul * m - (1 << 38)) * 2 <= m and mul < 1 << 31
        j = np.concatenate([np.arange(-top // m, -top // m + 3000), np.arange(-3000, 3000),
                            np.arange(top // m - 3000, top // m + 1),
                            rng.integers(-top // m, top // m, 100000)])
        # the values nearest to half-integer quotients, and around whole ones
        a = np.concatenate([j * m + d for d in (-1, 0, 1, m // 2 - 1, m // 2, m // 2 + 1)])
        a = a[np.abs(a) <= top].astype(np.int64)
        a = np.concatenate([a, [-top, top], rng.integers(-top, top + 1, 100000)])
        q = (a * mul + (1 << 37)) >> 38
        r = a - q * m
        lo, hi = -(m >> 1), (m - 1) >> 1
        assert r.min() >= lo and r.max() <= hi
        assert np.array_equal((r - a) % m, np.zeros_like(a))
