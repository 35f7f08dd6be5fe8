"""A CPU model of the two-digit residue form (csrc/ozaki.cu, scaled operands up to
2^30): the low word of v + 2^15 (1 + 2^16) gives balanced 16-bit digits b_0, b_1 with
v = b_0 + b_1 2^16, and s = b_0 + b_1 (2^16 mods m) is exact in FP32, below the 2^23
that the FP32 quotient needs, and congruent to v."""
import numpy as np
import pytest

MODULI = [255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193]


@pytest.mark.parametrize("m", MODULI)
def test_two_digits(m):
    rng = np.random.default_rng(m)
    top = 1 << 30
    v = np.concatenate([np.arange(-3, 4), [top, -top, top - 1, 1 - top, 32767, 32768, -32768, -32769],
                        rng.integers(-top, top + 1, 200000)])
    w = v + 32768 * 65537
    assert w.min() >= 0 and w.max() < 1 << 32
    b0, b1 = (w & 0xffff) - 32768, (w >> 16) - 32768
    assert np.array_equal(b0 + (b1 << 16), v)
    assert np.array_equal(w & 0xff, v & 0xff)  # modulus 256: the low byte is v's
    c = 65536 % m
    c = c - m if c > (m - 1) // 2 else c
    s = b0 + b1 * c
    assert np.abs(b1 * c).max() < 1 << 24 and np.abs(s).max() < 1 << 23
    assert not ((s - v) % m).any()
