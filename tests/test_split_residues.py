"""The residue bytes of the int8 products' epilogue, restated in numpy: the single-
precision quotient gives r = v - q p as a signed byte congruent to the accumulator v for
every modulus, at the largest |v| a K chunk allows and next to the half-multiples of p
where the quotient rounds, directly while p / 2 + |v| 2^-23 < 128 and after folding
v to (v mod 2^16) + floor(v / 2^16) (2^16 mod p) beyond."""
import numpy as np
import pytest

MODULI = [256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193]


def fma32(f, inv, c):
    """fma in float32: the double product and sum of these operands are exact."""
    return (f.astype(np.float64) * float(inv) + c).astype(np.float32)


def residue_byte(v, p, mode):
    if mode == "mask":
        return v.astype(np.int64)
    if mode == "fold":
        c16 = 65536 % p
        c16 = c16 - p if c16 > p // 2 else c16
        v = (v & 0xFFFF) + (v >> 16) * c16
        assert np.max(np.abs(v)) < 2 ** 21.1
    bits = fma32(v.astype(np.float32), np.float32(1.0) / np.float32(p), 12582912.0)
    q = bits.view(np.int32).astype(np.int64)
    return v - q * p


@pytest.mark.parametrize("k", [1, 128, 260, 900, 1536, 2048, 8192, 65536])
def test_residue_bytes(k):
    rng = np.random.default_rng(k)
    for p in MODULI:
        h = p // 2
        vmax = k * h * h
        assert vmax <= 2 ** 30
        half = rng.integers(-vmax // p - 1, vmax // p + 1, 20000) * p + h
        v = np.concatenate([rng.integers(-vmax, vmax + 1, 20000), half, half + 1, half - 1,
                            [vmax, -vmax, 0, 1, -1]])
        v = np.clip(v, -vmax, vmax).astype(np.int64)
        mode = "mask" if p == 256 else "fast" if 0.5 * p + vmax * 2.0 ** -23 < 127.99 else "fold"
        r = residue_byte(v, p, mode)
        stored = (r + 128) & 0xFF  # the byte kept, 128 more than the residue
        assert np.all((stored - 128 - v) % p == 0)
        if p != 256:
            off = r & 0xFF
            signed = np.where(off > 127, off - 256, off)
            assert np.array_equal(signed, stored - 128) and np.all(np.abs(signed) <= 128)
