"""The two identities the append kernel rounds by, over every input they are used for, in exact integers or
IEEE fp32 (csrc/pack_append.cu: codes from an approximate quotient, scales from a product)."""
import numpy as np
import pytest

APPROX = 21        # the approximate quotient is within 2^-21 of the exact one (reciprocal and product, 2^-23 each)


def _rint(num, den):
    """num / den to the nearest integer, ties to even (positive int64)."""
    q, r = np.divmod(num, den)
    up = (2 * r > den) | ((2 * r == den) & (q & 1 == 1))
    return q + up


@pytest.mark.parametrize("sign", [1, -1])
def test_codes_from_an_approximate_quotient(sign):
    """Every pair of an 11-bit significand and an 8-bit one, every exponent between them that gives a quotient
    the codes reach: the approximate quotient, to a multiple of 2^-14 and then to an integer, is the exact one
    to an integer -- at both ends of what the approximation may return, so for everything between."""
    x = np.arange(1024, 2048, dtype=np.int64)[:, None]
    s = np.arange(128, 256, dtype=np.int64)[None, :]
    for e in range(-7, 4):                                            # quotient x / s * 2^(e - 2)
        num, den = (x << (e + 7), s << 9)
        exact = _rint(num, den)
        quotient = num / den
        use = (quotient > 0.2) & (quotient < 7.6)
        assert use.any() or e < -3 or e > 2
        scaled = (num << 14) * ((1 << APPROX) + sign)                 # < 2^(21 + 14 + 22)
        assert int(scaled.max()) < 1 << 62
        fine = _rint(scaled, den << APPROX)                           # multiples of 2^-14: the fma against 768
        assert np.array_equal(_rint(fine, np.int64(1 << 14))[use], exact[use])


def _bf16(x):
    """Bits of x (positive fp32) to bf16, ties to even."""
    u = x.view(np.uint32)
    return (u + 0x7FFF + ((u >> 16) & 1)) >> 16


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("qmax", [1, 3, 7])
def test_scales_from_a_product(dtype, qmax):
    """Every magnitude of the input type up to 2^125: bf16(fp32(amax / qmax)) is what the product with the rounded
    reciprocal gives, to 16 significant bits first where the quotient can be a tie (fp16, qmax > 1).  And the
    largest code is never above qmax."""
    bits = np.arange(0, 0x7C00 if dtype == "fp16" else 0x7E00, dtype=np.uint16)
    amax = bits.view(np.float16).astype(np.float32) if dtype == "fp16" else (bits.astype(np.uint32) << 16).view(np.float32)
    floor = np.float32(1e-8)
    want = _bf16(np.maximum(amax / np.float32(qmax), floor))
    y = amax * np.float32(1.0 / qmax)
    if dtype == "fp16" and qmax > 1:
        y = ((y.view(np.uint32) + np.uint32(0x80)) & np.uint32(0xFFFFFF00)).view(np.float32)
    assert np.array_equal(_bf16(np.maximum(y, floor)), want)
    scale = (want.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
    assert np.rint(amax / scale).max() <= qmax
