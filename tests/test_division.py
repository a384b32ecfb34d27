"""The front end's division by its constants (the quotient with one step on its exact remainder)
against IEEE division, over every mantissa: both scale exactly with the dividend's exponent, so
that covers every dividend out of reach of overflow and underflow."""
import numpy as np
import pytest


def _round_to_f32(hi, lo):
    """RN32 of the exact sum hi + lo (float64, |lo| at most half an ulp of hi)."""
    f = hi.astype(np.float32)
    # where hi is a tie between two floats, the sign of lo decides
    other = np.nextafter(f, np.where(hi > f, np.float32(np.inf), np.float32(-np.inf)).astype(np.float32))
    tie = (hi != f) & (np.abs(hi - f.astype(np.float64)) == np.abs(hi - other.astype(np.float64)))
    up = np.maximum(f, other)
    down = np.minimum(f, other)
    return np.where(tie & (lo > 0), up, np.where(tie & (lo < 0), down, f))


# full-range maxima of 8- to 16-bit samples; luma and chroma spans (their scale is a power of
# two); the DCI reference white's normalisation
@pytest.mark.parametrize("d", [255, 511, 1023, 2047, 4095, 8191, 16383, 32767, 65535, 219, 224, 52.37])
def test_division_is_correctly_rounded(d):
    d = np.float32(d)
    r = np.float32(1) / d
    for part in range(8):
        a = (np.arange(part << 20, (part + 1) << 20, dtype=np.uint32) | np.uint32(0x3F800000)).view(np.float32)
        a64, d64, r64 = a.astype(np.float64), np.float64(d), np.float64(r)
        q = (a64 * r64).astype(np.float32)  # the product is exact in float64
        rem = (a64 - q.astype(np.float64) * d64)  # exact: 48 bits, then cancellation
        rem = rem.astype(np.float32).astype(np.float64)  # one rounding, as the fused operation
        p, q64 = rem * r64, q.astype(np.float64)
        s = q64 + p
        err = (q64 - s) + p  # |q| >= |p|: exact
        assert np.array_equal(_round_to_f32(s, err), a / d), part
