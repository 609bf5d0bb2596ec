"""The backprojector's division by a launch constant (Markstein's remainder correction with the
rounded reciprocal): every 24-bit fraction of x against the FP32 division, for the constants that
scans have (distances, spacings, radians per view) and divisors near both ends of a binade.  The
kernel's two FMAs are evaluated in FP64, where they are exact before the final rounding."""
import numpy as np
import pytest

DIVISORS = [570.0, 595.0, 0.6, 1.0, 0.5, 0.97, 2 * np.pi / 1152, 2 * np.pi / 1160, 2 * np.pi / 120,
            1.0 + 2.0 ** -23, 1.0 + 2.0 ** -22, 2.0 - 2.0 ** -22, 1.3333334, 1.9999995]


@pytest.mark.parametrize("d", DIVISORS)
def test_division_by_a_constant_is_correctly_rounded(d):
    f = np.float32
    x = (np.arange(1 << 23, 1 << 24, dtype=np.float64) / 2 ** 23).astype(f)
    d = f(d)
    r = f(1) / d
    q = x * r
    rem = (x.astype(np.float64) - q.astype(np.float64) * float(d)).astype(f)
    got = (rem.astype(np.float64) * float(r) + q.astype(np.float64)).astype(f)
    assert np.array_equal(got, x / d)
