"""GPU test of the FP64 reciprocal root and quotient that the pair sums use, against
80-bit long doubles.

Bounds, in units of 2^-53: the root takes its residual e exactly but for one rounding
of e itself, leaves 5 e^3 / 16 out (0.16 for an estimate good to 2^-19) and rounds
once, 1.2 with room for e's own rounding; the quotient rounds n y and the sum, 2, and
leaves e^3 out, 2.1.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble


def _operands(kind):
    rng = np.random.default_rng(7)
    if kind == "powers":  # the neighbours of every power of two, odd and even
        k = np.arange(-1021, 1023)
        return np.concatenate([np.ldexp(1.0 + j * 2.0 ** -52, k) for j in range(5)]
                              + [np.ldexp(2.0 - j * 2.0 ** -52, k) for j in range(1, 6)])
    if kind == "octaves":  # mantissas over two octaves, where the estimates' errors repeat
        return np.concatenate([np.linspace(1.0, 4.0, 2_000_001)[:-1],
                               rng.uniform(1.0, 4.0, 2_000_000)])
    return np.ldexp(rng.uniform(1.0, 2.0, 2_000_000), rng.integers(-1021, 1023, 2_000_000))


@pytest.mark.parametrize("kind", ["powers", "octaves", "range"])
def test_helpers_against_long_doubles(kind):
    from qvort_b200 import lib as L

    a = _operands(kind)
    rng = np.random.default_rng(8)
    # a numerator whose quotient is a normal number
    k = np.frexp(a)[1]
    b = np.ldexp(rng.uniform(1.0, 2.0, len(a)), np.clip(k + rng.integers(-300, 300, len(a)), -700, 1000))
    ok = (np.abs(np.frexp(b)[1] - k) < 1000) & (np.abs(k) < 1000)
    r, q = L.test_f64(a, b)
    er = np.abs(r.astype(LD) * np.sqrt(a.astype(LD)) - 1)
    eq = np.abs(q.astype(LD) * a.astype(LD) / b.astype(LD) - 1)[ok]
    print(kind, "root", float(er.max()) * 2.0 ** 53, "quotient", float(eq.max()) * 2.0 ** 53)
    assert er.max() <= 1.2 * 2.0 ** -53
    assert eq.max() <= 2.1 * 2.0 ** -53
