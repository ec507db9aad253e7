"""CPU checks of the sliced FP64 product's balanced digits (ozgemm_f64.cu): seven
base-256 digits per operand, exact in BF16, and the error of the 28 products
that are kept."""
import numpy as np
import pytest


def _balanced_digits(x, e):
    """The seven balanced base-256 digits of x against the scale 2^e (|x| < 2^e),
    as the device cuts them: +-round(|x| 2^(55-e)) plus 128 in the six low places,
    whose bytes less 128 are the low digits and whose top is the first."""
    m, q = np.frexp(abs(x))
    mant, sh = int(m * 2.0**53), int(q) - 53 - e + 55
    U = mant << sh if sh >= 0 else (0 if sh < -54 else (mant + (1 << (-sh - 1))) >> -sh)
    W = (-U if x < 0 else U) + 0x0000808080808080
    return [W >> 48] + [((W >> (8 * b)) & 255) - 128 for b in range(5, -1, -1)], U


@pytest.mark.parametrize("e", [0, 3, -40])
def test_balanced_digits(e):
    rng = np.random.default_rng(100 + e)
    xs = np.concatenate([rng.uniform(-1, 1, 500) * 2.0**e, rng.uniform(-1, 1, 300) * 2.0 ** (e - rng.integers(0, 60, 300)),
                         [0.0, np.nextafter(2.0**e, 0), -np.nextafter(2.0**e, 0), 2.0 ** (e - 1), -(2.0 ** (e - 56))]])
    for x in xs:
        a, U = _balanced_digits(float(x), e)
        assert all(-128 <= d <= 128 for d in a)  # exact in BF16, products of 256 at most 2^22
        v = sum(d * 256 ** (6 - s) for s, d in enumerate(a))
        assert v == (-U if x < 0 else U)
        assert abs(v * 2.0 ** (e - 55) - x) <= 2.0 ** (e - 56)
    # worst cases of the sums: four products exact in FP32
    assert 4 * 256 * 128 * 128 <= 1 << 24


def test_seven_slice_product_error():
    """Diagonals s + t <= 8 of the seven slices against the exact product: within
    2^-52 of the row and column scales (the dropped diagonals' random sum is
    sqrt(6 * 256) * 74^2 * 2^-70, about 2^-52.3, plus the cuts at 2^-56), and the
    64-bit integer that collects them stays below 2^63."""
    from fractions import Fraction

    rng = np.random.default_rng(5)
    K, worst = 256, 0.0
    for trial in range(40):
        a, b = rng.uniform(-1, 1, K), rng.uniform(-1, 1, K)
        da, db = [_balanced_digits(float(v), 0)[0] for v in a], [_balanced_digits(float(v), 0)[0] for v in b]
        P = {d: sum(x[s - 1] * y[d - s - 1] for x, y in zip(da, db) for s in range(max(1, d - 7), min(7, d - 1) + 1))
             for d in range(2, 9)}
        exact = sum(Fraction(float(x)) * Fraction(float(y)) for x, y in zip(a, b))
        got = sum(Fraction(p) * Fraction(2) ** (2 - 8 * d) for d, p in P.items())
        worst = max(worst, abs(float(got - exact)))
        assert abs(sum(p * 2.0 ** (56 - 8 * d) for d, p in P.items())) < 2.0**63
    assert worst < 4 * 2.0**-52


def _seven_slice_error(a, b):
    """|kept products - exact| of two vectors whose scales are 1, in exact arithmetic."""
    from fractions import Fraction

    da, db = [_balanced_digits(float(v), 0)[0] for v in a], [_balanced_digits(float(v), 0)[0] for v in b]
    got = sum(Fraction(sum(x[s - 1] * y[d - s - 1] for x, y in zip(da, db) for s in range(max(1, d - 7), min(7, d - 1) + 1)))
              * Fraction(2) ** (2 - 8 * d) for d in range(2, 9))
    return abs(float(got - sum(Fraction(float(x)) * Fraction(float(y)) for x, y in zip(a, b))))


@pytest.mark.parametrize("kind", ["constant", "one large", "254/255"])
def test_seven_slice_product_worst_case(kind):
    """Operands with a pattern: the dropped products are at most 6 256 128^2 2^-70 (d = 9) and
    1/300 of that beyond (d = 10 .. 14: 5, 4, .. products, each 2^-8 further down), the
    cuts 256 2^-55. All three are far above the few units of random operands."""
    K = 256
    if kind == "constant":
        a = np.full(K, 0.8)  # 0.1 against its own scale
    elif kind == "one large":
        a = np.full(K, float.fromhex("0x1.fdfdfdfdfdfcp-9"))
        a[0] = 0.75
    else:
        a = np.full(K, 254.0 / 255.0)
    err = _seven_slice_error(a, a)
    assert err <= 6 * K * 128**2 * 2.0**-70 * (1 + 1 / 300) + K * 2.0**-55
    assert err > 2.0**-47
