"""The digit cases of the INT8 exchange, on the CPU: their tolerance passes the eight
levels that are kept and tells apart what drops or mixes up a digit."""
import numpy as np

import i8_cases as I


def test_values_are_doubles_with_these_digits():
    for d in I.patterns(40, 1):
        v = I.value(d)
        assert int(float(v)) == v and abs(v) < 0.995 * 2**55 and abs(v) > 0.498 * 2**55


def test_tolerance_sees_a_missing_level_and_a_wrong_digit():
    pat = I.patterns(12, 2)
    for a in pat:
        for b in pat:
            exact = I.value(a) * I.value(b)
            assert I.relative_error(float(I.product(a, b, 8)), exact) <= I.PRODUCT_TOL
    exact = I.value(I.LARGEST) ** 2
    for levels in range(1, 8):
        assert I.relative_error(float(I.product(I.LARGEST, I.LARGEST, levels)), exact) > 2 * I.PRODUCT_TOL
    # one digit of an operand taken for another: seen with the random patterns
    for i in range(I.DIGITS):
        for j in range(i):
            worst = 0.0
            for a in pat:
                w = list(a)
                w[i], w[j] = w[j], w[i]
                worst = max([worst] + [I.relative_error(float(I.product(w, b, 8)), I.value(a) * I.value(b)) for b in pat])
            assert worst > 10 * I.PRODUCT_TOL
    assert np.isfinite(float(exact))
