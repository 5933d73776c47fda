"""Operands whose seven INT8 digits are all chosen, and exact products of them.

An element of value v is sum_i d_i 256^(6 - i) with the leading digit in 64 .. 126, so
that it is itself its row's largest magnitude and these are the digits the library
makes of it.  Products of them are whole numbers, computed exactly."""
import numpy as np

DIGITS = 7
# unit roundings of a product: one of the levels' sum, and a tenth for the levels that
# are dropped (2^-59.7 of the product for the largest digits)
PRODUCT_TOL = 1.1 * 2.0**-53

# the largest coherent low digits: level 7 (i + j = 7) is then 3 x 2^-53 of the product
LARGEST = (64, 127, 127, 127, 127, 127, 124)


def patterns(count, seed):
    """LARGEST, its negative and random digits; the last one a multiple of 4, so that an
    FP64 number holds the value."""
    rng = np.random.default_rng(seed)
    out = [LARGEST, tuple(-d for d in LARGEST)]
    while len(out) < count:
        d = [int(rng.integers(64, 127))] + [int(v) for v in rng.integers(-128, 128, 5)] + [4 * int(rng.integers(-32, 32))]
        out.append(tuple(v * (1 if i else int(rng.choice([-1, 1]))) for i, v in enumerate(d)))
    return out


def value(digits):
    return sum(d * 256 ** (DIGITS - 1 - i) for i, d in enumerate(digits))


def product(a, b, levels):
    """a b from the digit products of the levels i + j < levels."""
    return sum(x * y * 256 ** (2 * DIGITS - 2 - i - j) for i, x in enumerate(a) for j, y in enumerate(b) if i + j < levels)


def relative_error(got, exact):
    """|got - exact| / |exact| of a double against a whole number."""
    return abs(int(got) - exact) / abs(exact)
