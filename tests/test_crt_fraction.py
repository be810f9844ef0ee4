"""The contraction's CRT constants and the bits its recombination keeps.

With the library's constants the digits are exact, and the fraction x / M of
every integer below M / 2 is off by at most three roundings to 2^-72 and three
products cut at 2^-81: below 2^-71, and below the 2^-70 of the recombination
in doubles (weights split at 2^-34, low parts summed in double).
"""
import math
import random
from fractions import Fraction

import pytest

from crt_fraction import Weights


@pytest.mark.parametrize("n_mod", range(4, 13))
def test_fraction_of_every_size(n_mod):
    from atomx_b200.split_plan import crt_constants
    w = Weights(crt_constants(n_mod)[0])
    M, rng = math.prod(w.moduli), random.Random(n_mod)
    # the digits: coefficients are 1 for their modulus and 0 for the digit's others
    first = 0
    for end, D in zip(w.end, w.digit):
        assert D == math.prod(w.moduli[first:end]) < 1 << 32
        for i in range(first, end):
            assert abs(2 * w.coef[i]) <= D
            assert all(w.coef[i] % m == (1 % m if j == i else 0) for j, m in enumerate(w.moduli) if first <= j < end)
        first = end
    assert first == n_mod
    top = 3456 * 128 * 128                       # an accumulator's largest magnitude
    worst = Fraction(0)
    for bits in range(0, M.bit_length()):
        for _ in range(40):
            x = rng.randrange(min(1 << bits, M // 2)) * rng.choice((-1, 1))
            v = [x % m + m * rng.randrange(-top // m + 1, top // m) for m in w.moduli]
            err = abs(Fraction(w.fraction(v), 1 << 72) - Fraction(x, M))
            worst = max(worst, min(err, 1 - err))
    assert worst <= Fraction(3, 1 << 73) + Fraction(3, 1 << 81) < Fraction(1, 1 << 70)


def _contract(moduli, M):
    """Status of a contraction call that is refused before it looks at a device."""
    import ctypes

    import numpy as np
    from atomx_b200 import _native
    ms, some = np.ascontiguousarray(moduli, dtype=np.int32), 256
    return _native.load().rkb_split_contract_z(
        some, 0, 128, 128, 128, len(ms), ms.ctypes.data_as(ctypes.c_void_p), float(M), some, some, some, some, 0.0, 9,
        10, some, some, some, 0, some, some, 1, some, some, 0)


@pytest.mark.parametrize("moduli,scale", [
    ((256, 255, 254, 251), 1.0),       # 256 and 254
    ((256, 255, 253, 251, 51), 1.0),   # 255 and 51, in different digits
    ((13, 13, 17, 19), 1.0),
    ((256, 255, 253, 251), 1.0 + 1e-12),
    ((256, 255, 253, 251), 0.5),
    ((256, 255, 253, 251), float("nan")),
])
def test_wrong_moduli_or_product_is_refused(moduli, scale):
    import math

    from atomx_b200 import _native
    assert _contract(moduli, math.prod(moduli) * scale) == 1
    assert b"moduli" in _native.load().rkb_last_error()
    if scale == 1.0:
        with pytest.raises(ValueError):
            Weights(moduli)
