"""The contraction's recombination, step by step in Python integers, with the
library's own constants (rkb_split_crt_weights): three digits, each reduced
modulo its product of moduli and added, times its weight, to a 72-bit fraction
of M."""
import ctypes

import numpy as np

DIGITS = 3


class Weights:
    def __init__(self, moduli):
        from atomx_b200 import _native
        moduli = np.ascontiguousarray(moduli, dtype=np.int32)
        n = len(moduli)
        end, coef, digit, weight = ((ctypes.c_int * m)() for m in (DIGITS, n, DIGITS, 4 * DIGITS))
        _native.check(_native.load().rkb_split_crt_weights(moduli.ctypes.data, n, end, coef, digit, weight),
                      "rkb_split_crt_weights")
        self.moduli = [int(m) for m in moduli]
        self.end, self.coef = list(end), list(coef)
        self.digit = [d & 0xffffffff for d in digit]
        self.weight = [weight[4 * g:4 * g + 4] for g in range(DIGITS)]

    def fraction(self, v) -> int:
        """x / M mod 1 in units of 2^-72, signed, from accumulators ``v`` (one
        integer of x's residue class per modulus)."""
        f = first = 0
        for end, D, (hi, mid, lo, tail) in zip(self.end, self.digit, self.weight):
            acc = sum(v[i] * self.coef[i] for i in range(first, end))
            assert abs(acc) < 1 << 59
            d = acc - (2 * acc + D) // (2 * D) * D       # nearest zero
            # units of 2^-96; d to 16 bits in the product with the weight's end
            end96 = (d >> 16) * tail + d * lo
            f += ((d * hi << 64) + (d * mid << 32) + end96 + (1 << 23)) >> 24
            first = end
        f &= (1 << 72) - 1
        return f - (1 << 72) if f >> 71 else f
