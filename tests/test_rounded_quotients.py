"""The claim of fn_rounded.cuh that a quotient may use, in the place of a
correctly rounded reciprocal, the double on the other side of the middle next
to it: the sequence in exact rational arithmetic, over the mantissas whose
reciprocals lie closest to a middle and their quotients next to a middle."""
import math
from fractions import Fraction

import numpy as np

import test_gpu_rounded as rounded


def nearest(x):
    return Fraction(float(x))  # correctly rounded


def test_quotient_from_the_neighbour_of_a_reciprocal():
    hard = [int(b) for b in np.ldexp(rounded.hard_reciprocals(), 52)]
    tried = 0
    for m in hard:
        b = Fraction(m, 1 << 52)
        up = nearest(1 / b)
        down = Fraction(math.nextafter(float(up), 0.0))
        middle = (up + down) / 2
        near = abs(1 / b - middle) * b * (1 << 106) <= 16
        for y in (up, down) if near and m != (1 << 53) - 1 else (up,):
            for k in range(-15, 16, 2):
                for n in rounded.numerators(m, k):
                    a = Fraction(n, 1 << 52)
                    q = nearest(a * y)
                    assert nearest(q + y * nearest(a - b * q)) == nearest(a / b), (hex(m), hex(n))
                    tried += y == down
    assert tried > 0
