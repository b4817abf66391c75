"""CPU checks of the constants of the exponential that the FP64 pair loops run (exp_scaled,
bit_b200/csrc/fp64math.cuh), each recomputed here to 80 digits: the correction of 64 / ln 2 and the
Taylor coefficients with (ln 2 / 64)^k folded in."""
import math
import os
import re
from decimal import Decimal, getcontext

from test_fp64math import HDR


def test_constants_of_the_scaled_exponential():
    getcontext().prec = 80
    s = open(HDR).read()
    ln2 = Decimal(2).ln()
    hi = float(64 / ln2)
    lo = float.fromhex(re.search(r"kExpInvLlo = ([0-9a-fx.p+-]+);", s).group(1))
    assert lo == float(64 / ln2 - Decimal(hi))
    body = s[s.index("double exp_scaled("):]
    body = body[:body.index("p *= f;")]
    coef = [float.fromhex(c) for c in re.findall(r"0x1\.[0-9a-f]+p-\d+", body)]
    assert coef == [float((ln2 / 64) ** k / math.factorial(k)) for k in (5, 4, 3, 2, 1)]
