"""Row sums of 16-warp groups whose 1024 partial sums lie at the top of one
binade: the fixed-point total passes 2^63 and must come out rounded, with its
sign, as the sum does in exact arithmetic.
"""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M, LEN = 8, 1024  # rows on columns of their own: one level, one step per row


@pytest.mark.parametrize("flow", ["0", "1"])
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("last", [0, 1, 3])
def test_sums_past_64_bits(fair, monkeypatch, flow, sign, last):
    """Partial sums of 1 - 2^-20 (and one with lower bits set) and b = -1/2: the
    total is an integer of 64 bits and more. With relaxation 1 and ones in the
    row, x' = x + (b - sum) / 1024; the coefficient is exact to 2^-53 of itself
    and x' to another rounding."""
    monkeypatch.setenv("FAIR_SWEEP_FLOW", flow)
    IA = LEN * np.arange(M + 1)
    JA = np.arange(M * LEN, dtype=np.int32) + 1
    A = fair.CSRMatrix.construct(M, M * LEN, np.ones(M * LEN), IA, JA)
    x0 = np.full(M * LEN, sign * (1.0 - 2.0 ** -20))
    x0[5::LEN] += sign * last * 2.0 ** -53
    b = np.full(M, -0.5 * sign)
    got = fair.airms.art("kaczmarz", A, b, [1], x0=x0, opts=fair.airms.options(relaxpar=1.0))[:, 0]
    A.close()
    for r in (0, M - 1):
        xs = x0[r * LEN:(r + 1) * LEN]
        c = (Fraction(b[r]) - sum(Fraction(v) for v in xs)) / LEN
        want = np.array([float(Fraction(v) + c) for v in xs])
        # two roundings of c (the sum's and the weight's) and one of x + c
        tol = 3 * 2.0 ** -53 * (abs(float(c)) + np.abs(xs).max())
        assert np.abs(got[r * LEN:(r + 1) * LEN] - want).max() <= tol
