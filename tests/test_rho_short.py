"""FP32 rho with short charges: one 64-bit sum, one rounding, the same bits.

Charges whose mantissas are short once their common zeros are gone (powers of two,
as wp^2 / qm / ppc often is; up to 20 bits) take a 64-bit sum; longer ones, sums
that a node's weights could overflow, and exponents out of range take the general
path.  On-node particles make every node's weight sum known (units of 2^24), so rho
must be the correctly rounded FP32 of the exact rational."""
from fractions import Fraction

import numpy as np
import pytest

from test_rho_exact import _nearest_f32

pytestmark = pytest.mark.gpu

LONG = float((1 << 20) - 1) * 2.0 ** -20       # 20 bits: the short form's longest


@pytest.mark.parametrize("q,heavy", [
    ([-1.0 / 16, 1.0 / 16], 0),                 # one bit each
    ([0.75, -0.625, 2.0 ** -9], 0),             # three species, different exponents
    ([1.0, 0.0], 0),                            # a charge of zero
    ([-0.05, 0.05], 0),                         # full mantissas: general path
    ([LONG], 270_000),                          # past 2^42 units on one node: general path there
    ([3.0 * 2.0 ** -130, -2.0 ** -128], 0),     # results outside the normal range
    ([2.0 ** 100, 2.0 ** 99], 0),               # unit above the range of the short form
    ([0.5, -0.5, 0.25, -0.25, 1.0, 2.0, 4.0, -7.0], 0),
])
def test_short_charges_round_once(ohpic, q, heavy):
    P = ohpic
    n = (4, 4, 4)
    rng = np.random.default_rng(len(q))
    counts = [rng.integers(0, 40, size=n[::-1]) for _ in q]
    counts[0][1, 2, 3] += heavy
    cfg = P.make_config(n=n, dt=0.1, b0=(0.0, 0.0, 0.0), qm=[-1.0] * len(q), q=q,
                        capacity=[int(c.sum()) + 64 for c in counts], precision=P.FP32, sort_every=0,
                        weights=P.WEIGHTS_STANDARD)
    with P.PicContext(cfg) as ctx:
        for s, c in enumerate(counts):
            zz, yy, xx = np.nonzero(c)
            at = [np.repeat(v, c[zz, yy, xx]).astype(np.float64) for v in (xx, yy, zz)]
            zero = np.zeros_like(at[0])
            ctx.upload(s, dict(zip(("x", "y", "z", "vx", "vy", "vz"), at + [zero] * 3)))
        ctx.scatter()
        got = ctx.field(P.RHO).astype(np.float32)
    for idx in np.ndindex(*n[::-1]):
        exact = sum(Fraction(qs) * int(c[idx]) for qs, c in zip(q, counts))
        if 0 < abs(exact) < Fraction(2) ** -126:
            assert abs(Fraction(float(got[idx])) - exact) <= Fraction(2) ** -149
        else:
            assert got[idx] == _nearest_f32(exact), idx
