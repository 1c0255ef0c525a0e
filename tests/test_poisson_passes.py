"""The bounded field solve in one kernel per axis against the oracle, over its own edges.

Types I fold about the middle while the intervals stay even and above 16: sizes
with no fold (odd, small), one, several; extensions that share the FFT's table and
ones with their own; odd and even lengths of the other kinds; radices 2 to 8 and
larger primes; single-point axes; odd line counts (the last line has no partner);
four and eight pairs per CTA; and blocks left to cuFFT (a prime factor above 31, a
line too long).  Bar as in the other bounded-solve tests: 1e-11 of the maximum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

D, N, DN, ND, P_ = 1, 2, 3, 4, 0
CASES = [
    ((64, 34, 20), (D, N, D)), ((64, 34, 20), (N, D, N)),
    ((33, 17, 19), (D, N, D)), ((36, 72, 18), (N, D, N)),
    ((2, 3, 5), (D, N, D)), ((2, 2, 2), (D, D, D)), ((1, 2, 1), (N, P_, N)), ((1, 1, 1), (P_, DN, ND)),
    ((21, 25, 14), (DN, ND, P_)), ((16, 49, 27), (ND, P_, DN)), ((11, 13, 29), (P_, DN, D)),
    ((128, 10, 9), (D, ND, N)), ((9, 128, 16), (N, N, DN)), ((10, 9, 130), (DN, P_, N)),
    ((320, 6, 5), (ND, D, N)), ((6, 5, 640), (N, DN, D)),
    ((74, 8, 6), (N, D, P_)), ((8, 37, 10), (D, P_, N)), ((6, 5, 700), (D, N, DN)),
]


@pytest.mark.parametrize("table", [0, 1])
@pytest.mark.parametrize("n,kinds", CASES)
def test_passes_match_the_oracle(ohpic, oracle_mod, n, kinds, table):
    P, O = ohpic, oracle_mod
    rng = np.random.default_rng(sum(n) + 7 * table)
    rho = rng.normal(size=(n[2] + 1, n[1] + 1, n[0] + 1))
    bv = rng.normal(size=6)
    phi_o, e_o = O.poisson_bc(rho, kinds, bv, corrected=bool(table))
    with P.PoissonSolver(n, kinds, bv, table=table) as s:
        phi, e = s.solve(rho)
        assert np.array_equal(s.solve(rho, with_e=False), phi)
    scale = np.max(np.abs(phi_o))
    assert np.max(np.abs(phi - phi_o)) <= 1e-11 * scale
    assert np.max(np.abs(e - e_o)) <= 1e-11 * max(np.max(np.abs(e_o)), scale, 1e-300)
