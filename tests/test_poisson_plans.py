"""The bounded field solve's ways to transform, each where it must be taken: cuFFT over
extended lines (a prime factor above 67, a line too long), and the one-kernel passes with
two, four and eight pairs of lines per CTA, their table in shared memory or not.  Against
the oracle, to 1e-11 of the maximum as in the other bounded-solve tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P_, D, N, DN, ND = 0, 1, 2, 3, 4


def _compare(P, want, got):
    (phi_o, e_o), (phi, e) = want, got
    scale = np.max(np.abs(phi_o))
    assert np.max(np.abs(phi - phi_o)) <= 1e-11 * scale
    assert np.max(np.abs(e - e_o)) <= 1e-11 * max(np.max(np.abs(e_o)), scale)


def _solve(P, O, n, kinds, table):
    rng = np.random.default_rng(sum(n) + 7 * table)
    rho = rng.normal(size=(n[2] + 1, n[1] + 1, n[0] + 1))
    bv = rng.normal(size=6)
    with P.PoissonSolver(n, kinds, bv, table=table) as s:
        plan = s.plan()
        _compare(P, O.poisson_bc(rho, kinds, bv, corrected=bool(table)), s.solve(rho))
        assert np.array_equal(s.solve(rho, with_e=False), s.solve(rho)[0])
    return plan


@pytest.mark.parametrize("table", [0, 1])
@pytest.mark.parametrize("n,kinds", [
    # each kind on an axis with a factor of 71 or 73, which takes the other axes along
    ((71, 9, 10), (P_, D, N)), ((10, 71, 7), (DN, D, P_)), ((8, 6, 71), (ND, P_, N)), ((73, 8, 12), (DN, N, D)),
    ((9, 73, 5), (N, ND, DN)), ((71, 71, 6), (D, N, ND)), ((5, 6, 142), (P_, DN, P_)), ((146, 1, 2), (N, P_, D)),
    # longer than a CTA's buffers hold
    ((1100, 6, 5), (DN, D, N)), ((4, 7, 1100), (D, P_, P_)),
])
def test_blocks_that_go_through_cufft(ohpic, oracle_mod, n, kinds, table):
    assert _solve(ohpic, oracle_mod, n, kinds, table)["pairs"] == (0,) * 5


@pytest.mark.parametrize("n,kinds,at,pairs,shared", [
    ((33, 17, 19), (D, N, D), 2, 2, True),
    ((40, 64, 20), (N, N, ND), 2, 4, True),
    ((72, 72, 20), (N, D, D), 2, 8, True),       # 73 x 71 lines along z: 5183
    ((20, 70, 74), (P_, N, N), 0, 8, True),      # 5325 rows of x, the last one without a partner
    ((190, 190, 4), (N, N, N), 2, 8, False),     # 36481 lines
    ((182, 3, 183), (P_, DN, ND), 1, 8, False),
])
def test_passes_of_every_shape(ohpic, oracle_mod, n, kinds, at, pairs, shared):
    plan = _solve(ohpic, oracle_mod, n, kinds, 0)
    assert (plan["pairs"][at], plan["shared"][at]) == (pairs, shared), plan


@pytest.mark.parametrize("table", [0, 1])
def test_four_pairs_without_a_shared_table(ohpic, oracle_mod, table):
    """16640 long lines along z: a block repeated along its periodic axes has the block's
    own solution repeated."""
    P, O = ohpic, oracle_mod
    small, times, nz, kinds, bv = (13, 16), (10, 8), 216, (P_, P_, DN), (0.0,) * 4 + (0.3, 0.2)
    core = np.random.default_rng(table).normal(size=(nz + 1, small[1], small[0]))

    def block(a, reps):
        a = np.tile(a, (1,) * (a.ndim - 2) + reps)
        return np.pad(a, [(0, 0)] * (a.ndim - 2) + [(0, 1), (0, 1)], mode="wrap")
    phi, e = O.poisson_bc(block(core, (1, 1)), kinds, bv, corrected=bool(table))
    reps = (times[1], times[0])
    with P.PoissonSolver((small[0] * times[0], small[1] * times[1], nz), kinds, bv, table=table) as s:
        plan = s.plan()
        assert (plan["pairs"][2], plan["shared"][2]) == (4, False), plan
        _compare(P, (block(phi[..., :-1, :-1], reps), block(e[..., :-1, :-1], reps)), s.solve(block(core, reps)))
