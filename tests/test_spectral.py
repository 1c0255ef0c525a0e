"""The server's pooled field solve with our own transforms (spectral.cu) against numpy in FP64.

Grids cover every radix, primes up to the largest one kept in the kernels, odd
and even edges, edges of 2, planes of one CTA and of a cluster of two, and
grids that go to cuFFT instead (a large prime, a plane too large).

A served run of one step solves the charge of its injected particles; a single
context with the same injector and charges gives that charge to the bit (the
deposit is integer).  Tolerance: forward and inverse transforms commit about
3 eps per radix-2 level each, so phi is within 6 eps log2(N) of the exact one in
the 2-norm, the spectrum of the particles' noise being flat (each mode's error
is relative to that mode); a factor 2 is left for the sums of prime radices.
E is compared with the stencil of the served phi, in FP32, bit for bit."""
import numpy as np
import pytest

REF_PI = 3.14159265358979   # science_constants.f90:4

GRIDS = [(2, 2, 2), (2, 8, 5), (7, 3, 9), (4, 6, 2), (16, 16, 16), (13, 11, 31), (50, 36, 27), (64, 33, 48),
         (49, 25, 40), (29, 34, 23), (128, 126, 10), (9, 130, 20), (37, 12, 8), (8, 10, 67), (24, 20, 200),
         (162, 161, 3)]


def _phi(rho):
    nz, ny, nx = rho.shape

    def lam(n, k):
        return (2.0 * np.sin(REF_PI * np.minimum(k, n - k) / n)) ** 2
    den = (lam(nz, np.arange(nz))[:, None, None] + lam(ny, np.arange(ny))[None, :, None] +
           lam(nx, np.arange(nx // 2 + 1))[None, None, :])
    den[0, 0, 0] = np.inf
    return np.fft.irfftn(np.fft.rfftn(rho) / den, s=rho.shape, axes=(0, 1, 2))


def _stencil(phi, axis):
    half = phi.dtype.type(0.5)
    return half * ((np.roll(phi, 1, axis) - phi) + (phi - np.roll(phi, -1, axis)))


def _request(S, n, seed):
    ppc = 6
    r = S.thermal_request(n, ppc, 1, seed=seed)
    r.keep_fields = True
    return r


@pytest.mark.gpu
def test_served_solve_matches_numpy(ohpic):
    P = ohpic
    from ohhelppic3d_gb300 import serve as S
    reqs = [_request(S, n, (42, 52 + i)) for i, n in enumerate(GRIDS)]
    reqs += [_request(S, n, (7, 99)) for n in GRIDS[2:6]]   # two slots of a pool at once
    with S.Server(weights=P.WEIGHTS_STANDARD, hbm_budget=8 << 30) as server:
        ids = [server.submit(r) for r in reqs]
        server.wait(120.0)
        res = [server.result(i, r) for i, r in zip(ids, reqs)]
    for r, got in zip(reqs, res):
        n = r.n
        assert got["status"] == P.OK
        with P.PicContext(P.make_config(n=n, dt=r.dt, b0=r.b0, qm=r.qm, q=r.q,
                                        capacity=[6 * n[0] * n[1] * n[2] + 64] * 2, precision=P.FP32,
                                        weights=P.WEIGHTS_STANDARD)) as ctx:
            ctx.init_particles(r.species, seed=r.seed)
            ctx.scatter()
            rho = ctx.field(P.RHO)
        want = _phi(rho)
        eps = np.finfo(np.float32).eps / 2
        phi = got["fields"]["phi"]
        assert np.linalg.norm(phi - want) <= 12 * eps * np.log2(rho.size) * np.linalg.norm(want), n
        phi = phi.astype(np.float32)
        for axis, k in ((2, "ex"), (1, "ey"), (0, "ez")):
            assert np.array_equal(got["fields"][k].astype(np.float32), _stencil(phi, axis)), (n, k)


@pytest.mark.gpu
def test_weight_sums_and_tallies_are_cleared_by_the_solve(ohpic):
    """The solve clears the weight sums it reads and, in a step, the push's tallies: a
    deposit, reads of rho in between, and separate calls give the fused steps' bits."""
    P = ohpic
    n, ppc = (12, 10, 9), 8

    def make(prec):
        ctx = P.PicContext(P.make_config(n=n, dt=0.1, b0=(0, 0, 0.5), qm=[-1.0, 0.01, 0.02],
                                         q=[-0.125, 0.0625, 0.0625], capacity=[n[0] * n[1] * n[2] * ppc + 64] * 3,
                                         precision=prec, weights=P.WEIGHTS_STANDARD, sort_every=2))
        ctx.init_particles([P.species_init(ppc, v) for v in (1.0, 0.5, 0.1)])
        return ctx
    for prec in (P.FP64, P.FP32):
        with make(prec) as a, make(prec) as b:
            a.sort()
            b.sort()
            a.step(0.1, 4)
            for i in range(4):
                if i == 2:
                    b.sort()
                b.scatter()
                b.field(P.RHO)       # forms rho and clears the sums before the solve
                b.solve()
                b.diagnostics()
                b.solve()
                b.push(0.1)
            a.solve()
            b.scatter()
            b.solve()
            assert a.diagnostics()["crossings"] == b.diagnostics()["crossings"]
            for k in (P.RHO, P.PHI, P.EX, P.EY, P.EZ):
                assert np.array_equal(a.field(k), b.field(k)), k
