"""Steps replayed as a captured CUDA graph against separately launched ones.

ohpic_step replays a captured step on small grids; solve() and push() always
launch plainly.  Whatever changes between steps (dt, tracking, tile shape, cadence,
new particles, an uploaded charge) must reach the replayed step, and counts, step
numbers and tallies must be those of plain steps.  Every sum is integer, so the
states agree bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _context(P, precision, n=(12, 10, 9), ppc=8):
    ctx = P.PicContext(P.make_config(n=n, dt=0.1, b0=(0, 0.1, 0.5), qm=[-1.0, 0.01], q=[-1.0 / ppc, 1.0 / ppc],
                                     capacity=[n[0] * n[1] * n[2] * ppc + 64] * 2, precision=precision,
                                     weights=P.WEIGHTS_STANDARD, sort_every=4))
    ctx.init_particles([P.species_init(ppc, 1.0), P.species_init(ppc, 0.1)])
    return ctx


def _plain(ctx, dt, since, cadence):
    """One step by its parts, with ohpic_step's sorts."""
    if since == 0:
        ctx.sort()
    ctx.solve()
    ctx.push(dt)
    return 0 if cadence and since + 1 >= cadence else since + 1


def _same(P, a, b):
    a.solve()
    b.solve()
    for k in (P.RHO, P.PHI, P.EX, P.EY, P.EZ):
        assert np.array_equal(a.field(k), b.field(k)), k
    for s in range(2):
        x, y = a.download(s), b.download(s)
        for k in x:
            assert np.array_equal(x[k], y[k]), k
    da, db = a.diagnostics(), b.diagnostics()
    for k in ("count", "crossings", "step"):
        assert da[k] == db[k], k


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_replayed_steps_match_plain_ones(ohpic, precision):
    P = ohpic
    prec = P.FP64 if precision == "fp64" else P.FP32
    with _context(P, prec) as a, _context(P, prec) as b:
        since = 0

        def both(dt, k):
            nonlocal since
            a.step(dt, k)
            for _ in range(k):
                since = _plain(b, dt, since, 4)
        both(0.1, 7)
        _same(P, a, b)
        both(0.05, 3)                    # another dt, then back
        both(0.1, 6)
        _same(P, a, b)
        for ctx in (a, b):
            ctx.set_energy_tracking(True)
        both(0.1, 5)
        assert a.diagnostics()["kinetic_energy"] == pytest.approx(b.diagnostics()["kinetic_energy"], rel=1e-6)
        _same(P, a, b)
        for ctx in (a, b):
            ctx.set_tuning(tile=(4, 5, 3), halo=1, split=2)
        since = 0
        both(0.1, 6)
        _same(P, a, b)
        rho = np.random.default_rng(1).standard_normal((9, 10, 12))
        for ctx in (a, b):
            ctx.set_field(P.RHO, rho)
        both(0.1, 3)
        _same(P, a, b)
        p = a.download(0)
        for ctx in (a, b):
            ctx.upload(0, {k: v[:100] for k, v in p.items()})
        since = 0
        both(0.1, 6)
        _same(P, a, b)


def test_replayed_steps_count_their_launches(ohpic):
    P = ohpic
    with _context(P, P.FP32) as ctx:
        ctx.step(0.1, 3)
        ctx.synchronize()
        per_step = []
        for _ in range(2):
            l0 = ctx.stats()["launches"]
            ctx.set_tuning(sort_every=0)
            ctx.step(0.1, 10)
            per_step.append((ctx.stats()["launches"] - l0) / 10)
        assert per_step[0] == per_step[1] and per_step[0] >= 3
