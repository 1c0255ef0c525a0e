"""Default tiles of grids that no tile edge divides, and the split chosen per launch.

The deposit is integer and every particle advances on its own, so any tile shape
and split give the same bits: a context on its default tiles (the last tile of
an axis shorter than the others) against one on tiles that divide the grid, over
steps that cross a re-sort.  FP64 fields are bit-reproducible too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _context(P, n, ppc, precision, nspecies=2, tile=(0, 0, 0)):
    qm, q = [-1.0, 0.01][:nspecies], [-1.0 / ppc, 1.0 / ppc][:nspecies]
    cap = int(np.prod(n)) * ppc + 64
    ctx = P.PicContext(P.make_config(n=n, dt=0.1, b0=(0.1, 0.2, 0.5), qm=qm, q=q, capacity=[cap] * nspecies,
                                     precision=precision, weights=P.WEIGHTS_STANDARD, sort_every=3, tile=tile))
    ctx.init_particles([P.species_init(ppc, 1.0), P.species_init(ppc, 0.1)][:nspecies])
    return ctx


def _state(P, ctx, nspecies):
    ctx.step(0.1, 7)
    ctx.solve()
    fields = [ctx.field(k) for k in (P.RHO, P.PHI, P.EX, P.EY, P.EZ)]
    return fields, [ctx.download(s) for s in range(nspecies)], ctx.diagnostics()["crossings"]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n,ppc,nspecies", [
    ((13, 11, 7), 6, 2),       # shorter last tile on every axis, few particles
    ((27, 10, 17), 3, 1),
    ((5, 37, 41), 9, 2),
    ((50, 36, 27), 12, 2),
    ((16, 16, 16), 64, 1),     # divides; split into several CTAs per tile
])
def test_default_tiles_give_the_same_bits(ohpic, n, ppc, nspecies, precision):
    P = ohpic
    prec = P.FP64 if precision == "fp64" else P.FP32
    divides = tuple(next(t for t in (8, 4, 2, 1) if v % t == 0) for v in n)
    with _context(P, n, ppc, prec, nspecies) as a, _context(P, n, ppc, prec, nspecies, tile=divides) as b:
        b.set_tuning(split=3)
        assert b.get_tuning()["tile"] == divides
        (fa, pa, ca), (fb, pb, cb) = _state(P, a, nspecies), _state(P, b, nspecies)
        assert ca == cb
        for x, y in zip(fa, fb):
            assert np.array_equal(x, y)
        for x, y in zip(pa, pb):
            for k in x:
                assert np.array_equal(x[k], y[k]), k


def test_default_tile_can_be_set_again_and_others_must_divide(ohpic):
    P = ohpic
    with _context(P, (27, 10, 17), 3, P.FP32) as ctx:
        first = ctx.get_tuning()
        assert any(v % t for v, t in zip((27, 10, 17), first["tile"]))
        ctx.set_tuning(tile=(9, 5, 1))
        ctx.step(0.1, 2)
        ctx.set_tuning(tile=first["tile"])
        ctx.step(0.1, 2)
        with pytest.raises(P.OhpicError):
            ctx.set_tuning(tile=(9, 5, 2))
        assert ctx.get_tuning()["tile"] == first["tile"]
    with pytest.raises(P.OhpicError):
        P.PicContext(P.make_config(n=(27, 10, 17), dt=0.1, b0=(0, 0, 0), qm=[-1.0], q=[1.0], capacity=[64],
                                   tile=(8, 0, 0)))
