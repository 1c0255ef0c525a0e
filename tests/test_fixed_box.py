"""The FP32 push of tile (8,8,8), halo 2, has its box geometry compiled in; with halo 1 it
is read at run time.  Both give the same bits, through array and record pushes and on a
grid whose last tile is shorter."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ppc", [((40, 40, 40), 3), ((39, 40, 40), 2), ((40, 40, 40), 40)])
def test_compiled_box_gives_the_same_bits(ohpic, n, ppc):
    P = ohpic
    out = []
    for halo in (2, 1):
        cap = int(np.prod(n)) * ppc + 64
        cfg = P.make_config(n=n, dt=0.1, b0=(0.1, 0.2, 0.5), qm=[-1.0, 0.01], q=[-1.0 / ppc, 1.0 / ppc],
                            capacity=[cap] * 2, precision=P.FP32, weights=P.WEIGHTS_STANDARD, sort_every=3)
        with P.PicContext(cfg) as ctx:
            assert tuple(ctx.get_tuning()["tile"]) == (8, 8, 8)
            ctx.init_particles([P.species_init(ppc, 1.0), P.species_init(ppc, 0.1)])
            ctx.set_tuning(halo=halo)
            ctx.step(0.1, 8)
            ctx.solve()
            out.append([ctx.field(k) for k in (P.RHO, P.PHI, P.EX, P.EY, P.EZ)] +
                       [v for s in range(2) for v in ctx.download(s).values()])
    for x, y in zip(*out):
        assert np.array_equal(x, y)
