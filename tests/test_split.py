"""The CTAs per (species, tile): chosen by the library at 0, the default, and as asked
otherwise, one among them.  The results do not depend on it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_split_of_one_runs_one_cta_per_tile(ohpic):
    P = ohpic
    n, ppc = (16, 16, 16), 128
    ms, state = [], []
    for split in (None, 1, 3):
        with P.PicContext(P.make_config(n=n, dt=0.1, b0=(0, 0.1, 0.5), qm=[-1.0], q=[-1.0 / ppc], tile=(8, 8, 8),
                                        capacity=[4096 * ppc + 64], precision=P.FP64, sort_every=0)) as ctx:
            ctx.init_particles([P.species_init(ppc, 1.0)])
            if split is None:
                assert ctx.get_tuning()["split"] == 0
            else:
                ctx.set_tuning(split=split)
                assert ctx.get_tuning()["split"] == split
                ctx.set_tuning(halo=2)           # what is not named stays
                assert ctx.get_tuning()["split"] == split
            ctx.sort()
            ctx.step(0.1, 2)
            ctx.set_push_timing(True)
            ctx.step(0.1, 3)
            ms.append(ctx.stats()["push_ms"])
            for bad in (-1, 65):
                with pytest.raises(P.OhpicError):
                    ctx.set_tuning(split=bad)
            p = ctx.download(0)
            state.append([ctx.field(P.RHO)] + [p[k] for k in ("x", "y", "z", "vx", "vy", "vz")])
    for other in state[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(state[0], other))
    # eight CTAs of the chip's 304 against the library's 128: about 13 times as long
    assert ms[1] > 3.0 * ms[0], ms
