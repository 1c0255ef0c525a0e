"""The unsorted kernels over chunk sizes (counts around multiples of a chunk, empty and
tiny species) and the interpolation of one species at a time, against the oracle's
FP64 path through the module calls, bit for bit in the strict kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(1, 0), (511, 513), (3, 1025), (4096, 311300), (155648, 2), (2 * 304 * 512 + 1, 7)])
def test_unsorted_calls_match_the_oracle(ohpic, oracle_mod, counts):
    P, O = ohpic, oracle_mod
    n = (12, 10, 14)
    rng = np.random.default_rng(sum(counts))
    setup = O.Setup(n=n, dt=0.1, b0=(0.1, 0.2, 0.5),
                    species=[O.SpeciesInit(ppc=1, vth=1.0, qm=-1.0, wp=1.0),
                             O.SpeciesInit(ppc=1, vth=0.1, qm=0.01, wp=0.1)])
    parts = []
    for c in counts:
        p = {k: rng.random(c) * n[d] for d, k in enumerate(("x", "y", "z"))}
        p.update({k: rng.standard_normal(c) for k in ("vx", "vy", "vz")})
        parts.append(p)
    ref = O.Oracle(setup, capacity=[c + 8 for c in counts])
    q = [setup.charge(sp) for sp in setup.species]
    cfg = P.make_config(n=n, dt=0.1, b0=setup.b0, qm=[-1.0, 0.01], q=q, capacity=[c + 8 for c in counts],
                        precision=P.FP64, sort_every=0)
    with P.PicContext(cfg) as ctx:
        for s, p in enumerate(parts):
            ctx.upload(s, p)
            ref.set_particles(s, p)
        ctx.scatter()
        ref.deposit()
        rho = ref.get_field(O.RHO)
        assert np.max(np.abs(ctx.field(P.RHO) - rho)) <= 1e-13 * max(np.max(np.abs(rho)), 1.0)
        ref.solve()
        for k, w in ((P.EX, O.EX), (P.EY, O.EY), (P.EZ, O.EZ)):
            ctx.set_field(k, ref.get_field(w))
        for s, c in enumerate(counts):
            got = ctx.interp(s)
            assert got.shape == (c, 3)
            if c:
                p = parts[s]
                for i in rng.choice(c, size=min(c, 200), replace=False):
                    assert np.array_equal(got[i], ref.interp(p["x"][i], p["y"][i], p["z"][i])), (s, i)
        ctx.move(0.1)
        ref.push()
        for s in range(2):
            got, want = ctx.download(s), ref.get_particles(s)
            for k in ("x", "y", "z", "vx", "vy", "vz"):
                assert np.array_equal(got[k], want[k]), k
