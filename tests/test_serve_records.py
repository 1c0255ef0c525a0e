"""The served push right after a sort reads the sort's records; in the other launch shapes a
transpose writes them back first.  Same bits, particles in injection order, at segments
whose lengths are no multiple of a quad, a single particle and an empty tile among them."""
import numpy as np
import pytest

import ohhelppic3d_gb300 as P
from ohhelppic3d_gb300 import serve


@pytest.mark.gpu
@pytest.mark.parametrize("n,ppc", [((16, 16, 8), 1.37), ((16, 8, 8), 1.0 / 1024), ((24, 24, 24), 0.013),
                                   ((32, 32, 32), 17.01)])
def test_push_from_records(n, ppc):
    got = []
    for shape in (dict(lane_particles=4, sort_every=1), dict(lane_particles=2, sort_every=1),
                  dict(lane_particles=4, sort_every=100)):
        req = serve.Request(n=n, nsteps=6, qm=[-1, 0.01], q=[-0.5, 0.5],
                            species=[P.species_init(ppc, 1.0), P.species_init(ppc, 0.1)], b0=(0, 0.1, 0.5),
                            keep_fields=True, keep_particles=True)
        with serve.Server(weights=P.WEIGHTS_STANDARD, hbm_budget=4 << 30, **shape) as server:
            i = server.submit(req)
            server.wait()
            got.append(server.result(i, req))
    for other in got[1:]:
        assert other["count"] == got[0]["count"] and other["crossings"] == got[0]["crossings"]
        for k in ("rho", "phi", "ex", "ey", "ez"):
            np.testing.assert_array_equal(got[0]["fields"][k], other["fields"][k])
        for a, b in zip(got[0]["particles_by_species"], other["particles_by_species"]):
            for k in a:
                np.testing.assert_array_equal(a[k], b[k])
