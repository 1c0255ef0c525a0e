"""Queue items of the server: a run's fields do not depend on how its tiles are cut.

Alone, a run's tiles are cut into many items; among larger runs they stay whole.  The
deposit is in integers and a particle's push does not depend on its CTA, so both give
the same bits.
"""
import numpy as np
import pytest

import ohhelppic3d_gb300 as P
from ohhelppic3d_gb300 import serve


def _request(n, ppc, steps, seed, keep=True):
    return serve.Request(n=n, nsteps=steps, qm=[-1, 0.01], q=[-1.0 / ppc, 1.0 / ppc],
                         species=[P.species_init(ppc, 1.0), P.species_init(ppc, 0.1)], b0=(0, 0, 0.5),
                         seed=(42, seed), keep_fields=keep)


@pytest.mark.gpu
@pytest.mark.parametrize("n,ppc", [((16, 16, 16), 64), ((32, 16, 8), 5), ((24, 40, 16), 100)])
def test_fields_do_not_depend_on_the_cut(n, ppc):
    got = []
    for company in (0, 6):
        server = serve.Server(weights=P.WEIGHTS_STANDARD, hbm_budget=8 << 30)
        reqs = [_request(n, ppc, 11, 5)] + [_request((64, 64, 64), 4, 12, 9 + i, keep=False) for i in range(company)]
        ids = [server.submit(r) for r in reqs]
        server.wait()
        got.append(server.result(ids[0], reqs[0]))
        server.close()
    for k in ("rho", "phi", "ex", "ey", "ez"):
        np.testing.assert_array_equal(got[0]["fields"][k], got[1]["fields"][k])
    assert got[0]["crossings"] == got[1]["crossings"] and got[0]["count"] == got[1]["count"]
