"""Launches whose shared memory, static and dynamic together, passes 48 KB while the
dynamic part alone does not: each needs the opt-in for more, or it is refused.

The opt-in is a property of a kernel in its process, so every case runs in a process of
its own, where no larger launch has asked for it before."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def _alone(code):
    r = subprocess.run([sys.executable, "-c", "import ohhelppic3d_gb300 as P\n" + code], capture_output=True, text=True,
                       timeout=300, env={**os.environ, "PYTHONPATH": os.pathsep.join([os.path.dirname(HERE), HERE])})
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]


def test_served_solve_of_a_plane_at_the_limit(ohpic):
    # two buffers of 2992 complex numbers and 154 twiddles: 49104 bytes, and the charges' integer form
    _alone("import test_spectral as T\nT.GRIDS = [(66, 88, 4)]\nT.test_served_solve_matches_numpy(P)\n")


MODULES = """
import numpy as np
import oracle as O
n = (49, 49, 9)
setup = O.Setup(n=n, dt=0.1, b0=(0.1, 0.2, 0.5), species=[O.SpeciesInit(ppc=2, vth=1.0, qm=-1.0, wp=1.0),
                                                          O.SpeciesInit(ppc=2, vth=0.1, qm=0.01, wp=0.1)])
ref = O.Oracle(setup)
ref.init_particles()
caps = [ref.count(s) + 64 for s in range(2)]
ctx = P.PicContext(P.make_config(n=n, dt=0.1, b0=setup.b0, qm=[-1.0, 0.01], q=[setup.charge(s) for s in setup.species],
                                 capacity=caps, precision=P.FP64, sort_every=0))
# 12 x 12 x 8 nodes of 32 bytes and the particles' slots: 49152 bytes
assert ctx.get_tuning()["tile"] == (7, 7, 3) and ctx.get_tuning()["halo"] == 2
for s in range(2):
    ctx.upload(s, ref.get_particles(s))
ref.deposit()
ref.solve()
ctx.sort()
for k, w in ((P.EX, O.EX), (P.EY, O.EY), (P.EZ, O.EZ)):
    ctx.set_field(k, ref.get_field(w))
for s in range(2):
    e, ids, p = ctx.interp(s), ctx.download(s, order=False)["ids"], ref.get_particles(s)
    for i in range(0, len(ids), 97):
        j = ids[i]
        assert np.array_equal(e[i], ref.interp(p["x"][j], p["y"][j], p["z"][j]))
ctx.move(0.1)
ref.push()
for s in range(2):
    got, want = ctx.download(s), ref.get_particles(s)
    for k in ("x", "y", "z", "vx", "vy", "vz"):
        assert np.array_equal(got[k], want[k]), k
"""


def test_sorted_fp64_interpolation_and_move_at_the_limit(ohpic, oracle_mod):
    _alone(MODULES)


STEPS = """
import numpy as np
def run(n, tile, move):
    cap = 8 * n[0] * n[1] * n[2] + 64
    with P.PicContext(P.make_config(n=n, dt=0.1, b0=(0.1, 0.2, 0.5), qm=[-1.0], q=[-0.125], capacity=[cap],
                                    precision=P.FP32, weights=P.WEIGHTS_STANDARD, sort_every=0, tile=tile)) as ctx:
        ctx.init_particles([P.species_init(8, 1.0)])
        ctx.sort()
        for _ in range(3):
            ctx.move(0.1) if move else ctx.step(0.1, 1)
        ctx.solve()
        return [ctx.download(0)[k] for k in ("x", "y", "z", "vx", "vy", "vz")], ctx.field(P.EX)
for n, tile, move in {cases}:
    # the limit's tile first; then small tiles, far from it
    (pa, ea), (pb, eb) = run(n, tile, move), run(n, (2, 2, 2), move)
    assert np.array_equal(ea, eb) and all(np.array_equal(a, b) for a, b in zip(pa, pb)), (n, tile)
"""


@pytest.mark.parametrize("n,tile,move", [
    ((12, 12, 12), (2, 6, 6), False),    # 7 x 11 x 11 nodes of 24 bytes and the quads' stage: 49136 bytes
    ((22, 28, 10), (11, 14, 5), True),   # 16 x 19 x 10 nodes of 16 bytes: 48768 bytes
])
def test_fp32_launches_at_the_limit(ohpic, n, tile, move):
    _alone(STEPS.replace("{cases}", repr([(n, tile, move)])))


def test_served_push_at_the_limit(ohpic):
    # boxes of 9 x 9 x 9 nodes: 46304 bytes, and 5.9 KB for the run's descriptor and the queue
    _alone("import test_serve as T\np = T._probe((16, 16, 16), 9, (42, 78))\n"
           "got, _ = T._serve([p], tile=4, tile_x=4, halo=2)\nref, _ = T._serve([p])\nT._same_state(ref[0], got[0])\n")
