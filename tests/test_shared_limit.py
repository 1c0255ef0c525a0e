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
