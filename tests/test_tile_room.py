"""What a context takes for a tile: an edge left open (0) gets a default, which shrinks where
the staged box needs it, at least to the room that the largest powers of two dividing the
axes (at most 8) leave.

So a configuration is accepted whenever those edges' box fits a CTA's shared memory at the
default halo, and a tuning may widen the halo as far as those edges allow; where the default
tile has the room, it stands."""
import ctypes as C
import random

import numpy as np
import pytest


def _plain(n, tile):
    return [t or next(e for e in (8, 4, 2, 1) if v % e == 0) for v, t in zip(n, tile)]


def _fits(tile, halo, fp64):
    nodes = int(np.prod([t + 2 * halo + 1 for t in tile]))
    return nodes * (4 * 8 + 8 if fp64 else 4 * 4 + 8) <= 192 * 1024


def _create(P, n, tile, fp64, capacity=64):
    cfg = P.make_config(n=n, dt=0.1, b0=(0, 0, 0.5), qm=[-1.0, 0.01], q=[-1.0, 1.0], capacity=[capacity] * 2,
                        precision=P.FP64 if fp64 else P.FP32, tile=tile)
    out = C.c_void_p()
    rc = P.lib().ohpic_create(C.byref(cfg), C.byref(out))
    if rc == P.OK:
        P.lib().ohpic_destroy(out)
    return rc


def _configurations():
    fixed = [((512, 54, 54), (64, 0, 0), False), ((512, 54, 54), (48, 0, 0), False), ((480, 54, 54), (48, 0, 0), False),
             ((256, 54, 54), (32, 0, 0), True), ((256, 100, 100), (32, 0, 0), True), ((64, 64, 64), (64, 0, 0), False)]
    rnd = random.Random(5)
    for _ in range(1500):
        n = [rnd.choice([rnd.randint(1, 60), rnd.randint(1, 520)]) for _ in range(3)]
        tile = [0, 0, 0]
        for d in range(3):
            if rnd.random() < 0.4:
                tile[d] = rnd.choice([t for t in range(1, 65) if n[d] % t == 0])
        fixed.append((tuple(n), tuple(tile), rnd.random() < 0.5))
    return fixed


def test_open_edges_are_refused_only_where_no_box_fits(ohpic):
    """The shape is judged before any CUDA call, so this holds on any host."""
    P = ohpic
    for n, tile, fp64 in _configurations():
        if any(t and v % t for v, t in zip(n, tile)) or not _fits([t or 1 for t in tile], 2, fp64):
            assert _create(P, n, tile, fp64) == P.ERR_INVALID, (n, tile, fp64)
        elif n[0] * n[1] * n[2] < 1 << 21 and _fits(_plain(n, tile), 2, fp64):
            assert _create(P, n, tile, fp64) != P.ERR_INVALID, (n, tile, fp64)
    # few tiles: the default is smaller than the powers of two, and fits where they do not
    assert not _fits(_plain((64, 64, 64), (64, 0, 0)), 2, False)
    assert _create(P, (64, 64, 64), (64, 0, 0), False) != P.ERR_INVALID


@pytest.mark.gpu
@pytest.mark.parametrize("n,tile,fp64", [((45, 45, 45), (0, 0, 0), True), ((54, 18, 45), (0, 0, 0), True),
                                         ((64, 54, 27), (32, 0, 0), True), ((64, 27, 54), (64, 0, 0), False),
                                         ((45, 54, 18), (0, 0, 0), False)])
def test_default_tiles_take_every_halo(ohpic, n, tile, fp64):
    P = ohpic
    plain, ppc = _plain(n, tile), 2
    want = None
    with P.PicContext(P.make_config(n=n, dt=0.1, b0=(0, 0.1, 0.5), qm=[-1.0, 0.01], q=[-0.5, 0.5],
                                    capacity=[2 * ppc * n[0] * n[1] * n[2]] * 2, sort_every=2, tile=tile,
                                    precision=P.FP64 if fp64 else P.FP32, weights=P.WEIGHTS_STANDARD)) as ctx:
        ctx.init_particles([P.species_init(ppc, 1.0), P.species_init(ppc, 0.1)])
        start = [ctx.download(s) for s in range(2)]
        first = ctx.get_tuning()["tile"]
        for halo in [h for h in range(5) if _fits(plain, h, fp64)]:
            ctx.set_tuning(halo=halo)
            tile = ctx.get_tuning()["tile"]
            assert _fits(tile, halo, fp64) and (tile == first or not _fits(first, halo, fp64))
            for s in range(2):
                ctx.upload(s, {k: v for k, v in start[s].items() if k != "ids"})
            ctx.step(0.1, 3)
            got = [ctx.download(s)[k] for s in range(2) for k in ("x", "vx", "vz")]
            want = want or got
            assert all(np.array_equal(a, b) for a, b in zip(got, want)), halo
        assert halo >= 2
        ctx.set_tuning(halo=2)                 # the smaller tile goes on being taken
        assert ctx.get_tuning()["tile"] == tile
        ctx.set_tuning(tile=first)
        assert ctx.get_tuning()["tile"] == first
