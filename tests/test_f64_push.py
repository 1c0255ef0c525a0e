"""The FP64 push off the FP64 pipe: weight products in integers and rotations without
their zero products, bit for bit.

The CPU test restates the integer product of two weights (normalise, 64 x 64 -> 128
bits, sticky, round to 53 bits, nearest with ties to even) and compares it with the
FP64 multiply over weights of every size, including carries and ties.  On the GPU, a
field component B along an axis of 1e-300 makes the general rotation run with
products that change no bit, so a run with it must equal the run without; and a
particle on grid nodes (offset 0: the FP64 products) next to others must move as
it does alone."""
import numpy as np
import pytest

MASK = (1 << 64) - 1


def _unit(x: float):
    m, e = np.frexp(x)                        # x = m 2^e, m in [0.5, 1)
    return int(m * 2.0 ** 53) << 11, int(e) - 1


def _unit_mul(a, b):
    p = a[0] * b[0]
    hi, lo = p >> 64, p & MASK
    s = (hi >> 63) ^ 1
    hi = ((hi << s) | ((lo >> 63) & s)) & MASK
    lo = (lo << s) & MASK
    hi |= lo != 0
    t = (hi + 0x3ff + ((hi >> 11) & 1)) & MASK
    e = a[1] + b[1] + 1 - s
    return (1 << 63, e + 1) if t < hi else (t & ~0x7ff, e)


def _one_minus(x: float):
    b = int(np.float64(x).view(np.uint64))
    M, s = (b & ((1 << 52) - 1)) | (1 << 52), min(1022 - (b >> 52), 63)
    q, rem, half = M >> s, M & ((1 << s) - 1), (1 << s) >> 1
    R = (1 << 53) - q
    R -= rem > half or (rem == half and rem != 0 and R & 1)
    lz = 64 - R.bit_length()
    return R << lz, 63 - lz - 53


def _double(u) -> float:
    return float(np.ldexp(float(u[0] >> 11), u[1] - 52))


def test_integer_weight_products_are_the_fp64_ones():
    rng = np.random.default_rng(3)
    r = np.concatenate([rng.random(4000), rng.random(2000) * 2.0 ** -rng.integers(1, 50, 2000),
                        rng.integers(1, 1 << 20, 2000) * 2.0 ** -20, rng.integers(1, 1 << 48, 2000) * 2.0 ** -48,
                        1.0 - 2.0 ** -rng.integers(1, 53, 500).astype(float), 2.0 ** -rng.integers(1, 60, 500).astype(float)])
    r = r[(r > 0) & (r < 1)]
    for a, b, c in zip(r, rng.permutation(r), rng.permutation(r)):
        ab = _unit_mul(_unit(a), _unit(b))
        assert _double(ab) == a * b
        assert _double(_unit_mul(ab, _unit(c))) == (a * b) * c
    for x in np.concatenate([r, [0.5, 0.25, np.nextafter(0.5, 0), np.nextafter(0.5, 1), np.nextafter(1, 0), 2.0 ** -53,
                                 2.0 ** -54, 3 * 2.0 ** -54, 2.0 ** -300, 1.5 * 2.0 ** -53]]):
        assert _double(_one_minus(float(x))) == 1.0 - x, x
    # ties: (1 + 2^-27)(1 + 2^-26) / 4 has 54 significant bits
    for k in range(1, 60):
        a, b = (1 + k * 2.0 ** -27) / 2, (1 + 2.0 ** -26) / 2
        assert _double(_unit_mul(_unit(a), _unit(b))) == a * b


def _run(P, b0, parts, steps, weights=0, n=(12, 10, 9), e=None):
    cfg = P.make_config(n=n, dt=0.1, b0=b0, qm=[-1.0], q=[-0.1], capacity=[len(parts["x"]) + 8], precision=P.FP64,
                        weights=weights, sort_every=3)
    with P.PicContext(cfg) as ctx:
        ctx.upload(0, parts)
        ctx.step(0.1, steps)
        got = ctx.download(0)
        ctx.solve()
        return got, [ctx.field(k) for k in (P.RHO, P.PHI, P.EX, P.EY, P.EZ)]


def _parts(n, count, seed):
    rng = np.random.default_rng(seed)
    p = {k: rng.random(count) * n[d] for d, k in enumerate("xyz")}
    p.update({k: rng.standard_normal(count) for k in ("vx", "vy", "vz")})
    return p


@pytest.mark.gpu
@pytest.mark.parametrize("weights", [0, 1])
@pytest.mark.parametrize("bz", [0.5, 0.0])
def test_rotation_without_zero_products(ohpic, weights, bz):
    P = ohpic
    parts = _parts((12, 10, 9), 9000, 5)
    a, fa = _run(P, (0.0, 0.0, bz), parts, 7, weights)
    b, fb = _run(P, (1e-300, 0.0, bz), parts, 7, weights)
    for k in a:
        assert np.array_equal(a[k], b[k]), k
    for x, y in zip(fa, fb):
        assert np.array_equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("weights", [0, 1])
def test_offsets_at_the_edges_of_the_integer_products(ohpic, oracle_mod, weights):
    """Offsets of zero, one unit below 1, tiny ones in cell 0 (normal, subnormal, -0.0) and
    ordinary ones, one step against the oracle (1e-14 of the box: one step's rounding)."""
    P, O = ohpic, oracle_mod
    n = (12, 10, 9)
    special = [0.0, -0.0, 5e-324, 1e-310, 1e-200, 1e-90, 2.0 ** -52, 0.5, 1.0 - 2.0 ** -53, 1.0, 3.0, 7.5,
               np.nextafter(4.0, 0.0), np.nextafter(4.0, 5.0), 8.25, 8.999]
    rng = np.random.default_rng(11)
    c = 4000
    p = {k: rng.choice(special, c) for k in "xyz"}
    for k in "xyz":
        mix = rng.random(c) < 0.3
        p[k][mix] = rng.random(mix.sum()) * 9
    p.update({k: rng.standard_normal(c) * 1e-3 for k in ("vx", "vy", "vz")})
    setup = O.Setup(n=n, dt=0.1, b0=(0.0, 0.0, 0.5), weights=weights, species=[O.SpeciesInit(ppc=1, vth=1.0, qm=-1.0, q=-0.1)])
    ref = O.Oracle(setup, capacity=[c + 8])
    ref.set_particles(0, p)
    ref.step(1)
    want = ref.get_particles(0)
    got, _ = _run(P, (0.0, 0.0, 0.5), p, 1, weights, n)
    for d, k in enumerate("xyz"):
        diff = np.abs(got[k] - want[k])
        diff = np.minimum(diff, n[d] - diff)
        assert np.max(diff) <= 1e-13
    for k in ("vx", "vy", "vz"):
        assert np.max(np.abs(got[k] - want[k])) <= 1e-12 * max(np.max(np.abs(want[k])), 1.0)
