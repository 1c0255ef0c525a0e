"""The FP32 injector against the FP64 computation it rounds.

Velocities by pairs of floats and positions by integers store the float that the FP64
computation rounds to, or leave the particle to that computation: equality, no tolerance.
"""
import pathlib
import subprocess

import numpy as np
import pytest

import ohhelppic3d_gb300 as P

CSRC = pathlib.Path(P.__file__).parent / "csrc"

HOST = r"""
#include "normal_pair.cuh"
#include <cstdio>
#include <random>
using namespace ohpic;
static constexpr NormalTables T = make_normal_tables();
int main()
{
    std::mt19937_64 g(7);
    const double pi = 3.14159265358979;
    long open = 0, wrong = 0, plain = 0;
    for (long t = 0; t < 2000000; ++t) {
        uint32_t a = g(), b = g();
        const int sh = g() % 32;
        switch (t & 7) {   // near 0, near 1, whole and half steps of the tables, quarter turns
        case 1: a >>= sh; break;
        case 2: a = ~(a >> sh); break;
        case 3: b >>= sh; break;
        case 4: b = 0x40000000u * (b & 3) + (b >> sh) - (b >> sh >> 1); break;
        case 5: b = ((b & 255) << 24) + 0x800000u + (uint32_t)(g() % 3) - 1u; break;
        case 6: a = ((a & 255) << 24) + (uint32_t)(g() % 5) - 2u; break;
        }
        if (!a) continue;
        const double sigma = t % 5 ? std::ldexp(1.0 + (g() % 1000) * 1e-3, (int)(g() % 100) - 50) : 0.1;
        const double drift = t % 3 == 0 ? 0.0 : sigma * std::ldexp((t & 1 ? 1.0 : -1.0) / 3, (int)(g() % 16) - 8);
        const FloatPair s{(float)sigma, (float)(sigma - (float)sigma)}, d{(float)drift, (float)(drift - (float)drift)};
        const FloatPair m = pair_mul(radius(a, T.log), s);
        FloatPair sn, cs;
        turn(b, T.trig, sn, cs);
        const double r1 = a * 0x1p-32, r2 = b * 0x1p-32, M = sigma * std::sqrt(-2.0 * std::log(r1));
        for (int k = 0; k < 2; ++k) {
            double v = k ? M * std::cos(2.0 * pi * r2) : M * std::sin(2.0 * pi * r2);
            v = v < sigma * 6 ? v : sigma * 6;
            v = -sigma * 6 > v ? -sigma * 6 : v;
            float f;
            const bool ok = round_velocity(m, k ? cs : sn, d, (float)(5.99 * sigma), f);
            if ((t & 7) == 0) { ++plain; open += !ok; }
            wrong += ok && f != (float)(v + drift);
        }
    }
    std::printf("%ld %ld %ld\n", wrong, open, plain);
}
"""


def test_pairs_round_as_fp64(tmp_path):
    (tmp_path / "t.cpp").write_text(HOST)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(CSRC), "-o", str(tmp_path / "t"),
                    str(tmp_path / "t.cpp")], check=True)
    wrong, left, plain = map(int, subprocess.run([str(tmp_path / "t")], check=True, capture_output=True,
                                                 text=True).stdout.split())
    assert wrong == 0
    assert left <= plain / 2000       # 2 x bound / spacing of the floats: 2^-14 on average


# (grid, particles per cell, vth, drift, box): whole and broken faces, a box short of the
# grid, cold, tiny and wide thermal speeds, fewer particles than a CTA and than the grid
CASES = [
    ((32, 32, 32), 12, 1.0, (0, 0, 0), None),
    ((50, 36, 27), 9, 0.1, (0.3, -2.0, 1e-3), ((2, 0, 5), (47, 36, 20))),
    ((24, 20, 15), 8, 3.0, (0, 1e3, -1e-9), ((0.5, 0, 0.25), (23.5, 20, 14.0))),
    ((16, 16, 16), 8, 0.0, (0.25, 0, -0.1), None),
    ((16, 16, 16), 8, 1e-30, (0, 0, 0), None),
    ((8, 8, 8), 0.3, 1.0, (0, 0, 0), None),
]


@pytest.mark.gpu
@pytest.mark.parametrize("n,ppc,vth,drift,box", CASES)
def test_fp32_injector_rounds_the_fp64_one(n, ppc, vth, drift, box):
    out = []
    for prec in (P.FP64, P.FP32):
        cap = int(np.prod(n) * ppc) + 2
        cfg = P.make_config(n=n, dt=0.1, b0=(0, 0, 0), qm=[-1.0], q=[-1.0], capacity=[cap], precision=prec)
        with P.PicContext(cfg) as ctx:
            kw = {} if box is None else dict(lo=box[0], hi=box[1])
            ctx.init_particles([P.species_init(ppc, vth, drift=drift, **kw)], seed=(42, 61), advance=999)
            out.append({k: v.copy() for k, v in ctx.download(0, order=False).items()})
    a, b = out
    assert len(a["x"]) == len(b["x"])
    for d, k in enumerate("xyz"):
        cell = np.floor(a[k])
        off = (a[k] - cell).astype(np.float32)
        cell, off = cell + (off >= 1), np.where(off >= 1, np.float32(0), off)
        np.testing.assert_array_equal(b[k], np.where(cell >= n[d], cell - n[d], cell) + off.astype(np.float64))
        np.testing.assert_array_equal(b["v" + k], a["v" + k].astype(np.float32).astype(np.float64))
