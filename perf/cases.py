"""The work a user of this package has it do, as timed cases.

Five kinds of case:

  run      a plasma run advanced by a number of steps through PicContext, from particles the
           program uploads or from the device injector; then the solved fields, and for runs of
           up to 20 million particles every particle's velocity and place, by id
  job      upload of every particle from pinned host arrays, steps with a diagnostics read after
           each, download of every particle: a batch job that keeps its state on the host
  modules  the reference's main loop through its module API: scatter, solve, interpolate, move
  poisson  the field solve on a bounded block with a boundary kind per axis, on device arrays
  serve    a handful of independent small runs through the continuous-batching server

The FP32 form's state and fields hold FP32 values (the API hands them out as FP64 arrays), so its
outputs are returned as float32; everything else is float64.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import ohhelppic3d_gb300 as P
from ohhelppic3d_gb300 import serve

DT = 0.1
NAMES = ("x", "y", "z", "vx", "vy", "vz")
# Runs of up to this many particles start from uploaded arrays and return their particles.
MOST_RETURNED = 20_000_000
# ... and of up to this many particle-steps are repeated in 64 bits by exact().
MOST_EXACT = 500_000_000
REF_PI = 3.14159265358979   # the reference's literal (science_constants.f90:4)


def _run(name, n, ppc, steps, precision="fp32", weights="standard", plasma="pair", tile="default", halo=0, lead=0,
         wce=0.5, vth=1.0, sort_every=20, kind="run"):
    return {"name": name, "kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "ppc": ppc, "steps": steps,
            "precision": precision, "weights": weights, "plasma": plasma, "tile": tile, "halo": halo, "lead": lead,
            "wce": wce, "vth": vth, "sort_every": sort_every}


def _poisson(name, n, kinds, table):
    return {"name": name, "kind": "poisson", "nx": n[0], "ny": n[1], "nz": n[2], "kx": kinds[0], "ky": kinds[1],
            "kz": kinds[2], "table": table}


def listed():
    return [
        # The 32^3 configuration, 100 steps, in the plain form a code first switches to: FP64, the
        # reference's weights, everything else at its default.
        _run("thermal_32_fp64", (32, 32, 32), 16, 100, precision="fp64", weights="reference"),
        # The same plasma in the precision form.
        _run("thermal_32_fp32", (32, 32, 32), 16, 100),
        # The smallest run of a parameter scan: launches and latency.
        _run("thermal_16_fp32", (16, 16, 16), 8, 200),
        # A grid whose edges no power of two divides far: 50 = 2 x 25, 36 = 4 x 9, 27 = 27 x 1.
        _run("ragged_50x36x27_fp32", (50, 36, 27), 20, 40),
        # The headline configuration, 1.07e9 particles, one sort cycle, in the launch shape the
        # integration guide gives for it.
        _run("thermal_256_fp32", (256, 256, 256), 32, 20, tile="16x8x8", halo=2, lead=10),
        # The FP64 form on a dense box of 6.7e7 particles.
        _run("thermal_128x128x64_fp64", (128, 128, 64), 32, 5, precision="fp64", weights="reference"),
        # Clustered two-stream plasma (a beam through the central 30% of x and y): tiles of very
        # different particle counts, fast particles, no magnetic field; three species.
        _run("beam_64x64x256_fp32", (64, 64, 256), 16, 20, plasma="beam", wce=0.0),
        # A batch job: state in pinned host arrays before and after, energies read every step.
        _run("job_64_fp32", (64, 64, 64), 32, 20, kind="job"),
        # The reference's own loop, call by call, on a small odd box, particles in upload order.
        _run("modules_24x20x15_fp64", (24, 20, 15), 16, 5, precision="fp64", weights="reference", kind="modules",
             sort_every=0),
        # The bounded field solve at the headline grid: conducting walls all round.
        _poisson("poisson_256_walls", (256, 256, 256), ("dirichlet",) * 3, "corrected"),
        # A small odd block with a different kind on each axis, in the reference's own table.
        _poisson("poisson_60x45x33_mixed", (60, 45, 33), ("dirichlet", "neumann", "periodic"), "as_written"),
        # Sixteen runs of the serving mix at once (16^3 to 64^3 cells), steps shortened.
        {"name": "serve_16_runs", "kind": "serve", "runs": 16, "step_scale": 0.05},
    ]


def _edge(rng, lo, hi):
    """A grid edge, spread over the logarithm; half of them multiples of 8, the rest whatever comes."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, v // 8 * 8) if rng.random() < 0.5 else max(lo, v)


def draw(rng):
    kind = rng.choice(("run", "run", "run", "run", "job", "modules", "poisson", "poisson", "serve"))
    if kind == "poisson":
        names = ("periodic", "dirichlet", "neumann", "dirichlet_neumann", "neumann_dirichlet")
        c = _poisson("", [_edge(rng, 16, 200) for _ in range(3)], [rng.choice(names) for _ in range(3)],
                     rng.choice(("corrected", "as_written")))
    elif kind == "serve":
        c = {"name": "", "kind": "serve", "runs": rng.randint(4, 24), "step_scale": round(rng.uniform(0.01, 0.05), 4)}
    elif kind == "modules":
        c = _run("", [_edge(rng, 12, 48) for _ in range(3)], rng.choice((4, 8, 16)), rng.randint(2, 6),
                 precision=rng.choice(("fp64", "fp32")), kind=kind, sort_every=0, wce=round(rng.random(), 3))
    elif kind == "job":
        c = _run("", [_edge(rng, 16, 64) for _ in range(3)], rng.choice((8, 16, 32)), rng.randint(5, 40),
                 precision=rng.choice(("fp64", "fp32")), kind=kind, wce=round(rng.random(), 3))
    else:
        precision = rng.choice(("fp64", "fp32", "fp32"))
        c = _run("", [_edge(rng, 12, 96) for _ in range(3)], rng.choice((8, 16, 32, 64)), rng.randint(5, 60),
                 precision=precision, weights=rng.choice(("standard", "reference")) if precision == "fp64" else
                 "standard", plasma=rng.choice(("pair", "pair", "beam")), wce=round(rng.random(), 3),
                 vth=round(rng.uniform(0.5, 2.0), 3), sort_every=rng.choice((8, 10, 20)))
        if c["plasma"] == "beam":
            c["wce"] = 0.0
        c["steps"] = max(2, min(c["steps"], (100_000_000 if precision == "fp64" else 600_000_000) // _count(c)))
        if precision == "fp32" and rng.random() < 0.3:
            c["lead"] = c["sort_every"] // 2
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# Plasmas: the species of workloads.py (electrons and ions of mass ratio 100;
# the two-stream set adds a beam in the central 30% of x and y, drift +5 in z).
# ---------------------------------------------------------------------------
def _grid(case):
    return case["nx"], case["ny"], case["nz"]


def _species(case):
    """(qm, q, ppc, vth, drift_z, lo, hi, count) per species."""
    n, ppc, vth = _grid(case), case["ppc"], case["vth"]
    whole = ((0.0, 0.0, 0.0), tuple(float(v) for v in n))

    def one(qm, q, ppc, vth, drift=0.0, box=whole):
        return [qm, q, ppc, vth, drift, box[0], box[1], int(ppc * math.prod(h - l for l, h in zip(*box)))]

    if case["plasma"] == "pair":
        return [one(-1.0, -1.0 / ppc, ppc, vth), one(0.01, 1.0 / ppc, ppc, 0.1 * vth)]
    tube = ((0.35 * n[0], 0.35 * n[1], 0.0), (0.65 * n[0], 0.65 * n[1], float(n[2])))
    sp = [one(-1.0, -1.0 / ppc, ppc, vth), one(-1.0, -1.0 / ppc, ppc, 0.5 * vth, 5.0, tube),
          one(0.01, 0.0, 2 * ppc, 0.1 * vth)]
    sp[2][1] = (sp[0][7] + sp[1][7]) / ppc / sp[2][7]   # neutral in total
    return sp


def _count(case):
    return sum(s[7] for s in _species(case))


def _uploaded(case):
    return _count(case) <= MOST_RETURNED


def _arrays(case, seed):
    """The particles of every species as six device arrays, from the seed alone."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    out = []
    for qm, q, ppc, vth, drift, lo, hi, count in _species(case):
        p = {}
        for d, k in enumerate(NAMES[:3]):
            p[k] = lo[d] + (hi[d] - lo[d]) * torch.rand(count, generator=g, device="cuda", dtype=torch.float64)
        for k in NAMES[3:]:
            p[k] = vth * torch.randn(count, generator=g, device="cuda", dtype=torch.float64).clamp_(-6.0, 6.0)
        p["vz"] += drift
        out.append(p)
    return out


def _pinned(count, dtype):
    return torch.empty(max(count, 1), dtype=dtype, pin_memory=True)


def _context(case):
    sp = _species(case)
    cfg = P.make_config(n=_grid(case), dt=DT, b0=(0.0, 0.0, case["wce"]), qm=[s[0] for s in sp], q=[s[1] for s in sp],
                        capacity=[s[7] + 1024 for s in sp],
                        precision=P.FP32 if case["precision"] == "fp32" else P.FP64,
                        weights=P.WEIGHTS_STANDARD if case["weights"] == "standard" else P.WEIGHTS_REFERENCE,
                        sort_every=case["sort_every"])
    ctx = P.PicContext(cfg)
    shape = {}
    if case["tile"] != "default":
        shape["tile"] = tuple(int(v) for v in case["tile"].split("x"))
    if case["halo"]:
        shape["halo"] = case["halo"]
    if case["lead"]:
        shape["sort_lead"] = case["lead"]
    if shape:
        ctx.set_tuning(**shape)
    return ctx


def prepare(case, seed):
    kind = case["kind"]
    if kind == "poisson":
        return _prepare_poisson(case, seed)
    if kind == "serve":
        return _prepare_serve(case, seed)
    sp = _species(case)
    st = {"case": case, "ctx": _context(case), "dtype": torch.float32 if case["precision"] == "fp32" else torch.float64}
    if not _uploaded(case):
        st["ctx"].init_particles([P.species_init(s[2], s[3], (0.0, 0.0, s[4]), s[5], s[6]) for s in sp],
                                 seed=(int(seed), 52))
        return st
    parts = _arrays(case, seed)
    st["host"] = [{k: _pinned(s[7], torch.float64) for k in NAMES} for s in sp]
    st["ids"] = [_pinned(s[7], torch.int32) for s in sp]
    for p, h in zip(parts, st["host"]):
        for k in NAMES:
            h[k][:len(p[k])].copy_(p[k])
    torch.cuda.synchronize()
    st["count"] = [s[7] for s in sp]
    st["views"] = [{k: h[k].numpy() for k in NAMES} for h in st["host"]]
    if kind == "job":
        st["given"] = st["views"]
        st["host"] = [{k: _pinned(s[7], torch.float64) for k in NAMES} for s in sp]
        st["views"] = [{k: h[k].numpy() for k in NAMES} for h in st["host"]]
        st["ctx"].set_energy_tracking(True)
    else:
        for s, v in enumerate(st["views"]):
            st["ctx"].upload_n(s, v, st["count"][s])
    return st


def run(state):
    case = state.get("case")
    if case["kind"] == "poisson":
        return _run_poisson(state)
    if case["kind"] == "serve":
        return _run_serve(state)
    if case["kind"] == "modules":
        return _run_modules(state)
    if case["kind"] == "job":
        return _run_job(state)
    ctx = state["ctx"]
    ctx.step(DT, case["steps"])
    out = _fields(state)
    if "host" in state:
        out["particles"] = _particles(state)
    return out


def _fields(state):
    """The fields solved from the particles' charge, as a run writes them out."""
    ctx = state["ctx"]
    ctx.solve()
    return {k: torch.from_numpy(ctx.field(w)).to(state["dtype"])
            for k, w in (("rho", P.RHO), ("phi", P.PHI), ("ex", P.EX), ("ey", P.EY), ("ez", P.EZ))}


def _particles(state):
    """Velocity and place of every particle, in upload order."""
    out = []
    for s, m in enumerate(state["count"]):
        state["ctx"].download_into(s, state["views"][s], state["ids"][s].numpy().view(np.uint32))
        at = state["ids"][s][:m].to("cuda", non_blocking=True).long()
        now = torch.empty(6, m, dtype=torch.float64, device="cuda")
        for k, name in enumerate(NAMES):
            now[k][at] = state["host"][s][name][:m].to("cuda", non_blocking=True)
        out.append(_particle(now, _grid(state["case"]), state["dtype"]))
    return out


def _particle(now, n, dtype):
    """Velocities, and positions as points on the periodic box's circles: x = 0 and x = n are the same place."""
    turn = now[:3] * (2.0 * math.pi / torch.tensor(n, dtype=torch.float64, device="cuda").view(3, 1))
    return {"velocity": now[3:].to(dtype), "place": torch.cat((torch.cos(turn), torch.sin(turn))).to(dtype)}


def _run_job(state):
    """Upload, steps with the energies read after each, download into arrays of their own."""
    ctx, case = state["ctx"], state["case"]
    for s, v in enumerate(state["given"]):
        ctx.upload_n(s, v, state["count"][s])
    energy = []
    for _ in range(case["steps"]):
        ctx.step(DT, 1)
        d = ctx.diagnostics()
        energy.append((d["field_energy"], d["kinetic_energy"]))
    return {"energy": torch.tensor(energy, dtype=state["dtype"]), "particles": _particles(state)}


def _run_modules(state):
    """mainstep as the reference writes it, one module at a time over every particle."""
    ctx, case = state["ctx"], state["case"]
    scatter, solver, interp = P.Scatter(ctx), P.FieldSolver(ctx), P.Interpolator(ctx)
    mover = P.create_particle_mover("boris", ctx)
    felt = []
    for _ in range(case["steps"]):
        scatter.scatter_all()
        solver.solve()
        felt = [torch.from_numpy(interp.interp_all(s)).to(state["dtype"]) for s in range(len(state["count"]))]
        mover.move_all(DT)
    out = _fields(state)
    out["felt"] = felt
    out["particles"] = _particles(state)
    return out


# ---------------------------------------------------------------------------
# Bounded field solve
# ---------------------------------------------------------------------------
KINDS = {"periodic": P.BC_PERIODIC, "dirichlet": P.BC_DIRICHLET, "neumann": P.BC_NEUMANN,
         "dirichlet_neumann": P.BC_DIRICHLET_NEUMANN, "neumann_dirichlet": P.BC_NEUMANN_DIRICHLET}


def _kinds(case):
    return case["kx"], case["ky"], case["kz"]


def _rho(case, seed):
    """Charge of a plasma on the block: a few smooth humps and the particles' noise."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    nx, ny, nz = _grid(case)
    x, y, z = (torch.linspace(0.0, 1.0, v + 1, dtype=torch.float64, device="cuda") for v in (nx, ny, nz))
    rho = 0.2 * torch.randn(nz + 1, ny + 1, nx + 1, generator=g, device="cuda", dtype=torch.float64)
    for _ in range(4):
        a = torch.rand(4, generator=g, device="cuda", dtype=torch.float64).tolist()
        rho += (a[3] - 0.5) * (torch.exp(-30.0 * (z - a[2]) ** 2)[:, None, None] *
                               torch.exp(-30.0 * (y - a[1]) ** 2)[None, :, None] *
                               torch.exp(-30.0 * (x - a[0]) ** 2)[None, None, :])
    for d, k in enumerate(_kinds(case)):   # node n of a periodic axis is node 0
        if k == "periodic":
            rho.select(2 - d, -1).copy_(rho.select(2 - d, 0))
    return rho.contiguous()


def _prepare_poisson(case, seed):
    table = P.TABLE_CORRECTED if case["table"] == "corrected" else P.TABLE_AS_WRITTEN
    rho = _rho(case, seed)
    return {"case": case, "rho": rho, "solver": P.PoissonSolver(_grid(case), [KINDS[k] for k in _kinds(case)],
                                                                table=table)}


def _run_poisson(state):
    rho = state["rho"]
    phi = torch.empty_like(rho)
    e = torch.empty((3,) + tuple(rho.shape), dtype=rho.dtype, device=rho.device)
    state["solver"].solve_device(rho.data_ptr(), phi.data_ptr(), e.data_ptr(), torch.cuda.current_stream().cuda_stream)
    return {"phi": phi, "e": e}


# ---------------------------------------------------------------------------
# Serving
# ---------------------------------------------------------------------------
def _requests(case, seed):
    """The first runs of the serving stream; the seed picks their particles, not their sizes."""
    reqs = serve.ensemble_stream(case["runs"], step_scale=case["step_scale"])
    for i, r in enumerate(reqs):
        r.keep_fields = True
        r.seed = (int(seed), 52 + i)
    return reqs


def _prepare_serve(case, seed):
    # the server holds at most 24 runs of 64^3 x 128 particles: 24 x 2.2 GB
    return {"case": case, "requests": _requests(case, seed),
            "server": serve.Server(weights=P.WEIGHTS_STANDARD, hbm_budget=64 << 30)}


def _run_serve(state):
    server = state["server"]
    ids = [server.submit(r) for r in state["requests"]]
    server.wait()
    out = []
    for i, r in zip(ids, state["requests"]):
        res = server.result(i, r)
        server.release(i)
        out.append(torch.from_numpy(np.stack([res["fields"][k] for k in ("rho", "phi", "ex", "ey", "ez")])).float())
    return out


# ---------------------------------------------------------------------------
# Work: bytes and operations of one pass
# ---------------------------------------------------------------------------
def _step_work(n, particles, steps, es):
    """Each step reads and writes every particle (FP32 form 28 bytes, FP64 form 48), and per cell writes and
    reads rho, phi, the spectrum and E."""
    cells = math.prod(n)
    per_particle = 2 * (28 if es == 4 else 48)
    return {"bytes": steps * (particles * per_particle + cells * 18 * es),
            "flops": steps * (particles * 170 + cells * 10 * math.log2(max(cells, 2)))}


def work(case):
    n = None if case["kind"] == "serve" else _grid(case)
    if case["kind"] == "poisson":
        nodes = math.prod(v + 1 for v in n)
        return {"bytes": 40 * nodes, "flops": 10 * nodes * math.log2(nodes)}
    if case["kind"] == "serve":
        total = {"bytes": 0.0, "flops": 0.0}
        for r in _requests(case, 1):
            w = _step_work(r.n, r.particles(), r.nsteps, 4)
            total = {k: total[k] + w[k] for k in total}
        return total
    count = _count(case)
    w = _step_work(n, count, case["steps"], 4 if case["precision"] == "fp32" else 8)
    if case["kind"] == "job":
        w["bytes"] += 2 * 48 * count
    elif case["kind"] == "modules":
        w["bytes"] += case["steps"] * 24 * count
    return w


# ---------------------------------------------------------------------------
# The same in plain torch, 64 bits
# ---------------------------------------------------------------------------
class _Plasma:
    """Scatter, periodic solve, interpolation and Boris move of every particle."""

    def __init__(self, case, seed):
        self.n = _grid(case)
        self.sp = _species(case)
        self.b = case["wce"]
        self.floor_takes_r = case["weights"] == "reference"   # linear_scatter.f90:41-42
        self.parts = [torch.stack([p[k] for k in NAMES]) for p in _arrays(case, seed)]
        nx, ny, nz = self.n

        def wave(n, count):
            k = torch.arange(count, dtype=torch.float64, device="cuda")
            return (2.0 * torch.sin(REF_PI * torch.minimum(k, n - k) / n)) ** 2

        lam = wave(nz, nz)[:, None, None] + wave(ny, ny)[None, :, None] + wave(nx, nx // 2 + 1)[None, None, :]
        lam[0, 0, 0] = math.inf
        self.green = 1.0 / lam

    def corners(self, p):
        """(node index, weight) of a particle's eight corners."""
        nx, ny, nz = self.n
        low = torch.floor(p[:3])
        r = p[:3] - low
        low = low.long()
        w = (r, 1.0 - r) if self.floor_takes_r else (1.0 - r, r)
        for dz in (0, 1):
            iz = (low[2] + dz) % nz
            for dy in (0, 1):
                iy = (low[1] + dy) % ny
                for dx in (0, 1):
                    yield (low[0] + dx) % nx + nx * (iy + ny * iz), w[dx][0] * w[dy][1] * w[dz][2]

    def scatter(self):
        nx, ny, nz = self.n
        rho = torch.zeros(nx * ny * nz, dtype=torch.float64, device="cuda")
        for s, p in zip(self.sp, self.parts):
            for at, w in self.corners(p):
                rho.index_add_(0, at, s[1] * w)
        self.rho = rho.view(nz, ny, nx)

    def solve(self):
        self.phi = torch.fft.irfftn(torch.fft.rfftn(self.rho) * self.green, s=self.rho.shape)
        self.e = [0.5 * (self.phi.roll(1, 2 - d) - self.phi.roll(-1, 2 - d)) for d in range(3)]

    def felt(self, p):
        out = torch.zeros(3, p.shape[1], dtype=torch.float64, device="cuda")
        for at, w in self.corners(p):
            for d in range(3):
                out[d] += self.e[d].reshape(-1)[at] * w
        return out

    def move(self, s, p, e):
        qm = self.sp[s][0]
        h = e * (0.5 * DT * qm)
        t = 0.5 * DT * qm * self.b                       # B along z
        sn = 2.0 * t / (1.0 + t * t)
        u = p[3:] + h
        ux, uy = u[0] + u[1] * t, u[1] - u[0] * t
        p[3:] = u + h
        p[3] += uy * sn
        p[4] -= ux * sn
        for d in range(3):
            p[d] = torch.remainder(p[d] + p[3 + d] * DT, float(self.n[d]))
            p[d][p[d] >= self.n[d]] = 0.0

    def step(self):
        self.scatter()
        self.solve()
        fields = [self.felt(p) for p in self.parts]
        for s, p in enumerate(self.parts):
            self.move(s, p, fields[s])
        return fields

    def energies(self, fields):
        kinetic = sum(0.5 * s[1] / s[0] * float((p[3:] ** 2).sum()) for s, p in zip(self.sp, self.parts))
        return 0.5 * float(sum((e ** 2).sum() for e in fields)), kinetic


def exact(case, seed):
    if case["kind"] == "poisson":
        return _exact_poisson(case, seed)
    # served runs and the largest start from the device injector
    if case["kind"] == "serve" or not _uploaded(case) or _count(case) * case["steps"] > MOST_EXACT:
        return None
    w = _Plasma(case, seed)
    energy, felt = [], []
    for _ in range(case["steps"]):
        felt = w.step()
        if case["kind"] == "job":
            energy.append(w.energies(w.e))
    parts = [_particle(p, w.n, torch.float64) for p in w.parts]
    if case["kind"] == "job":
        return {"energy": torch.tensor(energy, dtype=torch.float64), "particles": parts}
    w.scatter()
    w.solve()
    out = {"rho": w.rho, "phi": w.phi, "ex": w.e[0], "ey": w.e[1], "ez": w.e[2], "particles": parts}
    if case["kind"] == "modules":
        out["felt"] = [f.t().contiguous() for f in felt]
    return out


def _axis(kind, n, corrected):
    """(first node, forward matrix, backward matrix, normaliser, table) of one axis: FFTW's real-to-real
    definitions and the reference's wave numbers (mpi_fftw3_solver.f90:151-207, poisson_solver3d.f90:104-132)."""
    def grid(L):
        i = torch.arange(L, dtype=torch.float64, device="cuda")
        return i[:, None], i[None, :], i

    if kind == "periodic":
        L, first, norm = n, 0, float(n)
        k, j, i = grid(L)
        turn = 2.0 * math.pi * torch.remainder(k * j, L) / L
        fwd = torch.where(k <= L // 2, torch.cos(turn), torch.sin(turn))   # row L-m: Im F_m = -sin(m..) = sin((L-m)..)
        twice = torch.where((j == 0) | (2 * j == L), 1.0, 2.0)
        bwd = torch.where(j <= L // 2, twice * torch.cos(turn), 2.0 * torch.sin(turn))
        eig = (2.0 * torch.sin(REF_PI * torch.minimum(i, n - i) / n)) ** 2
        return first, fwd, bwd, norm, eig
    if kind == "dirichlet":
        L, first, norm = n - 1, 1, 2.0 * n
        k, j, i = grid(L)
        fwd = bwd = 2.0 * torch.sin(math.pi * torch.remainder((j + 1) * (k + 1), 2 * n) / n)
        lap, sq = 2.0 - 2.0 * torch.cos(REF_PI * (i + 1) / n), 2.0 * (torch.cos(REF_PI * (i + 2) / (n + 1)) - 1.0)
    elif kind == "neumann":
        L, first, norm = n + 1, 0, 2.0 * n
        k, j, i = grid(L)
        fwd = bwd = torch.where((j == 0) | (j == n), 1.0, 2.0) * torch.cos(math.pi * torch.remainder(j * k, 2 * n) / n)
        lap, sq = 2.0 - 2.0 * torch.cos(REF_PI * i / n), 2.0 * (torch.cos(REF_PI * i / n) - 1.0)
    else:
        L, first, norm = n, 1 if kind == "dirichlet_neumann" else 0, 2.0 * n
        k, j, i = grid(L)
        half = math.pi / (2 * n)
        if kind == "dirichlet_neumann":   # DST-III forward, DST-II backward
            a = torch.remainder((2 * k + 1) * (j + 1), 4 * n)
            fwd = torch.where(j == L - 1, 1.0, 2.0) * torch.sin(half * a)
            bwd = 2.0 * torch.sin(half * torch.remainder((2 * j + 1) * (k + 1), 4 * n))
        else:                             # DCT-III forward, DCT-II backward
            fwd = torch.where(j == 0, 1.0, 2.0) * torch.cos(half * torch.remainder((2 * k + 1) * j, 4 * n))
            bwd = 2.0 * torch.cos(half * torch.remainder((2 * j + 1) * k, 4 * n))
        lap = 2.0 - 2.0 * torch.cos(REF_PI * (i + 0.5) / n)
        sq = 2.0 * (torch.cos(REF_PI * (i + first + 0.5) / (n + 1)) - 1.0)
    return first, fwd, bwd, norm, lap if corrected else sq ** 2


def _along(m, a, d):
    """Matrix m applied along axis d (0 = x, the last dimension)."""
    return torch.movedim(torch.tensordot(m, a, dims=([1], [2 - d])), 0, 2 - d)


def _exact_poisson(case, seed):
    rho, n, kinds = _rho(case, seed), _grid(case), _kinds(case)
    corrected = case["table"] == "corrected"
    axes = [_axis(k, v, corrected) for k, v in zip(kinds, n)]
    part = tuple(slice(a[0], a[0] + len(a[4])) for a in reversed(axes))
    v = rho[part]
    for d in range(3):
        v = _along(axes[d][1], v, d)
    den = axes[2][4][:, None, None] + axes[1][4][None, :, None] + axes[0][4][None, None, :]
    v = torch.where(den == 0.0, torch.zeros_like(v), v / den)
    if not corrected and all(a[0] == 0 for a in axes):
        v[0, 0, 0] = 0.0
    for d in (2, 1, 0):
        v = _along(axes[d][2], v, d)
    phi = torch.zeros_like(rho)
    phi[part] = v / math.prod(a[3] for a in axes)
    for d, k in enumerate(kinds):
        if k == "periodic":
            phi.select(2 - d, -1).copy_(phi.select(2 - d, 0))
    e = torch.empty((3,) + tuple(phi.shape), dtype=torch.float64, device="cuda")
    for d, k in enumerate(kinds):
        a, m, out = 2 - d, n[d], e[d]
        lo, hi = phi.narrow(a, 0, m - 1), phi.narrow(a, 2, m - 1)
        out.narrow(a, 1, m - 1).copy_(0.5 * (lo - hi))
        if k == "periodic":
            edge = 0.5 * (phi.select(a, m - 1) - phi.select(a, 1))
            out.select(a, 0).copy_(edge)
            out.select(a, m).copy_(edge)
        else:
            out.select(a, 0).copy_(phi.select(a, 0) - phi.select(a, 1))
            out.select(a, m).copy_(phi.select(a, m - 1) - phi.select(a, m))
    return {"phi": phi, "e": e}
