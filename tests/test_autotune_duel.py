"""The autotuner's second meeting of near-ties, driven by fake contexts that heat.

Every step makes the plasma's pushes slower, so a tile shape timed late in the pass looks
slower than it is; on a fresh plasma (16,8,8) wins by 2%.  The fake device has room for one
context, as it has when the grid itself is tuned."""
import pytest

P = pytest.importorskip("ohhelppic3d_gb300")
from ohhelppic3d_gb300 import autotune as A  # noqa: E402

HALO = {1: 0.0, 2: 0.5, 3: 1.0}
TILE = {(8, 8, 8): 11.0, (16, 8, 8): 10.78}


class Hot:
    alive = made = 0

    def __init__(self, cold=False):
        if Hot.alive:
            raise P.OhpicError(P.ERR_OOM, "out of memory")
        Hot.alive += 1
        Hot.made += 1
        self.open, self.cold = True, cold
        self.t = {"tile": (8, 8, 8), "halo": 1, "split": 0, "deposit": P.DEPOSIT_LANES, "lane_particles": 4,
                  "sort_every": 0, "sort_lead": 0}
        self.age = self.push_ms = self.push_launches = 0
        self.timing = False

    def get_tuning(self):
        return dict(self.t)

    def set_tuning(self, **kw):
        assert self.open
        self.t = {**self.t, **kw}

    def sort(self):
        pass

    def step(self, dt, n=1):
        assert self.open
        for _ in range(n):
            cost = TILE.get(tuple(self.t["tile"]), 14.0) + HALO[self.t["halo"]] + 0.1 * self.t["sort_lead"]
            cost += 0.0 if self.t["deposit"] == P.DEPOSIT_LANES and self.t["lane_particles"] == 4 else 3.0
            cost += 0.0 if self.t["split"] < 2 else 1.0
            self.push_ms += (cost + (0.0 if self.cold else 0.004 * self.age)) if self.timing else 0.0
            self.push_launches += self.timing
            self.age += 1

    def set_push_timing(self, on):
        self.timing, self.push_ms, self.push_launches = bool(on), 0.0, 0

    def stats(self):
        return {"push_ms": self.push_ms, "push_launches": self.push_launches, "launches": 0}

    def synchronize(self):
        pass

    def close(self):
        if self.open:
            self.open = False
            Hot.alive -= 1


@pytest.mark.parametrize("cold", [False, True])
@pytest.mark.parametrize("proxy", [False, True])
def test_near_ties_meet_on_a_fresh_plasma_one_context_at_a_time(monkeypatch, proxy, cold):
    Hot.alive = Hot.made = 0
    monkeypatch.setattr(A, "_ctx", lambda cfg_kw, species, seed=(42, 4242): Hot(cold))
    monkeypatch.setattr(A, "_sort_ms", lambda ctx: 1.0)
    best = A.tune(n=(64, 32, 32), dt=0.1, b0=(0, 0, 0.5), qm=[-1.0], q=[1.0], capacity_per_cell=[9.0], species=[None],
                  steps=6, max_cadence=5, proxy=proxy)
    assert tuple(best["tile"]) == (16, 8, 8) and best["halo"] == 1 and best["split"] == 1
    assert Hot.alive == 0
    # a plasma that does not heat shows the difference in the pass itself
    assert Hot.made == (1 if cold else 3)
    # in the pass the current shape looked better
    seen = {tuple(tr["tile"]): tr["push_ms"] for tr in best["trials"][::-1]
            if tr["halo"] == 1 and tr["sort_lead"] == 0 and tr["deposit"] == P.DEPOSIT_LANES and tr["lane_particles"] == 4}
    assert cold or seen[(16, 8, 8)] > seen[(8, 8, 8)]


class Few(Hot):
    """A grid of few tiles: the more CTAs share a tile, the faster, up to the library's own most."""

    def step(self, dt, n=1):
        super().step(dt, n)
        self.push_ms += n * self.timing * (16.0 / min(max(self.t["split"], 1), 16) - (self.t["split"] > 1))


def test_split_search_reaches_the_librarys_most(monkeypatch):
    Hot.alive = Hot.made = 0
    monkeypatch.setattr(A, "_ctx", lambda cfg_kw, species, seed=(42, 4242): Few(cold=True))
    monkeypatch.setattr(A, "_sort_ms", lambda ctx: 1.0)
    best = A.tune(n=(16, 16, 16), dt=0.1, b0=(0, 0, 0.5), qm=[-1.0], q=[1.0], capacity_per_cell=[9.0], species=[None],
                  steps=6, max_cadence=5)
    assert best["split"] == 16
