"""Which steps of a small grid run as a replayed graph: every step whose arguments are those
of the capture, after one capture.  The comparisons of replayed with plain steps rest on it:
where no step was replayed they would pass all the same."""
import pytest

from test_step_graph import _context, _plain, _same

pytestmark = pytest.mark.gpu


def _counts(ctx):
    s = ctx.graph_stats()
    return s["replays"], s["captures"]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_steps_are_replayed_after_one_capture(ohpic, precision):
    P = ohpic
    with _context(P, P.FP64 if precision == "fp64" else P.FP32) as ctx:
        ctx.step(0.1, 1)                        # the first deposit, the push of the sort's records
        assert _counts(ctx) == (0, 0)
        ctx.step(0.1, 3)
        assert _counts(ctx) == (3, 1)
        per_cycle = 3 if precision == "fp32" else 4
        ctx.step(0.1, 40)                       # ten cycles: all but the push of each sort's records
        assert _counts(ctx) == (3 + 10 * per_cycle, 1)
        ctx.step(0.05, 4)                       # another length: another capture
        assert _counts(ctx) == (3 + 11 * per_cycle, 2)
        ctx.set_push_timing(True)               # timed steps launch plainly
        ctx.step(0.05, 4)
        assert _counts(ctx) == (3 + 11 * per_cycle, 2)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_steps_of_changing_length_match_plain_ones(ohpic, precision):
    P = ohpic
    prec = P.FP64 if precision == "fp64" else P.FP32
    with _context(P, prec) as a, _context(P, prec) as b:
        since = 0
        for i in range(12):
            dt = 0.1 * 0.99 ** i if i < 8 else (0.1, 0.09)[i % 2]
            a.step(dt, 1)
            since = _plain(b, dt, since, 4)
        replays, captures = _counts(a)
        assert replays == captures == (9 if precision == "fp32" else 11)
        assert _counts(b) == (0, 0)
        _same(P, a, b)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_larger_grids_launch_plainly(ohpic, precision):
    P = ohpic
    with _context(P, P.FP64 if precision == "fp64" else P.FP32, n=(129, 64, 32), ppc=1) as ctx:
        ctx.step(0.1, 6)
        assert _counts(ctx) == (0, 0)
