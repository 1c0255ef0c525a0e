"""Blocks whose edges hold a large prime factor R, which costs the bounded solve's own passes
R operations an element: they take no longer for a node than blocks with the next prime,
which go through cuFFT as every block did before the passes."""
import pytest

pytestmark = pytest.mark.gpu


def _ns_per_node(P, torch, n, kind):
    solver = P.PoissonSolver(n, [kind] * 3, table=P.TABLE_CORRECTED)
    shape = tuple(v + 1 for v in reversed(n))
    rho = torch.randn(shape, dtype=torch.float64, device="cuda")
    phi, e = torch.empty_like(rho), torch.empty((3,) + shape, dtype=torch.float64, device="cuda")
    best = float("inf")
    for _ in range(6):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(8):
            solver.solve_device(rho.data_ptr(), phi.data_ptr(), e.data_ptr(), torch.cuda.current_stream().cuda_stream)
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 1e6 / 8)
    passes = solver.plan()["pairs"][0] > 0
    solver.close()
    return best / rho.numel(), passes


@pytest.mark.parametrize("kind", ["PERIODIC", "DIRICHLET", "NEUMANN"])
def test_passes_of_large_primes_are_no_slower_than_cufft(ohpic, kind):
    P = ohpic
    torch = pytest.importorskip("torch")
    kind = getattr(P, "BC_" + kind)
    own, passes = _ns_per_node(P, torch, (201, 67, 67), kind)
    library, other = _ns_per_node(P, torch, (213, 71, 71), kind)
    assert passes and not other
    assert own <= library, (own, library)
