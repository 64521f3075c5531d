"""Which route a solve takes, by the number of launches, and that a device that
refuses a resident solve's blocks (DALM_SM_COUNT plans for more multiprocessors
than it has) leaves it to the launched kernels."""
import pytest

from conftest import package
from test_gpu_resident import agree

pytestmark = pytest.mark.gpu

# as in test_gpu_resident.py: SOR and Jacobi contract, BiCGStab amplifies the
# rounding of its sums
CASES = [("tiny-sor", (97, 80, 79), 20, 1e-12), ("tiny-jacobi", (97, 80, 79), 20, 1e-12),
         ("tiny-bicg", (131, 75, 53), 3, 1e-11), ("tiny-sorpc", (97, 80, 79), 3, 1e-11)]


def solve(make_case, name, n, its, **options):
    spec, mesh, d, U0, prof = make_case(name, n=n, dt=1e-4, turbines=[], loglaw=None)
    s = package().Solver(d, **options)
    s.set_state(U0)
    s.set_poisson(its, 0.0)
    s.step(2)
    s.timings(reset=True)
    s.step(1)
    launches = s.timings()[1]
    st = s.stats()
    out = st["it"], st["err"], s.field("U"), s.field("p")
    s.finalize()
    return out, launches


@pytest.mark.parametrize("name,n,its,tol", CASES)
def test_refused_launch(make_case, monkeypatch, name, n, its, tol):
    resident, few = solve(make_case, name, n, its)
    monkeypatch.setenv("DALM_SM_COUNT", "400")
    refused, many = solve(make_case, name, n, its)
    assert few <= 12  # one launch for the solve, the rest of the step beside it
    assert many >= 2 * its
    agree(refused, resident, tol)


# the cluster V-cycle against one launch per half-sweep, of which a V-cycle has
# two per smoothing step and side on every level
@pytest.mark.parametrize("n", [(64, 32, 40), (48, 24, 100)])
def test_cluster_route(make_case, n):
    pkg = package()
    spec, mesh, d, U0, prof = make_case("tiny-loglaw", n=n, dt=1e-4)
    count = []
    for profile in (False, True):
        s = pkg.Solver(d, precision=pkg.MIXED, profile=profile)
        s.set_inflow_profile(prof)
        s.set_state(U0)
        s.step(2)
        s.timings(reset=True)
        s.step(1)
        count.append(s.timings()[1])
        s.finalize()
    assert count[0] < 0.6 * count[1], count


@pytest.mark.parametrize("name", ["tiny-sor", "tiny-jacobi", "tiny-bicg", "tiny-sorpc"])
@pytest.mark.parametrize("cap", [-1500, -1, 0, 1])
def test_smallest_caps(make_case, monkeypatch, capfd, name, cap):
    """A loop tests its cap after an iteration, so one is always done: launched,
    resident, and resident with the host waiting for it (a trace)."""
    its = []
    for options, trace in (({"profile": True}, "0"), ({}, "0"), ({}, "1")):
        monkeypatch.setenv("DALM_TRACE_POISSON", trace)
        its.append(solve(make_case, name, (24, 12, 12), cap, **options)[0][0])
    assert its == [1, 1, 1]
