"""The routes of the FP64 pressure solves against one another.

By default a grid that fits the device is solved by one cooperative kernel
(poisson_resident.cu) and a larger Jacobi(3)-BiCGStab solve by fused
half-iterations (poisson_fused.cu); with profile=True small grids, and with
fused_jacobi=True all grids, run one kernel per reference loop, the form the
parity tests pin to the oracle.  All compute a cell's value with the same
operations up to the order of a few additions, and sums in another order, so a
few iterations from the same state must agree to rounding.

Tolerances.  SOR and Jacobi contract: a relative rounding of 2^-53 per
operation, some ten operations a cell and 60 sweeps stay below 1e-12.
BiCGStab amplifies the rounding of its sums; one iteration of the existing
fused form is held to 1e-13 and five to 1e-10, so three are held to 1e-11.
"""
import numpy as np
import pytest

from conftest import package
from test_gpu_parity import rel

pytestmark = pytest.mark.gpu


def solve(make_case, name, n, its, tol=0.0, **options):
    spec, mesh, d, U0, prof = make_case(name, n=n, dt=1e-4, turbines=[], loglaw=None)
    s = package().Solver(d, **options)
    s.set_state(U0)
    s.set_poisson(its, tol)
    s.step(3)
    st = s.stats()
    out = st["it"], st["err"], s.field("U"), s.field("p")
    s.finalize()
    return out


def agree(a, b, tol):
    assert a[0] == b[0]
    assert abs(a[1] / b[1] - 1) <= 1e3 * tol
    assert rel(a[3], b[3]) <= tol
    assert rel(a[2], b[2]) <= tol


# one block; several blocks with odd sizes and half-filled pairs; the longest
# row pair of a warp; more cells than the registers hold (two sizes)
@pytest.mark.parametrize("n", [(24, 12, 12), (41, 13, 9), (37, 21, 64), (97, 80, 79), (61, 130, 77)])
def test_sor(make_case, n):
    agree(solve(make_case, "tiny-sor", n, 30), solve(make_case, "tiny-sor", n, 30, profile=True), 1e-12)


@pytest.mark.parametrize("n", [(33, 10, 65), (70, 50, 64)])
def test_jacobi(make_case, n):
    agree(solve(make_case, "tiny-jacobi", n, 30), solve(make_case, "tiny-jacobi", n, 30, profile=True), 1e-12)


# the sweep after the last one is computed and dropped: a stop inside the solve,
# at a tolerance just above the residual of 20 iterations
@pytest.mark.parametrize("name,n", [("tiny-sor", (24, 12, 12)), ("tiny-sor", (64, 40, 40)),
                                    ("tiny-sor", (97, 80, 79)), ("tiny-jacobi", (24, 12, 12))])
def test_stop(make_case, name, n):
    spec, mesh, d, U0, prof = make_case(name, n=n, dt=1e-4, turbines=[], loglaw=None)
    out = []
    for options in ({}, {"profile": True}):
        s = package().Solver(d, **options)
        s.advance_clock()
        s.set_state(U0)
        s.stage("predict")
        s.stage("flux_rhs")
        if not out:
            s.set_poisson(20, 0.0)
            s.stage("poisson")
            tol = s.stats()["err"] * (1 + 1e-9)
            s.set_field("p", np.zeros(s.field("p").shape))
        s.set_poisson(200, tol)
        s.stage("poisson")
        st = s.stats()
        assert st["it"] == 20 and st["err"] <= tol
        out.append((st["it"], st["err"], s.field("U"), s.field("p")))
        s.finalize()
    agree(*out, 1e-12)


def test_more_iterations_than_a_launch(make_case):
    agree(solve(make_case, "tiny-sor", (24, 12, 12), 1500),
          solve(make_case, "tiny-sor", (24, 12, 12), 1500, profile=True), 1e-11)


# one, two, four and eight planes a thread, with remainders in each direction
@pytest.mark.parametrize("n", [(9, 7, 5), (63, 41, 40), (91, 60, 51), (103, 77, 70)])
def test_bicg_resident(make_case, n):
    agree(solve(make_case, "tiny-bicg", n, 3), solve(make_case, "tiny-bicg", n, 3, profile=True), 1e-11)


# grids above the resident kernel's: partial tiles in j and k, odd rows, marches
# longer than one chunk, and rows of at most 32 cells (the narrow tile)
@pytest.mark.parametrize("n", [(130, 91, 67), (300, 31, 128), (331, 65, 31), (660, 40, 32)])
def test_bicg_fused(make_case, n):
    agree(solve(make_case, "tiny-bicg", n, 3), solve(make_case, "tiny-bicg", n, 3, fused_jacobi=True), 1e-11)


@pytest.mark.parametrize("n", [(31, 20, 33), (80, 60, 50)])
def test_bicg_sor(make_case, n):
    agree(solve(make_case, "tiny-sorpc", n, 3), solve(make_case, "tiny-sorpc", n, 3, profile=True), 1e-11)


def test_two_handles_in_two_threads(make_case):
    """Cooperative kernels of two handles share the device's SMs in turn."""
    import threading

    spec, mesh, d, U0, prof = make_case("tiny-sor", n=(64, 40, 40), dt=1e-4)
    pkg = package()
    solvers = [pkg.Solver(d) for _ in range(3)]
    for s in solvers:
        s.set_state(U0)
        s.set_poisson(200, 0.0)

    def run(s):
        for _ in range(5):
            s.step(1)

    threads = [threading.Thread(target=run, args=(s,)) for s in solvers[:2]]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    run(solvers[2])
    for f in ("U", "p"):
        want = solvers[2].field(f)
        for s in solvers[:2]:
            np.testing.assert_array_equal(s.field(f), want)
