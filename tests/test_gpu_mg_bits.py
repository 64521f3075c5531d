"""The cluster V-cycle gives the launched half-sweeps' bits (profile=True keeps
those): where the stop leaves the pressure loose, as with 128 cells along z at a
small time step, another rounding in the preconditioner shows in it."""
import numpy as np
import pytest

from conftest import package

pytestmark = pytest.mark.gpu

# one to four rows per lane, columns that fill their lanes' rows and columns
# that do not, levels that merge along z
SIZES = [((64, 32, 32), 5e-4), ((32, 16, 20), 5e-4), ((64, 32, 40), 5e-4), ((48, 20, 72), 5e-4),
         ((48, 24, 100), 1e-4), ((64, 64, 128), 1e-4)]


@pytest.mark.parametrize("n,dt", SIZES)
def test_cluster_cycle_bits(make_case, n, dt):
    pkg = package()
    spec, mesh, d, U0, prof = make_case("tiny-loglaw", n=n, dt=dt)
    out = []
    for profile in (False, True):
        s = pkg.Solver(d, precision=pkg.MIXED, profile=profile)
        s.set_inflow_profile(prof)
        s.set_state(U0)
        s.step(3)
        out.append((s.field("U"), s.field("p"), s.stats()["it"]))
        s.finalize()
    assert out[0][2] == out[1][2]
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
