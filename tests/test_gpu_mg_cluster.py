"""The cluster form of the multigrid V-cycle (multigrid_cluster.cu) against the
launched half-sweeps, which profile=True keeps.

Both do the same FP32 operations up to contraction, so a solve takes the same
number of conjugate-gradient iterations (one more or less where a residual
falls on the stop), and both forms are held to the envelope the mixed form is
held to against FP64: U within 1e-6 and p within 1e-2 over the steps, every
residual within the tolerance."""
import numpy as np
import pytest

from conftest import package
from test_gpu_parity import rel

pytestmark = pytest.mark.gpu

# whole cycles in the cluster and cycles whose finest levels stay launches; one
# to four rows per lane, columns that end inside a lane's rows, levels that
# merge along z, and planes and columns fewer than blocks and warps
SIZES = [(32, 16, 20), (16, 8, 57), (64, 32, 40), (48, 20, 72), (32, 16, 128), (128, 64, 32)]


@pytest.mark.parametrize("n", SIZES)
def test_cluster_cycle_matches_launches(make_case, n):
    pkg = package()
    spec, mesh, d, U0, prof = make_case("tiny-loglaw", n=n, dt=5e-4 if n[2] <= 80 else 1e-4)
    out = []
    for profile in (False, True):
        s = pkg.Solver(d, precision=pkg.MIXED, profile=profile)
        s.set_inflow_profile(prof)
        s.set_state(U0)
        steps = []
        for _ in range(4):
            s.step(1)
            steps.append(s.stats())
        out.append((steps, s.field("U"), s.field("p")))
        s.finalize()
    (sa, Ua, pa), (sb, Ub, pb) = out
    for a, b in list(zip(sa, sb))[1:]:
        assert a["err"] <= spec.tol and b["err"] <= spec.tol
        assert abs(a["it"] - b["it"]) <= 1
    assert rel(Ua, Ub) <= 1e-6
    assert rel(pa, pb) <= 1e-2
