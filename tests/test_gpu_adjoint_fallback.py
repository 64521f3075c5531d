"""Adjoint pressure solves that the refinement hands to the FP64 solver: their
statistics are those of the finished solve."""
import pytest

from conftest import casegen, package

pytestmark = pytest.mark.gpu


# cells longer along z, where the smoother solves lines, than along y, and one
# inner iteration per pass: it gains too little and the refinement gives up.
# At most 900 iterations, so that a resident solve takes one launch.
@pytest.mark.parametrize("ly", [2.0, 1.0])
def test_statistics_after_a_handed_over_solve(make_case, ly):
    rotor = casegen().Turbine(base=(4.0, ly / 2, 0.0))
    spec, mesh, d, U0, prof = make_case("tiny-turbine", lengths=(20.0, ly, 5.0), turbines=[rotor], dt=1e-4)
    out = []
    for profile in (False, True):  # True: the solves are launched kernel by kernel and waited for
        s = package().Solver(d, limiter=package().VAN_ALBADA, refine_inner_it=1, profile=profile)
        s.set_poisson(900, 1e-10)
        s.set_state(U0)
        s.power_gradient(1, 2)
        out.append(s.adjoint_stats())
        s.finalize()
    for st in out:
        assert st["solves"] == out[1]["solves"] > 0
        assert 0 < st["max_rel_residual"] <= 1e-10
        # the handed-over solves' iterations among them, some hundred each
        assert st["iterations"] > 50 * st["solves"]
