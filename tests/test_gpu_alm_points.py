"""Actuator lines with thousands of blade points: the projection lists a block's
points in shared memory beside its tables, whatever their number.

The force field against the oracle's untruncated serial sum.  A cell sums up to
n terms of one sign pattern, each within a few roundings u = 2^-53 of the
oracle's: n u = 12600 u = 1.4e-12 bounds the sum's, and the truncated far terms
are below u of the largest."""
import numpy as np
import pytest

from conftest import package
from test_gpu_parity import rel
import oracle as O

pytestmark = pytest.mark.gpu


# the last count whose list fits the default limit beside the tables, the first
# that does not, the last below a list of 32 KB, and one whose points' sums are
# not staged in shared memory
@pytest.mark.parametrize("points", [2237, 2238, 2730, 4200])
def test_many_points(make_case, points):
    spec, mesh, d, U0, prof = make_case("tiny-turbine", n=(24, 12, 12), points_per_blade=points)
    s, o = package().Solver(d), O.CRestatement(d)
    assert s.point_count == 3 * points
    for x in (s, o):
        x.set_state(U0)
    assert np.linalg.norm(o.field("f")) > 0
    assert rel(s.field("f"), o.field("f")) <= 2e-12
    s.finalize()
    o.close()
