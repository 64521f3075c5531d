"""Bit identity with the oracle at the ends of the double range.

Quotients by mesh spacings are formed from tabulated reciprocals; they are the
reference's quotients for every dividend: values whose remainders are subnormal
(below 2^-968), subnormal values, and values whose quotient overflows."""
import numpy as np
import pytest

from conftest import package
from test_gpu_parity import assert_identical
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-285, 1e-293, 1e-300, 1e-307, 1e-315, 1e307])
def test_stage_bits(make_case, scale):
    spec, mesh, d, U0, prof = make_case("tiny-sor", n=(40, 12, 40))
    rng = np.random.default_rng(7)
    U = np.zeros(U0.shape)
    U[2:-2, 2:-2, 2:-2] = scale * rng.uniform(-1, 1, U[2:-2, 2:-2, 2:-2].shape)
    U[..., 0] += 1.0 if scale < 1 else 0.0
    p = scale * rng.uniform(-1, 1, U.shape[:3])
    s, o = package().Solver(d, reference_sums=True), O.CRestatement(d)
    with np.errstate(all="ignore"):
        for x in (s, o):
            x.advance_clock()
            x.set_state(U)
        for x in (s, o):
            x.stage(0)
        assert_identical(s, o, ("U",), "predict")
        for x in (s, o):
            x.stage(1)
        assert_identical(s, o, ("JU", "b"), "flux_rhs")
        for x in (s, o):
            x.set_field("p", p)
            x.stage(3)
        assert_identical(s, o, ("U", "JU", "p"), "project")
    s.finalize()
    o.close()


@pytest.mark.parametrize("limiter", [0, 1])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_stage_bits_around_a_bad_cell(make_case, bad, limiter):
    """What a cell that is not finite makes of its neighbours: the reference's
    limiter takes the smaller of two differences and ignores one that is NaN."""
    spec, mesh, d, U0, prof = make_case("tiny-sor", n=(40, 12, 40))
    U, p = U0.copy(), np.random.default_rng(7).uniform(-1, 1, U0.shape[:3])
    U[20, 8, 19, 1] = bad
    U[30, 5, 35] = bad
    p[12, 9, 30] = bad
    s, o = package().Solver(d, reference_sums=True, limiter=limiter), O.CRestatement(d)
    o.set_limiter(limiter)
    for x in (s, o):
        x.advance_clock()
        x.set_state(U)
        x.stage(0)
    assert not np.all(np.isfinite(o.field("U")))
    assert_identical(s, o, ("U",), "predict")
    for x in (s, o):
        x.stage(1)
    assert_identical(s, o, ("JU", "b"), "flux_rhs")
    for x in (s, o):
        x.set_field("p", p)
        x.stage(3)
    assert_identical(s, o, ("U", "JU", "p"), "project")
    s.finalize()
    o.close()
