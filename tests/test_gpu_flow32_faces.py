"""The mixed form's flux and projection kernels (flow_mixed.cu) on every face
they own, the layer below the interior included, against the FP64 form's on the
same values.

Fluxes: u A with u and the two spacings of A rounded to FP32, the area's
product, the two face products and their sum: each face is within seven FP32
roundings (2^-24 each) of the larger of its two products.  Projection: both
forms get the same FP32 fluxes, velocity and FP64 pressure and compute in FP64,
the mixed form rounding once at the store; 1e-13 of the largest magnitude
covers the FP64 roundings (the reciprocal tables differ from the quotients by a
unit in the last place)."""
import numpy as np
import pytest

from conftest import package

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24

# tiles of 32 x 8 exactly, partial in k and j, one cell over, one tile, and
# several chunks of planes
SIZES = [(32, 16, 64), (33, 9, 31), (40, 25, 33), (16, 8, 20), (70, 17, 65)]


def faces(a):
    """Faces and cells from one below the interior (two guide cells) up."""
    return a[1:-2, 1:-2, 1:-2]


@pytest.mark.parametrize("n", SIZES)
def test_faces_and_projection(make_case, n):
    pkg = package()
    spec, mesh, d, U0, prof = make_case("tiny-loglaw", n=n, dt=1e-4)
    m, f = pkg.Solver(d, precision=pkg.MIXED), pkg.Solver(d)
    rng = np.random.default_rng(3)
    U = (U0 + 0.1 * rng.standard_normal(U0.shape)).astype(np.float32).astype(np.float64)
    for s in (m, f):
        s.set_inflow_profile(prof)
        s.set_state(U)
    dx = f.mesh()[3:6]
    Ju, Jf, Uf = m.field("JU"), f.field("JU"), f.field("U")
    for a in range(3):
        b, c = [q for q in range(3) if q != a]
        shape = [1, 1, 1]
        shape[b], shape[c] = -1, 1
        area = dx[b].reshape(shape)
        shape[b], shape[c] = 1, -1
        area = area * dx[c].reshape(shape)
        big = np.maximum(np.abs(Uf[..., a]), np.abs(np.roll(Uf[..., a], -1, a))) * area
        # (an inflow face is the profile's velocity times the area)
        big = np.maximum(big, np.abs(Jf[..., a]))
        assert np.all(faces(np.abs(Ju[..., a] - Jf[..., a])) <= faces(7 * EPS * big))
    p = rng.standard_normal(f.field("p").shape)
    f.set_field("U", m.field("U"))
    f.set_field("JU", Ju)
    for s in (m, f):
        s.set_field("p", p)
        s.stage("project")
    for name in ("JU", "U"):
        x, y = faces(m.field(name)), faces(f.field(name))
        if name == "U":  # cells of the interior
            x, y = x[1:, 1:, 1:], y[1:, 1:, 1:]
        assert np.all(np.abs(x - y) <= EPS * np.abs(y) + 1e-13 * np.abs(y).max())
    m.finalize()
    f.finalize()
