"""Independent handles on grids of different sizes, stepped in different host
threads.  The shared-memory limit of a kernel belongs to the function, not to a
handle: whatever one handle's launch asks for, another's must still be accepted,
and each handle's fields are those of the same steps taken alone."""
import threading

import numpy as np
import pytest

from conftest import package

pytestmark = pytest.mark.gpu

# the same kernel instances at two shared-memory sizes: SOR in one block;
# resident BiCGStab with the actuator line; the cluster V-cycle with it
CASES = [("tiny-sor", (24, 12, 12), (10, 6, 6), False), ("tiny-sorpc", (40, 30, 30), (12, 8, 8), False),
         ("tiny-turbine", (200, 20, 20), (40, 20, 20), False), ("tiny-loglaw", (64, 32, 32), (32, 16, 20), True)]
STEPS = 150


@pytest.mark.parametrize("name,large,small,mixed", CASES)
def test_two_grids_in_two_threads(make_case, tmp_path, name, large, small, mixed):
    pkg = package()

    def solver(n):
        spec, mesh, d, U0, prof = make_case(name, n=n, dt=1e-4, max_it=2)
        s = pkg.Solver(d, precision=pkg.MIXED if mixed else pkg.FP64)
        s.set_inflow_profile(prof)
        s.set_state(U0)
        return s

    def run(s, errors):
        try:
            for _ in range(STEPS):
                s.step(1)
        except Exception as e:  # reported in the main thread
            errors.append(e)

    alone, errors = [], []
    for n in (large, small):
        s = solver(n)
        run(s, errors)
        alone.append((s.field("U"), s.field("p")))
        s.finalize()
    assert not errors
    pair = [solver(n) for n in (large, small)]
    threads = [threading.Thread(target=run, args=(s, errors)) for s in pair]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    for s, (U, p) in zip(pair, alone):
        np.testing.assert_array_equal(s.field("U"), U)
        np.testing.assert_array_equal(s.field("p"), p)
        s.finalize()
