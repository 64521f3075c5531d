"""DALM_TRACE_POISSON: =1 a line per pressure solve, =2 also one per batch of
its iterations, whatever route the solve takes without it."""
import pytest

from conftest import package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["tiny-sor", "tiny-jacobi", "tiny-bicg", "tiny-sorpc"])
@pytest.mark.parametrize("level", ["1", "2"])
def test_trace_lines(make_case, monkeypatch, capfd, name, level):
    pkg = package()
    spec, mesh, d, U0, prof = make_case(name, n=(40, 20, 20), dt=1e-4, max_it=60, tol=0.0)
    monkeypatch.setenv("DALM_TRACE_POISSON", level)
    s = pkg.Solver(d, poisson_batch=5)
    s.set_state(U0)
    s.step(3)
    s.finalize()
    err = capfd.readouterr().err.splitlines()
    assert sum("poisson it" in r for r in err) == 2
    batches = [int(r.split("solve 0: ")[1].split()[0]) for r in err if "iterations, residual" in r]
    if level == "1":
        assert not batches
    else:
        assert len(batches) >= 6 and batches[0] <= 8
