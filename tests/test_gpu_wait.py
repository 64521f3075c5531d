"""A barrier wait of a resident solve that runs out (DALM_STALL_BARRIERS: it
counts arrivals from a number that they never bring to the goal, and gives up
after its limit of about a second) is reported, by every step, and other handles
are not touched by it."""
import pytest

from conftest import package

pytestmark = pytest.mark.gpu


# one launch's worth of iterations (the step does not wait for the solve), and
# more (it does)
@pytest.mark.parametrize("name,n", [("tiny-sor", (64, 40, 40)), ("tiny-sor", (97, 80, 79)),
                                    ("tiny-jacobi", (64, 40, 40)), ("tiny-bicg", (63, 41, 40)),
                                    ("tiny-sorpc", (64, 40, 40))])
@pytest.mark.parametrize("its", [100, 3000])
def test_wait_runs_out(make_case, monkeypatch, name, n, its):
    pkg = package()
    spec, mesh, d, U0, prof = make_case(name, n=n, dt=1e-4)
    monkeypatch.setenv("DALM_STALL_BARRIERS", "1")
    s = pkg.Solver(d)
    monkeypatch.delenv("DALM_STALL_BARRIERS")
    good = pkg.Solver(d)
    for h in (s, good):
        h.set_state(U0)
        h.set_poisson(its, 0.0)
        h.step(1)  # step 0: no solve
    for _ in range(2):
        with pytest.raises(pkg.DalmError) as e:
            s.step(1)
        assert e.value.code == 5, e.value
        s.stats()  # reported once
    good.step(2)
    assert good.stats()["it"] > 0
    s.finalize()
    good.finalize()


def test_nothing_is_written_of_a_failed_step(make_case, monkeypatch):
    import os

    pkg = package()
    spec, mesh, d, U0, prof = make_case("tiny-sor", n=(64, 40, 40), dt=1e-4, output_start_time=0.0,
                                        output_interval_time=1e-4, probes=[[5.0, 2.5, 1.0]])
    monkeypatch.setenv("DALM_STALL_BARRIERS", "1")
    s = pkg.Solver(d, write_output=True)
    s.set_state(U0)
    s.step(1)
    out = os.path.join(d, "output")
    before = sorted(os.listdir(out))
    with pytest.raises(pkg.DalmError) as e:
        s.step(3)
    assert e.value.code == 5
    assert sorted(os.listdir(out)) == before
    s.finalize()
    with open(os.path.join(out, "probe0.csv")) as f:
        assert len([r for r in f if r[0].isdigit()]) == 1  # step 0
