"""The run-out of every kind of line wait, on domains chosen so that the launch that has it
is the one that runs (test_launch_names.py has them by name): the pipelined red-black passes (rows of more cells
than the launch with every line in a warp takes), the passes with every line in a warp, the
exact order by rows, and by single visits (rows past 128 cells).  With a budget of one poll
the solve gives up, the step fails with AMCFD_E_TIMEOUT, and fresh solvers in the
same process agree bit for bit.  (The momentum chain's waits: test_chain_waits.py.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

E_TIMEOUT = -6


@pytest.mark.parametrize("order,prec,nx,ny,nz", [
    (1, 1, 530, 12, 9), (1, 0, 270, 13, 9), (1, 2, 530, 13, 9),  # pipelined
    (1, 1, 60, 13, 9), (1, 0, 130, 12, 9), (1, 2, 60, 12, 9),    # every line in a warp
    (0, 0, 60, 13, 9), (0, 0, 140, 13, 9), (0, 1, 140, 12, 9)])  # rows; single visits
@pytest.mark.parametrize("graphs", [0, 1])
def test_budget_of_one_poll_runs_out(graphs, order, prec, nx, ny, nz, tmp_path):
    import amcfd
    import amcfd_decks as D
    d = amcfd.Deck(D.small("wait", nx=nx, ny=ny, nz=nz, steps=2).write(str(tmp_path)))
    s = amcfd.Solver(d, order=order, precision=prec, use_graphs=graphs, wait_polls=1)

    def fails():
        with pytest.raises(amcfd.AmcfdError) as e:
            s.step()
        assert e.value.code == E_TIMEOUT, str(e.value)
        assert "device wait gave up" in str(e.value)

    fails()
    fails()  # the context keeps the error
    s.close()
    a = amcfd.Solver(d, order=order, precision=prec, use_graphs=graphs)
    b = amcfd.Solver(d, order=order, precision=prec, use_graphs=0)
    for _ in range(2):
        ra, rb = a.step(), b.step()
        assert ra["niter"] == rb["niter"]
    for f in ("temp", "uvel", "vvel", "wvel", "pressure", "enthalpy"):
        assert np.array_equal(a.get(f), b.get(f)), f
    a.close()
    b.close()
