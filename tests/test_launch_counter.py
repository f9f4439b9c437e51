"""The solver's launch counter (amcfd_kernel_launches) against the kernels that the profiler
sees, a step of direct launches at a time, in every form that launches differently."""
import pytest

from kernel_names import launched

pytestmark = pytest.mark.gpu

# the network's own kernels are not the solver's launches
NET = ("conv_tc", "pack_fwd", "pack_bwd", "features_kernel", "reduce_parts", "wgrad", "bgrad", "mse", "adam")


def _count(s):
    """Two steps: the counter's increase and the launches seen in each."""
    out = []
    for _ in range(2):
        c = s.launches
        n = launched(s.step)
        out.append((s.launches - c, sum(v for k, v in n.items() if not k.startswith(NET))))
    return out


@pytest.mark.parametrize("order,prec,species,opts", [
    (1, 1, False, {}), (1, 0, True, {}), (1, 2, False, {}), (1, 2, True, {}), (0, 0, False, {}), (0, 0, True, {}),
    (1, 1, True, {"pass_launch": 1}), (1, 1, False, {"small_box": 0}), (0, 0, False, {"small_box": 0})])
def test_counter_is_what_the_profiler_sees(order, prec, species, opts, tmp_path):
    import amcfd
    import amcfd_decks as D
    dk = D.small("count", nx=32, ny=16, nz=10, steps=3, power=350.0)
    if species:
        dk.species = (1.0, 5e-9, 0.3, 0.7)
    s = amcfd.Solver(amcfd.Deck(dk.write(str(tmp_path))), order=order, precision=prec, **opts)
    s.step()
    for counted, seen in _count(s):
        assert counted == seen
    s.close()


def test_counter_with_a_rejected_warm_start(tmp_path):
    """An output bias of 50 has both increments rejected, so every residual is formed."""
    import amcfd
    import amcfd_decks as D
    net = amcfd.Net(seed=5)
    w = net.params()
    w[-16:-14] = 50.0
    net.set_params(w)
    d = amcfd.Deck(D.small("wscount", nx=32, ny=16, nz=10, steps=3).write(str(tmp_path)))
    s = amcfd.Solver(d, order=amcfd.ORDER_REDBLACK, precision=amcfd.PREC_FP64)
    s.ws_attach(net, amcfd.WS_PREDICT)
    s.step()
    for counted, seen in _count(s):
        assert counted == seen
    assert s.ws_stats() == (0, 3)
    s.close()
    net.close()
