"""Which contexts of a batch take their first step alone: a kernel's first launch loads
it, which must not happen while another thread captures a graph, so a context may begin
beside the others only when one that launches the same kernels has stepped."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(tmp, name, species=False, solid=False, scheme="power_law", **kw):
    import amcfd
    import amcfd_decks as D
    d = D.small(name, nx=40, ny=22, nz=12, steps=4, power=350.0, scheme=scheme, toolpath=True)
    if species:
        d.species = (1.0, 5e-9, 0.3, 0.7)
    d.solidification = solid
    opts = dict(order=amcfd.ORDER_REDBLACK, precision=amcfd.PREC_FP32, use_graphs=1)
    return amcfd.Solver(amcfd.Deck(d.write(str(tmp / name))), **dict(opts, **kw))


def _calls():
    import amcfd
    lib = amcfd.lib()
    kind, stepped = lib._ZN5amcfd8ctx_kindEPK9amcfd_ctx, lib._ZN5amcfd11ctx_steppedEPK9amcfd_ctx
    kind.argtypes = stepped.argtypes = [C.c_void_p]
    kind.restype, stepped.restype = C.c_int, C.c_bool
    return (lambda s: kind(s._h)), (lambda s: stepped(s._h))


def test_kinds_tell_the_kernels_apart(tmp_path):
    import amcfd
    kind, _ = _calls()
    forms = [dict(), dict(species=True), dict(solid=True), dict(scheme="upwind"), dict(scheme="exponential_law"),
             dict(pass_launch=1), dict(serial_launch=1), dict(small_box=0), dict(host_loop=1), dict(use_graphs=0),
             dict(precision=amcfd.PREC_FP64), dict(precision=amcfd.PREC_FP32_DC),
             dict(precision=amcfd.PREC_FP64, order=amcfd.ORDER_EXACT)]
    keys = []
    for q, f in enumerate(forms):
        a, b = _solver(tmp_path, f"a{q}", **f), _solver(tmp_path, f"b{q}", **f)
        assert kind(a) == kind(b) >= 0, f
        keys.append(kind(a))
        a.close()
        b.close()
    assert len(set(keys)) == len(forms), keys


def test_a_context_has_stepped_as_what_it_is_now(tmp_path):
    import amcfd
    _, stepped = _calls()
    s = _solver(tmp_path, "now")
    assert not stepped(s)
    s.run_phase("laser")
    s.run_phase("energy_assemble")
    assert not stepped(s)
    s.step()
    assert stepped(s)
    net = amcfd.Net(seed=3)
    s.ws_attach(net, amcfd.WS_PREDICT)
    assert not stepped(s)
    s.step()
    assert stepped(s)
    s.close()
    net.close()


def test_new_features_beside_stepped_contexts(tmp_path):
    """Stepped plain contexts and fresh ones with species and G/R in one batch: every
    instance's fields are those of running it alone."""
    import amcfd

    def make(tag):
        return [_solver(tmp_path, tag + "p0"), _solver(tmp_path, tag + "p1"), _solver(tmp_path, tag + "s", species=True),
                _solver(tmp_path, tag + "g", solid=True)]

    batch, alone = make("b"), make("a")
    for s in batch[:2] + alone[:2]:
        s.step()
    amcfd.run_batch(batch, 3)
    for q, (x, y) in enumerate(zip(batch, alone)):
        for _ in range(3):
            y.step()
        for f in ("temp", "uvel", "pressure") + (("avgconcentration",) if q == 2 else ()) + (("grad",) if q == 3 else ()):
            assert np.array_equal(x.get(f), y.get(f)), (q, f)
        x.close()
        y.close()
