"""The exponential scheme's launch shapes of the energy assembly against one another (which
form it takes: test_launch_names.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STATE = ("enthalpy", "hnot", "fracl", "fraclnot", "temp", "uvel", "vvel", "wvel", "unot", "vnot", "wnot",
         "pressure", "diff", "rho", "vis")
OUT = ("an", "as", "ae", "aw", "at", "ab", "ap", "su", "diff_next", "rho_next", "vis_next")


def _deck(tmp, scheme, nx, ny, nz):
    import amcfd
    import amcfd_decks as D
    d = D.Deck(name="sch", x_zones=[(33e-6 * nx, nx, 1.0)], y_zones=[(33e-6 * ny, ny, 1.0)],
               z_zones=[(15e-6 * nz, nz, 1.0)], power=250.0, scheme=scheme,
               single_track=(1.0, 33e-6 * nx * 0.4, 33e-6 * ny * 0.5, 1.0), finaltime=1e-3)
    return amcfd.Deck(d.write(str(tmp / scheme)))


@pytest.mark.parametrize("prec", [0, 1])  # (defect correction keeps its coefficients to itself)
def test_exponential_launch_shapes_give_the_same_coefficients(prec, tmp_path):
    """A flow everywhere (the power-law run's fields with a drift added), so that most
    coefficients are numbers; bit for bit, NaNs in the same places."""
    import amcfd
    nx, ny, nz = 120, 60, 40
    kw = dict(order=amcfd.ORDER_REDBLACK, precision=prec, check_finite=0)
    s = amcfd.Solver(_deck(tmp_path, "power_law", nx, ny, nz), **kw)
    for _ in range(3):
        s.step()
    state = {f: s.get(f) for f in STATE}
    s.close()
    rng = np.random.default_rng(5)
    for f, quiet in (("uvel", 0.0), ("vvel", 0.0), ("wvel", 0.02)):
        drift = rng.uniform(0.01, 0.2, state[f].shape)
        state[f] = state[f] + np.where(rng.random(drift.shape) < quiet, 0.0, drift)
    deck = _deck(tmp_path, "exponential_law", nx, ny, nz)
    ref = None
    for kseg in (16, 8, 4):
        a = amcfd.Solver(deck, asm_kseg=kseg, **kw)
        for f in STATE:
            a.set(f, state[f])
        a.run_phase("laser")
        a.run_phase("energy_assemble")
        out = {f: a.get(f) for f in OUT}
        a.close()
        if ref is None:
            ref = out
            assert 0.5 < np.mean(np.isfinite(out["ap"])) < 1.0
        planes = [k for k in range(nz + 2) if prec != 0 or k % 4]
        for f in OUT:
            x, y = ref[f][planes], out[f][planes]
            assert np.array_equal(x, y, equal_nan=True), (kseg, f)
