"""The pipelined launch of the red-black passes against a launch per pass on domains that no
other launch takes (rows of more cells than the launch with every line in a warp has
rounds for: 512 in FP32, 256 in FP64; by name in test_launch_names.py), of odd sizes, with
the species equation, and on a powder bed that grows out of the one launch into the other.
The line arithmetic is the same: the tolerance is zero."""
import numpy as np
import pytest

from kernel_names import POWDER

pytestmark = pytest.mark.gpu


def _same(d, steps, prec, fields, **kw):
    import amcfd
    kw = dict(kw, order=amcfd.ORDER_REDBLACK, precision=prec)
    a, b = amcfd.Solver(d, pass_launch=1, **kw), amcfd.Solver(d, **kw)
    for q in range(steps):
        ra, rb = a.step(), b.step()
        for k in ("niter", "resorh", "resorm", "tpeak", "alen"):
            assert np.array_equal(ra[k], rb[k], equal_nan=True), (q + 1, k, ra[k], rb[k])
        for f in fields:
            x, y = a.get(f), b.get(f)
            assert np.array_equal(x, y, equal_nan=True), (q + 1, f, int((x != y).sum()))
    a.close()
    b.close()


@pytest.mark.parametrize("prec,nx,ny,nz,species", [
    (1, 511, 13, 8, False), (1, 512, 12, 7, True), (1, 530, 13, 7, False), (1, 639, 5, 9, True), (1, 700, 1, 6, False),
    (1, 600, 6, 1, False), (2, 530, 13, 7, True), (2, 641, 12, 6, False), (0, 255, 12, 8, False), (0, 256, 13, 8, True),
    (0, 319, 7, 5, False), (0, 520, 12, 4, False)])
def test_long_rows_bit_identical(prec, nx, ny, nz, species, tmp_path):
    import amcfd
    import amcfd_decks as D
    dx = 30e-6
    dk = D.Deck(name="long", x_zones=[(dx * nx, nx, 1.0)], y_zones=[(dx * ny, ny, 1.0)], z_zones=[(20e-6 * nz, nz, 1.0)],
                power=300.0 if min(ny, nz) > 2 else 30.0, fluid_flow=min(ny, nz) > 2,
                single_track=(1.0, dx * nx * 0.4, dx * ny * 0.5, 1.0), finaltime=1e-3)
    if species:
        dk.species = (1.0, 5e-9, 0.3, 0.7)
    _same(amcfd.Deck(dk.write(str(tmp_path))), 3, prec,
          ("temp", "enthalpy", "uvel", "pressure") + (("avgconcentration",) if species else ()))


@pytest.mark.parametrize("graphs", [0, 1])
def test_powder_bed_grows_out_of_the_resident_launch(graphs, tmp_path):
    """The second layer, in step 4, no longer fits (test_launch_names.py)."""
    import amcfd
    import amcfd_decks as D
    _same(amcfd.Deck(D.powder_layers("grow", **POWDER).write(str(tmp_path))), 5, 0, ("temp", "enthalpy", "rho", "csfrac"),
          use_graphs=graphs, check_finite=0)
