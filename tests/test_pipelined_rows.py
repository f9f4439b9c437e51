"""The pipelined launch of the red-black passes against a launch per pass on domains that no
other launch takes (rows of more cells than the launch with every line in a warp has
rounds for: 512 in FP32, 256 in FP64), of odd sizes, with the species equation, and on a
powder bed that grows out of the one launch into the other.  The line arithmetic is the
same: the tolerance is zero."""
import numpy as np
import pytest

from kernel_names import launched

pytestmark = pytest.mark.gpu


def _same(d, steps, prec, fields, **kw):
    """Both forms step by step, the names of the second's kernels."""
    import amcfd
    kw = dict(kw, order=amcfd.ORDER_REDBLACK, precision=prec)
    a, b = amcfd.Solver(d, pass_launch=1, **kw), amcfd.Solver(d, **kw)
    names = []
    for q in range(steps):
        ra, rb = a.step(), None

        def step():
            nonlocal rb
            rb = b.step()

        names.append({k.split("<")[0] for k in launched(step)})
        for k in ("niter", "resorh", "resorm", "tpeak", "alen"):
            assert np.array_equal(ra[k], rb[k], equal_nan=True), (q + 1, k, ra[k], rb[k])
        for f in fields:
            x, y = a.get(f), b.get(f)
            assert np.array_equal(x, y, equal_nan=True), (q + 1, f, int((x != y).sum()))
    a.close()
    b.close()
    return names


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
    names = _same(amcfd.Deck(dk.write(str(tmp_path))), 3, prec,
                  ("temp", "enthalpy", "uvel", "pressure") + (("avgconcentration",) if species else ()))
    long_row = nx > (256 if prec == 0 else 512) - 1
    want = "sweep_rb_pipe_kernel" if long_row else "sweep_resident_kernel"
    assert all(want in n for n in names), names


@pytest.mark.parametrize("graphs", [0, 1])
def test_powder_bed_grows_out_of_the_resident_launch(graphs, tmp_path):
    """250x60 cells in FP64: 64 planes of 30 slots fit 148 CTAs of 13 (224 KB of rows), the 68
    planes with the second layer do not."""
    import amcfd
    import amcfd_decks as D
    dk = D.powder_layers("grow", nx=250, ny=60, nz=56, tracks=2, track_steps=2, dwell_steps=1, ncvzlayer=4)
    names = _same(amcfd.Deck(dk.write(str(tmp_path))), 5, 0, ("temp", "enthalpy", "rho", "csfrac"), use_graphs=graphs,
                  check_finite=0)
    if not graphs:
        kinds = [("sweep_resident_kernel" in n, "sweep_rb_pipe_kernel" in n) for n in names]
        assert kinds == [(True, False)] * 3 + [(False, True)] * 2, kinds
