"""The exact-order sweep of the whole domain by rows of visits (a warp walks along j, the
neighbours' values carry their version) against the sweep by single visits: the same
visits see the same values and the line arithmetic is the same code, so the two give
the same bits (tolerance zero)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# lines of one to four cells a lane and either side of each, lines too long for it (129,
# 200: by single visits), more rows than warps
@pytest.mark.parametrize("prec,nx,ny,nz,species", [
    (0, 24, 14, 10, False), (0, 20, 12, 3, False), (0, 31, 13, 8, True), (0, 32, 12, 9, False), (0, 33, 12, 8, False),
    (0, 64, 14, 8, False), (0, 65, 13, 9, False), (0, 96, 13, 8, False), (0, 97, 12, 8, False),
    (0, 128, 12, 8, False), (0, 129, 12, 8, False), (0, 200, 12, 8, False), (0, 61, 31, 21, False), (0, 24, 60, 30, False),
    (1, 24, 14, 10, False), (1, 65, 13, 9, True), (1, 130, 40, 20, False)])
def test_rows_bit_identical(prec, nx, ny, nz, species, tmp_path):
    import amcfd
    import amcfd_decks as D
    dx = 30e-6
    dk = D.Deck(name="rows", x_zones=[(dx * nx, nx, 1.0)], y_zones=[(dx * ny, ny, 1.0)], z_zones=[(20e-6 * nz, nz, 1.0)],
                power=300.0, single_track=(1.0, dx * nx * 0.4, dx * ny * 0.5, 1.0), finaltime=1e-3)
    if species:
        dk.species = (1.0, 5e-9, 0.3, 0.7)
    d = amcfd.Deck(dk.write(str(tmp_path)))
    a = amcfd.Solver(d, precision=prec, serial_launch=1)
    b = amcfd.Solver(d, precision=prec, use_graphs=nx % 2)
    for q in range(3):
        ra, rb = a.step(), b.step()
        for k in ("niter", "resorh", "resorm", "tpeak", "alen"):
            assert np.array_equal(ra[k], rb[k], equal_nan=True), (q + 1, k, ra[k], rb[k])
        for f in ("temp", "enthalpy", "uvel", "pressure") + (("avgconcentration",) if species else ()):
            x, y = a.get(f), b.get(f)
            assert np.array_equal(x, y), (q + 1, f, int((x != y).sum()), float(np.abs(x - y).max()))
    a.close()
    b.close()


@pytest.mark.parametrize("ny,nz", [(1, 6), (2, 5), (6, 1), (5, 2), (1, 1)])
def test_rows_on_thin_domains(ny, nz, tmp_path):
    """One or two interior rows or planes, against the oracle (conduction only: a pool
    needs more); fields within 1e-10 relative L2, as the sweeps' scans differ from the
    serial recurrences by rounding."""
    import amcfd
    import amcfd_decks as D
    import oracle_py
    dk = D.Deck(name="thin", x_zones=[(30e-6 * 40, 40, 1.0)], y_zones=[(30e-6 * ny, ny, 1.0)],
                z_zones=[(20e-6 * nz, nz, 1.0)], power=30.0, fluid_flow=False,
                single_track=(1.0, 30e-6 * 16, 15e-6 * ny, 1.0), finaltime=1e-3)
    d = amcfd.Deck(dk.write(str(tmp_path)))
    ref = oracle_py.Oracle(d.params)
    s = amcfd.Solver(d)
    for _ in range(2):
        ro, rs = ref.step(), s.step()
        assert ro["niter"] == rs["niter"]
        for f in ("temp", "enthalpy"):
            x, y = s.get(f), ref.field(f)
            assert np.linalg.norm(x - y) <= 1e-10 * np.linalg.norm(y), f
    s.close()
