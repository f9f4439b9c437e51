"""The red-black passes with every line kept by a warp (the resident launch of small
domains) against a launch per pass: the line arithmetic is the same, so the two
give the same bits (tolerance zero)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("temp", "enthalpy", "uvel", "pressure")


def _deck(tmp, nx, ny, nz, species=False):
    """A uniform grid whose beam melts within the first steps."""
    import amcfd
    import amcfd_decks as D
    dx = 30e-6
    d = D.Deck(name="res", x_zones=[(dx * nx, nx, 1.0)], y_zones=[(dx * ny, ny, 1.0)],
               z_zones=[(20e-6 * nz, nz, 1.0)], power=300.0, single_track=(1.0, dx * nx * 0.4, dx * ny * 0.5, 1.0),
               finaltime=1e-3)
    if species:
        d.species = (1.0, 5e-9, 0.3, 0.7)
    return amcfd.Deck(d.write(str(tmp)))


# x-lines either side of a whole number of rounds (128 cells in FP32, 64 in FP64) up
# to four, odd and even row counts, a single row of a colour, domains whose rows
# only partly fit shared memory (200x100x60)
@pytest.mark.parametrize("prec,nx,ny,nz,species", [
    (1, 24, 14, 10, False), (1, 127, 21, 9, False), (1, 128, 20, 9, True), (1, 255, 13, 8, False),
    (1, 256, 12, 8, False), (1, 383, 12, 7, False), (1, 384, 11, 8, False), (1, 510, 12, 8, False),
    (1, 30, 13, 3, False), (1, 200, 100, 60, False), (2, 200, 100, 60, False), (2, 61, 31, 21, True),
    (0, 63, 14, 9, False), (0, 64, 13, 9, True), (0, 127, 12, 8, False), (0, 128, 13, 8, False),
    (0, 191, 12, 7, False), (0, 192, 11, 8, False), (0, 254, 12, 8, False), (0, 131, 67, 41, False)])
def test_resident_passes_bit_identical(prec, nx, ny, nz, species, tmp_path):
    import amcfd
    d = _deck(tmp_path, nx, ny, nz, species)
    kw = dict(order=amcfd.ORDER_REDBLACK, precision=prec, use_graphs=1)
    a = amcfd.Solver(d, pass_launch=1, **kw)
    b = amcfd.Solver(d, **kw)
    for q in range(3):
        ra, rb = a.step(), b.step()
        for k in ("niter", "resorh", "resorm", "tpeak", "alen"):
            assert np.array_equal(ra[k], rb[k], equal_nan=True), (q + 1, k, ra[k], rb[k])
        for f in FIELDS + (("avgconcentration",) if species else ()):
            x, y = a.get(f), b.get(f)
            assert np.array_equal(x, y), (q + 1, f, int((x != y).sum()), float(np.abs(x - y).max()))
    a.close()
    b.close()
