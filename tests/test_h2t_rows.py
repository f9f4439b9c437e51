"""The enthalpy inversion over rows of every make-up of chunks (a warp keeps to one
chunk of the row, 128 cells in FP32 and 64 in FP64): every node's temperature and liquid
fraction against the closed form in FP64, and the peak against the field."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _deck(tmp, nx, ny, nz):
    import amcfd_decks as D
    dx = 30e-6
    d = D.Deck(name="h2t", x_zones=[(dx * nx, nx, 1.0)], y_zones=[(dx * ny, ny, 1.2)],
               z_zones=[(20e-6 * nz, nz, 1.1)], power=400.0, single_track=(1.0, dx * nx * 0.4, dx * ny * 0.5, 1.0),
               finaltime=1e-3)
    return d, d.write(str(tmp))


# rows of one chunk and less, of whole chunks either side, of more chunks than a
# small launch has warps for, and boxes of three planes
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("nx,ny,nz", [(5, 4, 3), (62, 9, 6), (64, 8, 5), (126, 6, 5), (128, 7, 4), (254, 5, 4),
                                      (257, 30, 9), (700, 4, 3), (1400, 3, 3),
                                      (1502, 3, 3), (90, 120, 3)])
def test_inversion_of_every_node(prec, nx, ny, nz, tmp_path):
    import amcfd
    d, path = _deck(tmp_path, nx, ny, nz)
    deck = amcfd.Deck(path)
    s = amcfd.Solver(deck, order=amcfd.ORDER_REDBLACK, precision=prec)
    p = deck.params
    hlcal = p.hsmelt + (p.acpa * p.tsolid + p.acpb + p.acpl) * 0.5 * (p.tliquid - p.tsolid)
    for _ in range(2):
        s.run_phase("laser")
        for _ in range(4):
            for ph in ("energy_assemble", "energy_solve", "h2t", "meltpool"):
                r = s.run_phase(ph)
    h = s.get("enthalpy").astype(np.float64)
    temp, fracl = s.get("temp"), s.get("fracl")
    with np.errstate(invalid="ignore"):
        solid = (np.sqrt(p.acpb ** 2 + 2 * p.acpa * h) - p.acpb) / p.acpa
    fl = np.clip((h - p.hsmelt) / (hlcal - p.hsmelt), 0.0, 1.0)
    t = np.where(h >= hlcal, (h - hlcal) / p.acpl + p.tliquid,
                 np.where(h <= p.hsmelt, solid, (p.tliquid - p.tsolid) * fl + p.tsolid))
    # FP64: a handful of roundings, the root's cancellation (b / (a T), below 100) on them;
    # FP32: those and one rounding of the result (2^-24)
    tol = 100 * 16 * 2.0 ** -53 + (2.0 ** -24 if prec else 0.0)
    assert np.all(np.isfinite(t))
    assert np.max(np.abs(temp - t) / t) <= tol
    assert np.max(np.abs(fracl - fl)) <= tol
    assert np.any(fracl > 0) or nx * ny * nz > 1000
    assert r["tpeak"] == float(temp.max())
    s.close()
