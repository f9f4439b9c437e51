"""The enthalpy inversion with solid, mushy and liquid cells at every place of a row: the
enthalpy is set, the h2t phase alone runs, and every node's temperature and liquid fraction
are compared with the closed form in FP64.  The enthalpies follow each other with a period
that is prime to the vectors (2 or 4 cells), chunks (64 or 128) and row lengths, so that
each branch comes to every lane and vector position (asserted)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("nx,ny,nz", [(5, 4, 3), (62, 9, 6), (64, 8, 5), (126, 6, 5), (129, 7, 4), (257, 30, 9),
                                      (700, 4, 3), (1502, 3, 3), (90, 120, 3)])
def test_every_branch_at_every_place(prec, nx, ny, nz, tmp_path):
    import amcfd
    import amcfd_decks as D
    dx = 30e-6
    dk = D.Deck(name="h2t", x_zones=[(dx * nx, nx, 1.0)], y_zones=[(dx * ny, ny, 1.2)], z_zones=[(20e-6 * nz, nz, 1.1)],
                power=400.0, single_track=(1.0, dx * nx * 0.4, dx * ny * 0.5, 1.0), finaltime=1e-3)
    deck = amcfd.Deck(dk.write(str(tmp_path)))
    s = amcfd.Solver(deck, order=amcfd.ORDER_REDBLACK, precision=prec)
    p = deck.params
    hlcal = p.hsmelt + (p.acpa * p.tsolid + p.acpb + p.acpl) * 0.5 * (p.tliquid - p.tsolid)
    mush = hlcal - p.hsmelt
    kinds = np.array([0.3 * p.hsmelt, p.hsmelt + 0.25 * mush, hlcal + 0.4 * p.hsmelt, 0.9 * p.hsmelt, p.hsmelt + 0.75 * mush,
                      hlcal + 2.0 * mush, 0.999 * p.hsmelt, p.hsmelt, hlcal, hlcal + 0.01 * mush, 0.5 * p.hsmelt,
                      p.hsmelt + 0.01 * mush, 0.7 * p.hsmelt, hlcal + 0.1 * p.hsmelt, p.hsmelt + 0.99 * mush, 0.2 * p.hsmelt,
                      hlcal + 0.8 * p.hsmelt])  # 17
    h = np.resize(kinds, s.shape)
    if prec:
        h = h.astype(np.float32).astype(np.float64)
    s.run_phase("laser")
    s.set("enthalpy", h)
    assert np.array_equal(s.get("enthalpy"), h)
    s.run_phase("h2t")
    r = s.run_phase("meltpool")
    temp, fracl = s.get("temp"), s.get("fracl")
    fl = np.clip((h - p.hsmelt) / mush, 0.0, 1.0)
    t = np.where(h >= hlcal, (h - hlcal) / p.acpl + p.tliquid,
                 np.where(h <= p.hsmelt, (np.sqrt(p.acpb ** 2 + 2 * p.acpa * np.minimum(h, p.hsmelt)) - p.acpb) / p.acpa,
                          (p.tliquid - p.tsolid) * fl + p.tsolid))
    # all three branches in every column, so at every lane and place of a vector
    for kind in (h <= p.hsmelt, (h > p.hsmelt) & (h < hlcal), h >= hlcal):
        assert kind.any(axis=(0, 1)).all()
    # FP64: a handful of roundings (16), times the root's cancellation (acpb / (acpa T), below
    # 100); FP32: those and one rounding of the result (2^-24)
    tol = 100 * 16 * 2.0 ** -53 + (2.0 ** -24 if prec else 0.0)
    assert np.max(np.abs(temp - t) / t) <= tol
    assert np.max(np.abs(fracl - fl)) <= tol
    assert r["tpeak"] == float(temp.max())
    s.close()
