"""The forms of the energy assembly's cell (with and without a mass flux) and its launch
shapes against one another.

A warp whose cells see no flow takes a shorter form of the same cell; which
instantiation runs follows from the number of CTAs, which the planes per CTA
(asm_kseg) set.  From one state -- a melt pool with flow in a solid, still plate --
every shape must give the same coefficients, sources and properties, bit for bit: the
short form skips operations whose result is exact (A(0) = 1, + 0), nothing else, and where
rows have six tiles and more a warp away from the boundary skips its choices too.
FP64 compares the planes that begin no segment in either shape: a segment's first plane
forms its bottom face afresh instead of carrying it from the plane below, in an
expression that FP64 may round differently.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STATE = ("enthalpy", "hnot", "fracl", "fraclnot", "temp", "uvel", "vvel", "wvel", "unot", "vnot", "wnot",
         "pressure", "diff", "rho", "vis")
OUT = ("an", "as", "ae", "aw", "at", "ab", "ap", "su", "diff_next", "rho_next", "vis_next")


# 70x30x20: 24 CTAs at 16 planes, 72 at 4 (at most one a SM: the long form only);
# 120x60x40: 96 and 352; 201x91x61: 336 and 1344 (FP32: four CTAs a SM); 160x38x20 and
# 190x38x20 (rows of six tiles, the last one short and whole): 60 and 180, the long form
# against the short one without boundary faces
@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("scheme", ["power_law", "upwind"])
@pytest.mark.parametrize("nx,ny,nz", [(70, 30, 20), (120, 60, 40), (160, 38, 20), (190, 38, 20),
                                      (201, 91, 61)])
def test_launch_shapes_give_the_same_coefficients(prec, scheme, nx, ny, nz, tmp_path):
    import amcfd
    import amcfd_decks as D
    d = D.Deck(name="forms", x_zones=[(33e-6 * nx, nx, 1.0)], y_zones=[(33e-6 * ny, ny, 1.0)],
               z_zones=[(15e-6 * nz, nz, 1.0)], power=250.0, scheme=scheme,
               single_track=(1.0, 33e-6 * nx * 0.4, 33e-6 * ny * 0.5, 1.0), finaltime=1e-3)
    deck = amcfd.Deck(d.write(str(tmp_path)))
    kw = dict(order=amcfd.ORDER_REDBLACK, precision=prec)
    s = amcfd.Solver(deck, **kw)
    for _ in range(4):
        s.step()
    state = {f: s.get(f) for f in STATE}
    assert np.any(state["uvel"] != 0.0) and np.mean(state["uvel"] != 0.0) < 0.2
    s.close()
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
        planes = [k for k in range(nz + 2) if prec != 0 or k % 4]
        for f in OUT:
            x, y = ref[f][planes], out[f][planes]
            assert np.array_equal(x, y), (kseg, f, int((x != y).sum()))
