"""The one-launch momentum chain (one cluster of CTAs, lines exchanging values through
distributed shared memory) against the multi-launch forms of the same chain.

Every operation of the chain is that of the multi-launch kernels, the residual sums
included, so the two give the same bits: the tolerance is zero.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("temp", "enthalpy", "uvel", "vvel", "wvel", "pressure", "pp", "dux", "dvy", "dwz")
REPORT = ("niter", "resorh", "resorm", "resoru", "resorv", "resorw", "tpeak", "alen", "depth", "width", "ratio")


def _same(d, steps, every=1, **kw):
    import amcfd
    a = amcfd.Solver(d, serial_launch=1, small_box=0, **kw)
    b = amcfd.Solver(d, **kw)
    la = lb = 0
    most = (0, 0, 0)
    for q in range(steps):
        la, lb = a.launches, b.launches
        ra, rb = a.step(), b.step()
        n, nj, nk = rb["iend"] - rb["istat"] - 1, rb["jend"] - rb["jstat"] + 1, b.shape[0] - 1 - rb["kstat"]
        most = max(most, (n, nj, nk), key=lambda v: v[0] * v[1] * v[2])
        where = (q + 1, "box", n, nj, nk)
        for k in REPORT:
            assert np.array_equal(ra[k], rb[k], equal_nan=True), (where, k, ra[k], rb[k])
        if q % every == every - 1 or q == steps - 1:
            for f in FIELDS:
                x, y = a.get(f), b.get(f)
                assert np.array_equal(x, y), (where, f, int((x != y).sum()), float(np.abs(x - y).max()))
    assert most[0] > 0
    fewer = (b.launches - lb) < (a.launches - la)
    a.close()
    b.close()
    return most, fewer


@pytest.mark.parametrize("prec,order,graphs", [(0, 0, 0), (0, 0, 1), (0, 1, 1), (1, 1, 0), (1, 1, 1), (2, 1, 1), (1, 0, 1)])
@pytest.mark.parametrize("nx,ny,nz,power", [(24, 14, 10, 350.0), (23, 13, 9, 300.0), (40, 22, 6, 400.0)])
def test_chain_matches_multi_launch_chain(prec, order, graphs, nx, ny, nz, power, tmp_path):
    """Small decks (boxes that reach the domain's faces, odd row counts, one-line
    colours) in both orders and every precision, with graphs and direct launches."""
    import amcfd
    import amcfd_decks as D
    d = amcfd.Deck(D.small("chain", nx=nx, ny=ny, nz=nz, steps=4, power=power, toolpath=True).write(str(tmp_path)))
    _, fewer = _same(d, 4, precision=prec, order=order, use_graphs=graphs)
    assert fewer


def _wide(name, nx, ny, nz, power, radius, dx=30e-6, dy=30e-6, dz=8e-6):
    """A uniform grid under a flat-topped beam: the pool is as wide as the beam."""
    import amcfd_decks as D
    d = D.Deck(name=name, x_zones=[(dx * nx, nx, 1.0)], y_zones=[(dy * ny, ny, 1.0)], z_zones=[(dz * nz, nz, 1.0)],
               power=power, radius=radius, laser_factor=1e-7,
               single_track=(1.0, dx * nx * 0.4, dy * ny * 0.5, 1.0), finaltime=1e-3)
    return d


@pytest.mark.parametrize("prec,order", [(1, 1), (0, 1), (0, 0)])
@pytest.mark.parametrize("nx,ny,nz,power,radius,dy,lines", [
    (60, 60, 30, 5.75e3, 500e-6, 30e-6, "two cells a lane"),       # 32 < cells a line <= 64
    (120, 110, 30, 27.8e3, 1100e-6, 30e-6, "past the capacity"),      # more than 64 cells a line: the multi-launch path
    (76, 130, 30, 14e3, 780e-6, 20e-6, "two lines a warp"),        # more than 256 lines
])
def test_chain_capacity_edges(prec, order, nx, ny, nz, power, radius, dy, lines, tmp_path):
    """Boxes whose lines hold 33-64 cells, boxes with more lines than the cluster has
    warps, and boxes that outgrow the chain within a step (solved in place by the
    chain in that iteration, by the multi-launch path from the next one on)."""
    import amcfd
    d = amcfd.Deck(_wide("edge", nx, ny, nz, power, radius, dy=dy).write(str(tmp_path)))
    most, _ = _same(d, 6, precision=prec, order=order, use_graphs=1)
    n, nj, nk = most
    print(lines, most)
    if lines == "two cells a lane":
        assert 32 < n <= 64, most
    elif lines == "past the capacity":
        assert n > 64, most
    else:
        assert n <= 64 and nj * nk > 256, most
