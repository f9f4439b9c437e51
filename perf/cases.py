"""Timing cases: what a user of the solver has it do, through its public entry points.

A "step" case is one instance of a keyword deck advancing `steps` time steps and
then reading the fields that the deck's output asks for into pinned host memory;
a "batch" case is a process-parameter sweep sharing one GPU; a "train" case is
one training update of the warm-start network.  The decks scale the package's
own configurations: "track" is the single-track deck family (33 um cells,
4.0 x 2.0 x 0.7 mm at 120 x 60 x 40 cells), "diagonal" the fine deck of the
400 x 200 x 100 benchmark, "raster" the 600 x 300 x 120 one.  The beam re-scans one
straight track back and forth, so that a solver can be stepped for as long as one
likes with a melt pool of much the same size.
"""
import math
import os
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "am-cfd_b200"))

import amcfd  # noqa: E402
import amcfd_decks as decks  # noqa: E402

PRECISION = {"fp64": amcfd.PREC_FP64, "fp32": amcfd.PREC_FP32, "dc": amcfd.PREC_FP32_DC}
ORDER = {"exact": amcfd.ORDER_EXACT, "redblack": amcfd.ORDER_REDBLACK}
MAXIT = 20  # outer iterations a step, the decks' own limit (fluid flow never meets the tolerance)


def _step(name, grid, nx, ny, nz, precision="fp32", order="redblack", graphs=1, scheme="power_law",
          feature="none", steps=1, warm=6):
    return {"name": name, "kind": "step", "grid": grid, "nx": nx, "ny": ny, "nz": nz, "precision": precision,
            "order": order, "graphs": graphs, "scheme": scheme, "feature": feature, "steps": steps, "warm": warm}


def listed():
    return [
        # the smallest instance of the parameter sweep, watched step by step: launches and latency
        _step("small_fp32", "track", 60, 30, 20),
        # the 120 x 60 x 40 single-track deck, fields read after every step
        _step("track_fp32", "track", 120, 60, 40),
        # the same process in plain FP64 on odd sizes, upwind scheme
        _step("track_fp64", "track", 131, 67, 41, precision="fp64", scheme="upwind"),
        # the defaults of a caller that sets no option: FP64 in the reference's sweep order, no graphs
        _step("default_fp64", "track", 61, 31, 21, precision="fp64", order="exact", graphs=0),
        # mixed-precision defect correction on the 200 x 100 x 60 evaluation deck
        _step("evaluation_dc", "track", 200, 100, 60, precision="dc"),
        # alloy concentration solved beside the flow, ragged sizes
        _step("species_fp32", "track", 141, 73, 45, feature="species"),
        # the grid follows the beam; G and R of the solidification front after every step
        _step("moving_fp32", "diagonal", 163, 81, 50, feature="moving"),
        # the 8 M cell diagonal scan, the output field read every third step
        _step("diagonal_fp32", "diagonal", 400, 200, 100, steps=3, warm=20),
        # the same deck in plain FP64
        _step("diagonal_fp64", "diagonal", 400, 200, 100, precision="fp64", warm=10),
        # the largest deck, 21.6 M cells
        _step("raster_fp32", "raster", 600, 300, 120, steps=2, warm=6),
        # a process-parameter sweep: eight instances of different grids side by side on one GPU
        {"name": "sweep_fp32", "kind": "batch", "instances": 8, "nx_min": 60, "nx_max": 240, "steps": 2, "warm": 4},
        # one update of the warm-start network on the evaluation deck's grid
        {"name": "train", "kind": "train", "ni": 202, "nj": 102, "nk": 62},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 8 + ["batch", "train"])
    if kind == "batch":
        hi = _spread(rng, 90, 240)
        return {"kind": "batch", "instances": rng.randint(2, 8), "nx_min": 60, "nx_max": hi,
                "steps": rng.randint(1, 2), "warm": 4}
    if kind == "train":
        n = _spread(rng, 30, 200)
        return {"kind": "train", "ni": n + rng.randint(0, 2), "nj": n // 2 + rng.randint(2, 4),
                "nk": n * 3 // 10 + rng.randint(2, 4)}
    precision = rng.choice(["fp32", "fp32", "fp32", "fp64", "dc"])
    grid = rng.choice(["track", "track", "diagonal", "raster"])
    feature = rng.choice(["none"] * 4 + ["species", "moving"])
    order = "redblack"
    hi = 420
    if precision == "fp64" and rng.random() < 0.4:
        order, hi = "exact", 120
    if feature == "moving":
        grid = "diagonal" if grid == "track" else grid
    nx = _spread(rng, 60, hi)
    ny = max(24, int(nx * rng.uniform(0.42, 0.56)))
    nz = max(18, int(nx * rng.uniform(0.2, 0.34)))
    return {"kind": "step", "grid": grid, "nx": nx, "ny": ny, "nz": nz, "precision": precision, "order": order,
            "graphs": 0 if order == "exact" and rng.random() < 0.5 else 1,
            "scheme": rng.choice(["power_law", "power_law", "upwind"]), "feature": feature,
            "steps": 1 if nx < 300 else 2, "warm": 6}


def _rescan(p0, p1, z, speed, until):
    """Toolpath rows of a beam that goes back and forth between p0 and p1, always on."""
    rows, t, q = [(0.0, p0[0], p0[1], z, 1, 1)], 0.0, 0
    leg = math.hypot(p1[0] - p0[0], p1[1] - p0[1]) / speed
    while t < until:
        t += leg
        q += 1
        x, y = (p1, p0)[(q + 1) % 2]
        rows.append((t, x, y, z, 1, 1))
    return rows


def _deck(grid, nx, ny, nz, rng, scheme="power_law", feature="none"):
    if grid == "track":
        lx, ly, lz = 4.0e-3 * nx / 120, 2.0e-3 * ny / 60, 0.7e-3 * nz / 40
        ny1, nz1 = ny // 4, int(round(nz * 0.375))
        x = [(lx, nx, 1.0)]
        y = [(ly * 0.35, ny1, -1.5), (ly * 0.30, ny - 2 * ny1, 1.0), (ly * 0.35, ny1, 1.5)]
        z = [(lz * 5 / 7, nz1, -1.5), (lz * 2 / 7, nz - nz1, 1.0)]
        power, radius, dt, p0, p1 = rng.uniform(180, 260), 50e-6, 1e-5, (0.3, 0.5), (0.7, 0.5)
    else:
        fine = grid == "raster"
        sx, sy, sz = (nx / 600, ny / 300, nz / 120) if fine else (nx / 400, ny / 200, nz / 100)
        fx, fy, fz = (1 / 6, 1 / 6, 1 / 3) if fine else (0.15, 0.15, 0.3)
        zx, zy, zz = ([3.0e-3, 4.0e-3, 3.0e-3], [1.5e-3, 2.0e-3, 1.5e-3], [0.8e-3, 0.4e-3]) if fine else \
            ([1.0e-3, 3.0e-3, 2.0e-3], [1.0e-3, 3.0e-3, 2.0e-3], [0.6e-3, 0.4e-3])
        ax, ay, az = int(nx * fx), int(ny * fy), int(nz * fz)
        x = [(zx[0] * sx, ax, -1.2), (zx[1] * sx, nx - 2 * ax, 1.0), (zx[2] * sx, ax, 1.2)]
        y = [(zy[0] * sy, ay, -1.2), (zy[1] * sy, ny - 2 * ay, 1.0), (zy[2] * sy, ay, 1.2)]
        z = [(zz[0] * sz, az, -1.5), (zz[1] * sz, nz - az, 1.0)]
        lx, ly = sum(v[0] for v in x), sum(v[0] for v in y)
        power, radius, dt = (rng.uniform(180, 220), 50e-6, 1e-5) if fine else (rng.uniform(270, 320), 60e-6, 5e-6)
        p0, p1 = ((0.4, 0.45), (0.6, 0.45)) if fine else ((0.3, 0.3), (0.5, 0.5))
    d = decks.Deck(name="case", x_zones=x, y_zones=y, z_zones=z, power=power, radius=radius, dt=dt, scheme=scheme,
                   finaltime=0.2, maxit=MAXIT)
    d.toolpath = _rescan((p0[0] * lx, p0[1] * ly), (p1[0] * lx, p1[1] * ly), sum(v[0] for v in z),
                         rng.uniform(0.8, 1.2), 0.2)
    if feature == "species":
        d.species = (1.0, 5e-9, 0.3, 0.7)
    elif feature == "moving":
        d.moving_mesh = (2, 2)
        d.solidification = True
    return d


def _solver(deck, **options):
    with tempfile.TemporaryDirectory() as folder:
        return amcfd.Solver(amcfd.Deck(deck.write(folder)), **options)


def _fields(case):
    if case["feature"] == "species":
        return ("temp", "uvel", "avgconcentration")
    if case["feature"] == "moving":
        return ("temp", "grad", "rate")
    # the velocities too, except on decks whose output is the temperature alone
    return ("temp", "uvel", "vvel", "wvel") if case["nx"] * case["ny"] * case["nz"] < 500_000 else ("temp",)


class _Reader:
    """Fields of one solver in pinned host memory, in the solver's own precision."""

    def __init__(self, solver, names, single):
        self.solver, self.names = solver, names
        self.wide = {n: torch.empty(solver.shape, dtype=torch.float64, pin_memory=True) for n in names}
        self.out = {n: torch.empty(solver.shape, dtype=torch.float32) for n in names} if single else self.wide

    def read(self):
        for n in self.names:
            self.solver.get_into(n, self.wide[n].data_ptr())
            if self.out is not self.wide:
                self.out[n].copy_(self.wide[n])
        return dict(self.out)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "train":
        n = case["ni"] * case["nj"] * case["nk"]
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        feat = torch.randn((n, 11), device="cuda", generator=g)
        target = 0.3 * feat[:, :2] + 0.1 * torch.randn((n, 2), device="cuda", generator=g)
        return {"net": amcfd.Net(seed=int(seed) % 1000 + 1), "dims": (case["ni"], case["nj"], case["nk"]),
                "feat": feat, "target": target.contiguous(), "y": torch.zeros((n, 2), device="cuda")}
    if case["kind"] == "batch":
        solvers = []
        for q in range(case["instances"]):  # largest first, as amcfd_run_batch asks
            nx = case["nx_max"] - (case["nx_max"] - case["nx_min"]) * q // max(1, case["instances"] - 1)
            d = _deck("track", nx, nx // 2, max(20, nx // 4), rng)
            solvers.append(_solver(d, order=amcfd.ORDER_REDBLACK, precision=amcfd.PREC_FP32, use_graphs=1))
        amcfd.run_batch(solvers, case["warm"])
        return {"solvers": solvers, "steps": case["steps"], "readers": [_Reader(s, ("temp",), True) for s in solvers]}
    d = _deck(case["grid"], case["nx"], case["ny"], case["nz"], rng, case["scheme"], case["feature"])
    s = _solver(d, order=ORDER[case["order"]], precision=PRECISION[case["precision"]], use_graphs=case["graphs"])
    for _ in range(case["warm"]):
        s.step()
    return {"solver": s, "steps": case["steps"], "reader": _Reader(s, _fields(case), case["precision"] == "fp32")}


def _summary(r):
    return {k: r[k] for k in ("niter", "tpeak", "alen", "depth", "width")}


def run(state):
    if "net" in state:
        net = state["net"]
        net.forward(state["feat"].data_ptr(), state["dims"], state["y"].data_ptr())
        loss = net.backward(state["target"].data_ptr())
        grads = net.grads()
        net.adam(1e-3)
        return {"y": state["y"], "loss": loss, "grads": grads}
    if "solvers" in state:
        reports, _ = amcfd.run_batch(state["solvers"], state["steps"])
        return [{**_summary(r), **reader.read()} for r, reader in zip(reports, state["readers"])]
    s = state["solver"]
    for _ in range(state["steps"]):
        report = s.step()
    return {**_summary(report), **state["reader"].read()}


def work(case):
    if case["kind"] == "train":
        n = case["ni"] * case["nj"] * case["nk"]
        layers = 16 * 32 + 32 * 32 + 32 * 32 + 32 * 16
        # forward, weight gradients, and the input gradients of all layers but the first
        return {"bytes": 4 * n * (11 + 2 + 2), "flops": 2 * 27 * n * (3 * layers - 16 * 32)}
    if case["kind"] == "batch":
        sizes = [case["nx_max"] - (case["nx_max"] - case["nx_min"]) * q // max(1, case["instances"] - 1)
                 for q in range(case["instances"])]
        n = sum(v * (v // 2) * max(20, v // 4) for v in sizes)
        word, fields = 4, 1
    else:
        n = case["nx"] * case["ny"] * case["nz"]
        word, fields = (4 if case["precision"] == "fp32" else 8), len(_fields(case))
    # an outer iteration reads the enthalpy, temperature, liquid fraction, their previous-step
    # values, three velocities and three properties and writes six of them; about 400
    # operations a cell (coefficients, eight line passes, inversion)
    species = 2 if case.get("feature") == "species" else 1
    return {"bytes": case["steps"] * MAXIT * n * 17 * word * species + 8 * n * fields,
            "flops": case["steps"] * MAXIT * n * 400.0 * species}


def exact(case, seed):
    """The network's outputs and gradients in 64 bits.  A time step has no closed
    value: it is twenty unconverged iterations of the solver's own scheme."""
    if case["kind"] != "train":
        return None
    state = prepare(case, seed)
    ni, nj, nk = state["dims"]
    params = torch.from_numpy(state["net"].params().astype(np.float64)).cuda().requires_grad_()
    inner = torch.zeros((1, 1, nk, nj, ni), dtype=torch.float64, device="cuda")
    inner[:, :, 1:-1, 1:-1, 1:-1] = 1.0
    x = torch.zeros((1, 16, nk, nj, ni), dtype=torch.float64, device="cuda")
    x[0, :11] = state["feat"].double().T.reshape(11, nk, nj, ni)
    x, at = x * inner, 0
    for layer, (cin, cout) in enumerate(((16, 32), (32, 32), (32, 32), (32, 16))):
        w = params[at:at + 27 * cin * cout].reshape(3, 3, 3, cout, cin).permute(3, 4, 0, 1, 2)
        at += 27 * cin * cout
        x = torch.nn.functional.conv3d(x, w, params[at:at + cout], padding=1)
        at += cout
        x = (torch.relu(x) if layer < 3 else x) * inner
    y = x[0, :2].reshape(2, -1).T
    mask = inner.reshape(-1, 1)
    loss = (((y - state["target"].double()) * mask) ** 2).sum() / (2 * mask.sum())
    loss.backward()
    return {"y": y.detach().contiguous(), "loss": float(loss), "grads": params.grad.cpu().numpy()}
