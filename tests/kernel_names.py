"""Which kernels a call launches, by the profiler's names: the scenarios of
test_launch_names.py, run in a process of their own (`python tests/kernel_names.py`, one JSON
line), since the profiler loses launches in a process that has run for long.  Direct launches
only: for a replayed graph it can report the names of one that has been destroyed.  Every
stretch is bracketed by fills that have to be seen themselves."""
import json
import os
import re
import sys
import tempfile
from collections import Counter

# (order, precision, nx, ny, nz): the launch that the whole-domain line solve takes
SWEEPS = {
    (1, 1, 60, 13, 9): "sweep_resident_kernel<float, 1>", (1, 1, 511, 13, 8): "sweep_resident_kernel<float, 4>",
    (1, 1, 512, 12, 7): "sweep_rb_pipe_kernel<float>", (1, 1, 530, 12, 9): "sweep_rb_pipe_kernel<float>",
    (1, 2, 60, 12, 9): "sweep_resident_kernel<float, 1>", (1, 2, 530, 13, 9): "sweep_rb_pipe_kernel<float>",
    (1, 0, 130, 12, 9): "sweep_resident_kernel<double, 3>", (1, 0, 255, 12, 8): "sweep_resident_kernel<double, 4>",
    (1, 0, 256, 13, 8): "sweep_rb_pipe_kernel<double>", (1, 0, 270, 13, 9): "sweep_rb_pipe_kernel<double>",
    (0, 0, 60, 13, 9): "sweep_rows_kernel<double, 2>", (0, 0, 128, 12, 8): "sweep_rows_kernel<double, 4>",
    (0, 0, 140, 13, 9): "sweep_exact_kernel<double, false>", (0, 1, 140, 12, 9): "sweep_exact_kernel<float, false>",
}
# (precision, nx, ny, nz): the autotuner on domains that fit the resident launch and that do not
TUNING = [(1, 40, 20, 14), (2, 40, 20, 14), (0, 40, 20, 14), (1, 530, 12, 7), (0, 270, 12, 7)]
# (scheme, precision, nx, ny, nz): at most one CTA a SM, at most three, more
SCHEMES = [(s, p, *n) for s in ("exponential_law", "power_law") for p in (0, 1, 2)
           for n in ((60, 30, 20), (120, 60, 40), (200, 100, 60))]
# (order, precision, species, options): forms of a step that launch differently
COUNTS = [(1, 1, 0, ""), (1, 0, 1, ""), (1, 2, 0, ""), (1, 2, 1, ""), (0, 0, 0, ""), (0, 0, 1, ""),
          (1, 1, 1, "pass_launch=1"), (1, 1, 0, "small_box=0"), (0, 0, 0, "small_box=0"), (1, 0, 0, "warm start")]
POWDER = dict(nx=250, ny=60, nz=56, tracks=2, track_steps=2, dwell_steps=1, ncvzlayer=4)
# the network's own kernels are not the solver's launches
NET = ("conv_tc", "pack_fwd", "pack_bwd", "features_kernel", "reduce_parts", "wgrad", "bgrad", "mse", "adam")


def launched(run):
    """Kernel names ("sweep_rb_pipe_kernel<float>") and counts of what run() launches, or None
    where the profiler has not seen all of it."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    mark = torch.zeros(1 << 16, device="cuda")

    def fill():
        mark.fill_(1.0)
        torch.cuda.synchronize()

    fill()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        fill()
        run()
        torch.cuda.synchronize()
        fill()
    names, marks = Counter(), 0
    for e in prof.events():
        m = re.match(r"(?:void )?amcfd::(\w+(?:<[^>(]*>)?)\(", e.name)
        if m:
            names[m.group(1)] += 1
        elif "FillFunctor" in e.name:
            marks += 1
    return dict(names) if marks == 2 else None


def scenarios(tmp):
    import amcfd
    import amcfd_decks as D

    def deck(dk):
        return amcfd.Deck(dk.write(tempfile.mkdtemp(dir=tmp)))

    out = {}
    for order, prec, nx, ny, nz in SWEEPS:
        s = amcfd.Solver(deck(D.small("k", nx=nx, ny=ny, nz=nz, steps=2)), order=order, precision=prec)
        out[f"sweep {order} {prec} {nx} {ny} {nz}"] = launched(s.step)
        s.close()
    for prec, nx, ny, nz in TUNING:
        made = []
        d = deck(D.small("k", nx=nx, ny=ny, nz=nz, steps=2))
        n = launched(lambda: made.append(amcfd.Solver(d, order=1, precision=prec, autotune=1)))
        out[f"tuning {prec} {nx} {ny} {nz}"] = n and {"create": n, "step": launched(made[0].step),
                                                        "stride": made[0].tuning()["pipe_stride"]}
        made[0].close()
    for scheme, prec, nx, ny, nz in SCHEMES:
        d = D.Deck(name="k", x_zones=[(33e-6 * nx, nx, 1.0)], y_zones=[(33e-6 * ny, ny, 1.0)],
                   z_zones=[(15e-6 * nz, nz, 1.0)], power=250.0, scheme=scheme,
                   single_track=(1.0, 33e-6 * nx * 0.4, 33e-6 * ny * 0.5, 1.0), finaltime=1e-3)
        s = amcfd.Solver(deck(d), order=1, precision=prec, check_finite=0)
        s.run_phase("laser")
        out[f"scheme {scheme} {prec} {nx} {ny} {nz}"] = launched(lambda: s.run_phase("energy_assemble"))
        s.close()
    for order, prec, species, opts in COUNTS:
        dk = D.small("k", nx=32, ny=16, nz=10, steps=3, power=350.0)
        if species:
            dk.species = (1.0, 5e-9, 0.3, 0.7)
        warm = opts == "warm start"
        kw = {} if warm or not opts else {opts.split("=")[0]: int(opts.split("=")[1])}
        s = amcfd.Solver(deck(dk), order=order, precision=prec, **kw)
        if warm:  # an output bias of 50 has both increments rejected, so every residual is formed
            net = amcfd.Net(seed=5)
            w = net.params()
            w[-16:-14] = 50.0
            net.set_params(w)
            s.ws_attach(net, amcfd.WS_PREDICT)
        s.step()
        pairs = []
        for _ in range(2):
            c = s.launches
            n = launched(s.step)
            pairs.append(n and (s.launches - c, sum(v for k, v in n.items() if not k.startswith(NET))))
        out[f"count {order} {prec} {species} {opts}"] = pairs if all(pairs) else None
        s.close()
    s = amcfd.Solver(deck(D.powder_layers("k", **POWDER)), order=1, precision=0, check_finite=0)
    steps = [launched(s.step) for _ in range(5)]
    out["powder"] = steps if all(steps) else None
    s.close()
    return out


if __name__ == "__main__":
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    sys.path.insert(0, os.path.join(root, "am-cfd_b200"))
    with tempfile.TemporaryDirectory() as folder:
        print(json.dumps(scenarios(folder)))
